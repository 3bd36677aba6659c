"""Source-level guarantees that need no GPU: no cluster-multicast bulk loads, no unbounded traps,
SM-budget model behaviour, packaging of native sources."""

import math
import re
from pathlib import Path

from nanoep_b200.utils import sms
from nanoep_b200.utils.build import SOURCES, source_dir

ROOT = Path(__file__).resolve().parent.parent


def _native_sources():
    return [p for p in (ROOT / "csrc").rglob("*") if p.suffix in {".cu", ".cuh", ".hpp", ".cpp", ".h"}]


def test_no_cluster_multicast_loads_and_no_traps():
    # patterns are assembled from pieces so that this file does not itself contain them
    banned = re.compile("|".join(["multi" + "cast::cluster", "_MULTI" + "CAST", r"__tr" + r"ap\s*\(", r"asm[^;]*\btr" + r"ap;", "Memcpy" + "Batch" + "Async"]))
    for path in _native_sources():
        text = path.read_text()
        assert not banned.search(text), f"{path} uses a construct that is banned in this project"


def _loops(text):
    """(header, body) of every `for`/`while`/`do` loop in C-like source; bodies are brace-matched, a loop
    without braces ends at its first semicolon."""
    for m in re.finditer(r"\b(for|while|do)\b", text):
        i = m.end()
        header = ""
        if m.group(1) != "do":
            while i < len(text) and text[i].isspace():
                i += 1
            if i >= len(text) or text[i] != "(":
                continue
            depth, j = 0, i
            while j < len(text):
                depth += text[j] == "("
                depth -= text[j] == ")"
                j += 1
                if depth == 0:
                    break
            header, i = text[i:j], j
        while i < len(text) and text[i].isspace():
            i += 1
        if i < len(text) and text[i] == "{":
            depth, j = 0, i
            while j < len(text):
                depth += text[j] == "{"
                depth -= text[j] == "}"
                j += 1
                if depth == 0:
                    break
            body = text[i:j]
        else:
            j = text.find(";", i)
            body = text[i : j + 1]
            if m.group(1) == "while" and not body.strip(" ;"):
                continue  # the tail of a do { } while (...);
        yield header, body


def test_every_device_wait_is_bounded():
    """Every loop in the native sources that polls memory, an mbarrier or sleeps must compare a timer (or an
    iteration count) against a limit inside the loop."""
    polls = re.compile(r"ld_acquire|ld_relaxed_sys|try_wait|mbar_try|__nanosleep|volatile")
    bounded = re.compile(r"timeout_ns|limit_ns|deadline|max_spins|kMaxSpins")
    # a counted loop (declares its index, compares it with a bound, steps it) ends by itself unless its header polls
    counted = re.compile(r"^\(\s*(?:int|unsigned|int64_t|uint32_t|size_t)\s+\w+\s*=[^;]*;[^;]*[<>][^;]*;[^;]*(?:\+=|\+\+|-=|--)[^;]*\)$", re.S)
    checked = 0
    for path in _native_sources():
        if path.suffix == ".cpp" or path.name.endswith(".hpp"):
            continue  # host code: its waits are wall-clock bounded and tested separately
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for header, body in _loops(text):
            if counted.match(header.strip()) and not polls.search(header):
                continue
            if polls.search(header) or (polls.search(body) and re.search(r"\b(break|return)\b", body) and not re.search(r"\bfor\b|\bwhile\b", body[1:])):
                checked += 1
                assert bounded.search(header + body), f"{path.name}: unbounded wait loop: {header} {body[:200]}"
    assert checked >= 6, "the scan found no wait loops; the patterns are stale"


def test_build_lists_existing_sources():
    for name in SOURCES:
        assert (source_dir() / name).exists(), name


def test_sm_budget_model():
    assert sms.theoretical_num_sms(148, 1, 256, 8, 810.0) == 148
    assert sms.theoretical_num_sms(148, 8, 256, 8, 0.0) == 148  # unknown NVLink -> all SMs
    n = sms.theoretical_num_sms(148, 8, 256, 8, 810.0)
    assert 16 <= n <= 148 and n % 4 == 0
    assert sms.theoretical_num_sms(148, 2, 64, 6, 810.0) <= 148
    p = sms.send_probability(8, 256, 8)
    assert abs(p - (1 - math.comb(224, 8) / math.comb(256, 8))) < 1e-12
    assert sms.nvlink_gbs(("a",)) == 0.0
    assert sms.nvlink_gbs(("no-such-gpu-1", "no-such-gpu-2")) == 0.0  # nvidia-smi missing or GPUs unknown


def test_nvtx_range_is_a_shared_noop_when_disabled():
    from nanoep_b200.utils import tracing

    if not tracing._ENABLED:
        assert tracing.nvtx_range("a") is tracing.nvtx_range("b")
    with tracing.nvtx_range("anything"):
        pass


def _body(text, name):
    """Brace-matched body of the function whose definition starts at ``name(``."""
    start = text.index("{", text.index(f"{name}("))
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start : i + 1]
    raise AssertionError(name)


def test_receive_counts_follow_the_offsets_a_gated_consumer_reads():
    """A GEMM gated by tile counters runs on another stream and reads expert_offsets once the host has N and C, ordered by
    nothing but the mailbox: both planning kernels finish those tensors first and a gated dispatch fences in between."""
    text = re.sub(r"//[^\n]*", "", (ROOT / "csrc" / "ep_kernels.cu").read_text())
    publish = _body(text, "void publish_counts")
    assert re.search(r"if \(ordered\) __threadfence_system\(\);.*mailbox\[1\] = .*mailbox\[0\] = ", publish, re.S)
    assert set(re.findall(r"mailbox\[[01]\] = ([^;]+);", text.replace(publish, ""))) == {"-2"}, "only the failure code goes another way"
    for kernel in ("bool stage_body", "void local_plan_body"):
        body = _body(text, kernel)
        assert body.count("publish_counts(") == 1 and re.search(r"__syncwarp\(\);\s*if \(lane == 0[^)]*\) publish_counts\([^;]*p\.gated", body)
        after = body[body.index("publish_counts(") :]
        assert not re.search(r"p\.expert_(offsets|counts)\[[^\]]*\] = ", after), kernel
    host = (ROOT / "csrc" / "pipeline.cpp").read_text()
    assert re.search(r"gated = gated \|\| t\.has_value\(\);.*p\.gated = gated;.*lp\.gated = sp\.gated;", host, re.S)


def test_an_invalid_expert_id_is_reported_before_the_counts():
    """The call that follows a dispatch raises what the dispatch found, so the host sees the status word no later than N and C.
    In a group the peer barrier's system fence lies between; a single rank fences, in the one-launch plan when a CTA of its
    cluster reported."""
    text = re.sub(r"//[^\n]*", "", (ROOT / "csrc" / "ep_kernels.cu").read_text())
    body = _body(text, "void local_plan_body")
    assert re.search(r"report\(status, kBadExpertId[^;]*;\s*s_invalid = 1;", body)
    assert body.index("s_invalid = 1;") < body.index("cluster_wait();") < body.index("ld_cluster_smem(&s_invalid")
    assert re.search(r"publish_counts\([^;]*s_any_invalid", body)
    stage = _body(text, "bool stage_body")
    assert re.search(r"publish_counts\([^;]*R == 1", stage)
    assert stage.index("kBadExpertId") < stage.index("peer_barrier_warp(") < stage.index("publish_counts(")
    assert re.search(r"if \(R > 1\) \{\s*__threadfence_system\(\);\s*__syncthreads\(\);\s*if \(warp == 0\) \{\s*const bool ok = peer_barrier_warp", stage)


def test_cluster_barriers_ask_for_a_whole_warp_only_behind_a_block_barrier():
    """The `.aligned` cluster barrier needs every thread of a warp at the same instruction.  Lanes of the one-launch plan leave
    its loops at different points; the GEMM kernels reach theirs through __syncthreads()."""
    for path in _native_sources():
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"barrier\.cluster\.(arrive|wait)\.\w+\.aligned", text):
            assert path.name == "tc_prim.cuh" and "void cluster_sync" in text[max(0, m.start() - 250) : m.start()], path.name
        for m in re.finditer(r"\bcluster_sync\(\);", text):
            assert re.search(r"__syncthreads\(\);\s*$", text[: m.start()]), path.name


def test_gemm_kernels_clear_their_abort_flag_before_anyone_sets_it():
    """Every thread checks offsets and may set the flag; the thread that clears it must have done so before."""
    for name in ("grouped_gemm_sm100.cu", "grouped_gemm_sm100_2cta.cu", "expert_gemm_sm100.cu"):
        text = re.sub(r"//[^\n]*", "", (ROOT / "csrc" / name).read_text())
        assert "__syncthreads();" in text[text.index("sh.abort = 0;") : text.index("sh.abort = 1;")], name


def test_what_starts_early_reads_only_what_ended_kernels_wrote():
    """The expert GEMM reads offsets and counts in front of its wait for the previous kernel.  Behind a dispatch that is safe where
    the last kernel has not written them itself: the single-launch fresh dispatch has."""
    host, layer = (re.sub(r"//[^\n]*", "", (ROOT / "csrc" / name).read_text()) for name in ("pipeline.cpp", "gemm_bindings.cpp"))
    assert re.findall(r"out\.early = ([^;]+);", host) == ["behind && !fuse_fresh"]
    assert re.findall(r"\.dependents = ([^;]+);", host) == ["out.early"]
    assert host.index("const bool fuse_fresh =") < host.index("out.early =") < host.index("p.dependents =")
    body = _body(layer, "pybind11::tuple moe_forward")
    up = re.search(r"grouped_gemm\(rows, w13,[^;]*;", body).group(0)
    assert "got.early" in up and "true" not in up
    steps = (ROOT / "nanoep_b200" / "models" / "moe_layer.py").read_text()
    assert re.search(r"self\._grouped\(h_in, self\.w13,[^)]*, False\)", steps)


def test_a_unit_is_acknowledged_behind_its_read():
    """A relaxed arrival orders no read in front of it, and an operand that the statement does not use orders nothing: the address
    that the arrival goes to is computed from the value read."""
    text = re.sub(r"//[^\n]*", "", (ROOT / "csrc" / "expert_gemm_sm100.cu").read_text())
    assert text.count("mbarrier.arrive.relaxed") == 1
    body = _body(text, "void arrive_behind")
    assert re.search(r"(\w+) = \(uint32_t\(unit\) \+ 1u\) >> 31;.*_, \[%0\];\" *::\"r\"\(cluster_addr \+ 8u \* \1\)", body, re.S)
    # the value that is acknowledged is the one read from the slot
    assert re.search(r"next = \*\(volatile int\*\)&sh\.next_unit\[slot\];\s*arrive_behind\([^;]*, next\);", text)
