"""Dispatch and combine on one GPU at the sizes where a kernel's split changes: edges of waves, tiles and launch shapes.

Everything is compared with the CPU oracle bit for bit."""

import pytest
import torch

from nanoep_b200 import EmulatedGroup, EPConfig
from nanoep_b200.testing.cases import make_case
from nanoep_b200.testing.checks import assert_dispatch_matches

pytestmark = pytest.mark.gpu


def _cuda(ts):
    return [t.cuda() for t in ts]


@pytest.mark.parametrize("world", [1, 2])
@pytest.mark.parametrize("experts_per_rank", [31, 33, 257])
@pytest.mark.parametrize("alignment", [1, 3, 128])
def test_padding_rows_of_many_experts(world, experts_per_rank, alignment):
    """Gap rows are numbered 32 experts at a time, eight such waves per pass; rows longer than the zero source."""
    case = make_case(world, kind="mixed", seed=experts_per_rank, hidden=8192, tokens=19, experts_per_rank=experts_per_rank, topk=4)
    cfg = EPConfig(case.num_experts, case.num_topk, case.hidden, case.capacity)
    with EmulatedGroup(world, cfg) as group:
        first = group.dispatch(_cuda(case.xs), topk_idx=_cuda(case.indices), weights=_cuda(case.weights), do_expand=True, alignment=alignment,
                               zero_padding=True)
        again = group.dispatch(_cuda(case.xs), handles=[f.handle for f in first], weights=_cuda(case.weights), zero_padding=True)
        torch.cuda.synchronize()
        group.check_status()
        for got in (first, again):
            for r in range(world):
                assert_dispatch_matches(got[r], case.xs, case.indices, case.weights, case.num_experts, r, expand=True, alignment=alignment,
                                        zero_padding=True)
