"""The expert sort in each of its forms (ids kept by their threads, or read twice)."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,experts,width", [(1024, 2, torch.int32), (1025, 8192, torch.int64), (4097, 60, torch.int32),
                                                 (16384, 128, torch.int64), (16384, 8192, torch.int32),
                                                 (16385, 8, torch.int32), (50001, 300, torch.int64),
                                                 (2048, 31, torch.int32), (2049, 31, torch.int64), (4096, 32, torch.int32),
                                                 (6144, 32, torch.int64), (6145, 32, torch.int32), (6145, 31, torch.int64)])
def test_expert_sort_at_the_edges_of_its_forms(slots, experts, width):
    from test_pair_gemm_gpu import test_moe_sort_lists_every_valid_slot_once as lists_every_slot_once

    lists_every_slot_once(slots, experts, width)
