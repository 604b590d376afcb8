"""Device memory of a context: the shuffles' words (BatchScratch::perm) are sized by the gridboxes
that can hold superdroplets, 64 bytes each and 128 for those of more than 64, and only the batched
schedule has them."""
import gc

import pytest

from cleo_b200 import abi
from cleo_b200.config import cartesian_grid, make_params
from cleo_b200.sdm import SDM

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _created(grid, capacity, mode):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    p = make_params(condtstep=1.0, colltstep=1.0, motiontstep=1.0, exec_mode=mode)
    gc.collect()  # contexts that earlier tests left behind
    before = torch.cuda.mem_get_info()[0]
    s = SDM(p, grid, capacity, lib=abi.load_library())
    used = before - torch.cuda.mem_get_info()[0]
    s.close()
    return used


def test_shuffle_words_follow_what_the_domain_can_hold():
    _created(cartesian_grid((4, 4, 4), (1.0, 1.0, 1.0)), 10, abi.EXEC_BATCHED)
    grid = cartesian_grid((64, 128, 128), (1.0, 1.0, 1.0))
    ng = grid["ngbxs"]
    # allocations come in steps of 2 MiB: one for each of the two arrays, at most
    few = 1000
    assert (_created(grid, few, abi.EXEC_BATCHED) - _created(grid, few, abi.EXEC_PLAIN)
            <= 4 * MIB)
    # an empty domain: its maps, states, budgets and free slots came to 628 bytes a gridbox before
    # there were shuffles in memory; 16 MiB for rounding
    assert _created(grid, few, abi.EXEC_PLAIN) <= 628 * ng + 16 * MIB
    many = 1 << 24
    assert (_created(grid, many, abi.EXEC_BATCHED) - _created(grid, many, abi.EXEC_PLAIN)
            <= 64 * ng + 128 * (many // 65) + 4 * MIB)
