"""Sizes at which the sorts, the solve ordering and the ordered sums change their launches, against
numpy, the plain schedule and the correctly rounded oracle: all results equal bit for bit (whole
numbers, or the same double operations in the same order)."""
import ctypes as C

import numpy as np
import pytest

import checkers as K
from cleo_b200 import abi, workloads as W
from cleo_b200.config import make_params
from cleo_b200.sdm import SDM, make_sdm
from cleo_b200.surrogate import condensation_solve, to_device
from test_monitors import run_monitored

pytestmark = pytest.mark.gpu

TILE = 4096


@pytest.fixture(scope="module")
def lib():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return abi.load_library()


@pytest.mark.parametrize("n,ngbxs,in_place,starts", [
    (1, 1, False, True), (255, 254, True, True), (4 * TILE - 1, 255, False, False),
    (4 * TILE, 256, True, True), (4 * TILE + 1, 255, True, True), (4 * TILE + 1, 65536, False, True),
    (64 * TILE, 65535, False, True), (64 * TILE + 1, 1 << 24, False, False),
    (70 * TILE + 5, 200, True, True), (1 << 20, 40000, False, True)])
def test_static_sort_at_its_edges(lib, n, ngbxs, in_place, starts):
    """One block or passes over tiles, two launches a pass or more, one to four passes; the order
    written over the input; no gridbox starts wanted."""
    import torch
    rng = np.random.default_rng(n)
    keys = rng.integers(0, ngbxs + 3, n).astype(np.uint32)  # some at and past the domain's end
    keys[rng.random(n) < 0.02] = abi.OOB
    dev = torch.tensor(keys.view(np.int32), device="cuda")
    order = dev if in_place else torch.full((n,), -1, dtype=torch.int32, device="cuda")
    gstart = torch.full((ngbxs + 2,), -1, dtype=torch.int32, device="cuda") if starts else None
    torch.cuda.synchronize()
    assert lib.cleo_b200_sort_by_gridbox_static(
        C.c_void_p(dev.data_ptr()), n, ngbxs, C.c_void_p(order.data_ptr()),
        C.c_void_p(gstart.data_ptr()) if starts else None,
        C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    capped = np.minimum(keys, ngbxs)
    expect = np.argsort(capped, kind="stable")
    assert np.array_equal(order.cpu().numpy().view(np.uint32), expect)
    if starts:
        assert np.array_equal(gstart.cpu().numpy(),
                              np.searchsorted(capped[expect], np.arange(ngbxs + 2)))


@pytest.mark.parametrize("n", [1, 33, 1023, 1025, 20000])
def test_long_restarts_beside_short_ones(lib, n):
    """Direct solves whose second iterate lies at the floor restart far below the root: they are
    placed behind the other restarts."""
    w = W.condsolve(n, seed=n)
    rng = np.random.default_rng(n)
    small = rng.random(n) < 0.4
    w["radius"][small] = np.maximum(w["rdry"][small] * rng.uniform(1.0, 3.0, small.sum()), 0.02)
    w["s_ratio"][small] = rng.uniform(0.2, 0.9, small.sum())
    p = make_params(condtstep=1.0, maxniters=200, rtol=0.0, atol=1e-8)
    rc, r, its = K.condsolve(K.oracle_lib(cr=True), "oc", p, w)
    assert rc == 0
    s = SDM(p, W.cartesian_grid((1, 1, 1), (1.0, 1.0, 1.0), nspacedims=0), 1, lib=lib)
    out, nit = condensation_solve(s, to_device(w))
    assert np.array_equal(out.cpu().numpy().view(np.uint64), r.view(np.uint64))
    assert np.array_equal(nit.cpu().numpy().astype(np.uint32), its)
    if n > 1000:  # both kinds are there
        assert (its > 24).sum() > n // 50 and (its < 12).sum() > n // 4
    s.close()


def test_many_movers_where_few_were_expected(lib):
    """Two still steps, then winds that move tens of thousands of superdroplets in one step: the
    page re-sort has launched the one-block sort alone and takes them in it."""
    w = W.bubble3d(ndims=(16, 40, 25), seed=5)
    w["params"].motion_tv = abi.TV_NULL
    still = dict(w["state"])
    winds = [f for f in abi.STATE_FIELDS if "vel_" in f]
    for f in winds:
        still[f] = np.zeros_like(still[f])
    runs = []
    oracle = K.oracle_lib(cr=True)
    K.oracle_threads(oracle)
    before = None
    for library, prefix in ((lib, "cleo_b200"), (oracle, "oc")):
        s = make_sdm(w, lib=library, prefix=prefix)
        s.upload_state(still)
        for k in range(5):
            if k == 3:
                before = s.download_supers()
                st = s.download_state()
                for f in winds:
                    st[f] = w["state"][f]
                s.upload_state(st)
            s.run_step(k * w["tstep"], (k + 1) * w["tstep"])
            if k == 3:
                after = s.download_supers()
                a = np.zeros(int(before["sdid"].max()) + 1, dtype=np.int64)
                b = np.zeros_like(a)
                a[before["sdid"]] = before["sdgbxindex"]
                b[after["sdid"]] = after["sdgbxindex"]
                assert (a != b).sum() > 20000
        s.check()
        runs.append(s)
    K.assert_identical_run(*runs, "many movers")


@pytest.mark.parametrize("ndims", [(10, 25, 40), (16, 40, 50)])
def test_ordered_sums_by_a_few_gridboxes_a_warp(lib, ndims):
    """Two and four gridboxes a warp (one on smaller domains, 32 on large ones), with a remainder."""
    w = W.uneven3d(ndims=ndims, seed=6, median=10.0)
    g, mg = run_monitored(lib, "cleo_b200", w, 2)
    oracle = K.oracle_lib(cr=True)
    K.oracle_threads(oracle)
    o, mo = run_monitored(oracle, "oc", w, 2)
    K.assert_identical_run(g, o, "sums")
    for f, _ in abi.MONITOR_FIELDS:
        assert np.array_equal(mg[-1][f], mo[-1][f], equal_nan=mg[-1][f].dtype.kind == "f"), f
