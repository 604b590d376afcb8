"""Lines between two forms of a kernel: the same results beside them, and no call just below a line
slower than the larger one just above it (by more than a seventh, for noise)."""
import statistics
import time

import pytest

import checkers as K
from cleo_b200 import abi, workloads as W
from cleo_b200.sdm import make_sdm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return abi.load_library()


def _fastest(call, reps):
    import torch
    times = []
    for _ in range(reps):
        torch.cuda.synchronize()
        t = time.perf_counter()
        call()
        torch.cuda.synchronize()
        times.append(time.perf_counter() - t)
    return statistics.median(times[2:])


@pytest.mark.parametrize("n", [15935, 15936, 15937])
def test_one_box_beside_its_line(lib, n):
    """A store of 16,000 slots (64 of them free), one less and one more."""
    w = W.box_golovin(n_sd=n, seed=n)
    w["params"].exec_mode = abi.EXEC_BATCHED
    g, o = make_sdm(w, lib=lib), make_sdm(w, lib=K.oracle_lib(cr=True), prefix="oc")
    for k in range(4):
        for s in (g, o):
            s.run_step(k * w["tstep"], (k + 1) * w["tstep"])
    g.check()
    K.assert_identical_run(g, o, f"one box of {n}")


@pytest.mark.parametrize("below,above", [(15900, 16100), (27900, 28100)])
def test_one_box_no_slower_below_a_line(lib, below, above):
    def step(n):
        w = W.box_golovin(n_sd=n, seed=1)
        s = make_sdm(w, lib=lib)
        t = [0]

        def steps():
            for _ in range(100):
                s.run_step(t[0], t[0] + w["tstep"])
                t[0] += w["tstep"]
        return _fastest(steps, 9)
    assert step(below) < step(above) * 7 / 6


def test_a_smaller_box_beside_a_larger_one(lib):
    """Members of an ensemble in one process: a later, smaller one leaves the larger one's
    shared-memory limit alone."""
    w = [W.box_golovin(n_sd=n, seed=n) for n in (15000, 500)]
    runs = [make_sdm(x, lib=lib) for x in w]
    for k in range(2):
        for x, s in zip(w, runs):
            s.run_step(k * x["tstep"], (k + 1) * x["tstep"])
    for x, s in zip(w, runs):
        s.check()
        o = make_sdm(x, lib=K.oracle_lib(cr=True), prefix="oc")
        for k in range(2):
            o.run_step(k * x["tstep"], (k + 1) * x["tstep"])
        K.assert_identical_run(s, o, "ensemble")


def _static_sort(lib, n, ngbxs):
    import ctypes as C
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    keys = torch.randint(0, ngbxs + 2, (n,), dtype=torch.int32, device="cuda", generator=gen)
    order = torch.empty_like(keys)

    def call():
        assert lib.cleo_b200_sort_by_gridbox_static(
            C.c_void_p(keys.data_ptr()), n, ngbxs, C.c_void_p(order.data_ptr()), None,
            C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    return call, keys, order


@pytest.mark.parametrize("ngbxs", [200, 20000, 200000])
@pytest.mark.parametrize("n", [8191, 8192, 8193, 16384, 16385])
def test_static_sort_beside_its_line(lib, n, ngbxs):
    import torch
    call, keys, order = _static_sort(lib, n, ngbxs)
    call()
    expect = torch.sort(keys.clamp(max=ngbxs), stable=True)[1]
    assert torch.equal(order.long(), expect)


@pytest.mark.parametrize("below,above", [(8192, 8193), (16384, 16385)])
def test_static_sort_no_slower_below_a_line(lib, below, above):
    def sorts(n):
        call = _static_sort(lib, n, 200000)[0]
        return _fastest(lambda: [call() for _ in range(100)], 15)
    assert sorts(below) < sorts(above) * 7 / 6
