"""Performance cases of the framework: what its users have it do, through its public entry points.

Kinds of case:
  box    a zero-dimensional box model with Golovin's kernel: one member of an ensemble, uploaded,
         stepped and observed (the member's whole run, at 1 s steps);
  steps  a domain from its initial conditions to an observation: states and superdroplets
         uploaded, coupling steps of 1 s (motion, re-sort, condensation, collisions and breakup),
         the superdroplets gathered into pinned host memory in the output types and the
         condensation budgets read back (with options: condensation feeding back on the states,
         states uploaded and budgets read at every step, monitors, the Newton solves seeded by
         the surrogate, launch shapes autotuned);
  solve  implicit-Euler condensation steps of independent droplets held on the device;
  train  Adam steps of the condensation surrogate (forward and backward);
  infer  the surrogate's tensor-core inference;
  sort   the allocation-free stable sort of superdroplets by gridbox.

Populations have the shapes of cleo_b200.workloads; they are drawn on the GPU from the seed.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from cleo_b200 import abi
from cleo_b200 import workloads as W
from cleo_b200.config import (LLIM, MR0, Mr_ratio, Mr_sol, P0, R0, RHO0, Rho_sol, TEMP0,
                              TIME0, VOL0, cartesian_grid, make_params)
from cleo_b200.sdm import SDM, CleoError
from cleo_b200.surrogate import Surrogate, condensation_solve, train_surrogate

STEP = 100  # a coupling step in model steps of 0.01 s
TIGHT = dict(maxniters=200, rtol=0.0, atol=1e-8)
NORMAL = dict(maxniters=50, rtol=0.0, atol=0.01)
# converged roots, without the rounding noise that keeps a rare droplet iterating at TIGHT
CONVERGED = dict(maxniters=50, rtol=0.0, atol=1e-6)


def _box(n, steps):
    return dict(kind="box", n=n, steps=steps)


def _steps(flow, nz, nx, ny, steps, median=32.0, sigma=0.586, tight=False, seeded=False,
           coupled=False, monitors=False, tuned=False, feedback=False):
    return dict(kind="steps", flow=flow, nz=nz, nx=nx, ny=ny, steps=steps, median=median,
                sigma=sigma, tight=tight, seeded=seeded, coupled=coupled, monitors=monitors,
                tuned=tuned, feedback=feedback)


def listed():
    return [
        # the Golovin box model at its usual size: short kernels, launches count
        dict(_box(8192, 600), name="box_8k"),
        # the same model at the size of convergence studies
        dict(_box(131072, 60), name="box_131k"),
        # the 1-D rain shaft, 256 superdroplets in each of 256 gridboxes
        dict(_steps("column", 256, 1, 1, 60, median=256.0, sigma=0.0), name="shaft_256x256"),
        # a small 3-D domain (156 thousand superdroplets): latency and launches again
        dict(_steps("still", 16, 16, 16, 100, feedback=True), name="small_16x16x16"),
        # a ragged 3-D domain with all SDMMonitor members on, as for budgets of a rain event
        dict(_steps("still", 21, 45, 53, 60, monitors=True), name="monitored_21x45x53"),
        # the uneven 3-D workload with surrogate seeds at the tight tolerance
        dict(_steps("still", 32, 64, 64, 60, tight=True, seeded=True), name="seeded_32x64x64"),
        # the bubble flow driven by a host model: states up and budgets down at every step
        dict(_steps("bubble", 64, 64, 64, 20, median=16.0, sigma=0.9005, coupled=True),
             name="bubble_64x64x64"),
        # the uneven 3-D workload at its full size (40 million superdroplets), autotuned
        dict(_steps("still", 64, 128, 128, 40, tuned=True), name="uneven_64x128x128"),
        # independent condensation solves to converged roots, as training data is made
        dict(kind="solve", n=(1 << 21) + 77, name="solve_2M"),
        # a slice of the surrogate's training at its usual minibatch
        dict(kind="train", n=1 << 20, batch=8192, steps=64, name="train_64x8192"),
        # the trained surrogate evaluated on a population
        dict(kind="infer", n=4_000_037, name="infer_4M"),
        # a host model's own superdroplets sorted without allocations
        dict(kind="sort", n=1_000_003, ngbxs=32768, name="sort_1M"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "steps", "steps", "steps", "solve", "train", "infer", "sort"])
    if kind == "box":
        n = _log_int(rng, 1000, 200_000)
        return _box(n, max(20, min(600, 6_000_000 // n)))
    if kind == "solve":
        return dict(kind=kind, n=_log_int(rng, 5000, 1 << 21))
    if kind == "train":
        return dict(kind=kind, n=_log_int(rng, 1 << 14, 1 << 20), batch=128 * rng.randint(4, 96),
                    steps=rng.randint(20, 64))
    if kind == "infer":
        return dict(kind=kind, n=_log_int(rng, 2000, 8_000_000))
    if kind == "sort":
        return dict(kind=kind, n=_log_int(rng, 2000, 1_048_576), ngbxs=_log_int(rng, 20, 200_000))
    flow = rng.choice(["column", "still", "still", "bubble"])
    if flow == "column":
        return _steps(flow, rng.randint(50, 400), 1, 1, 30, sigma=0.0,
                      median=float(_log_int(rng, 40, 700)))
    nz = rng.randint(12, 64)
    nx = rng.randint(max(8, nz // 2), min(80, 2 * nz))
    ny = rng.randint(5, 70)
    opt = dict(median=16.0, sigma=0.9005) if flow == "bubble" else {}
    flag = lambda: rng.random() < 0.3  # noqa: E731
    return _steps(flow, nz, nx, ny, rng.randint(20, 60), coupled=flag(), monitors=flag(),
                  tuned=flag(), feedback=flag(), **opt)


# ------------------------------------------------------------------------------------------
# populations
# ------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(n, lo, hi, gen):
    return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)


def _dry_radii(n, gen):
    z = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
    return (math.log(0.02) + math.log(1.5) * z).exp().clamp(1e-3, 10.0)


def _msol(rdry):
    return rdry ** 3 * (4.0 * math.pi / 3.0) * Rho_sol


def _kohler(msol, temp):
    return ((3.3e-7 / (TEMP0 * R0)) / temp, (4.3e-6 * RHO0 / MR0) * msol * 2.0 / Mr_sol)


def _equilibrium(rdry, msol, s_ratio, temp):
    """Stable Kohler equilibrium radii, at most just below the critical supersaturation."""
    a, b = _kohler(msol, temp)
    scrit = 1.0 + torch.sqrt(4.0 * a ** 3 / (27.0 * b))
    sm1 = torch.minimum(s_ratio, 1.0 + 0.999 * (scrit - 1.0)) - 1.0
    lo = rdry * (1.0 + 1e-9)
    hi = torch.maximum(torch.sqrt(3.0 * b / a), lo)
    for _ in range(44):
        mid = 0.5 * (lo + hi)
        up = b / (mid * mid * mid) - a / mid + sm1 > 0.0
        lo = torch.where(up, mid, lo)
        hi = torch.where(up, hi, mid)
    return torch.maximum(0.5 * (lo + hi), rdry)


def _domain(case, seed):
    """Grid, states and superdroplets of a steps case (pinned host arrays). The gridboxes'
    counts belong to the case; all else is drawn from the seed."""
    rng = np.random.default_rng(seed)
    gen = _gen(seed)
    column = case["flow"] == "column"
    volume = 8000.0 if column else (25.0 if case["flow"] == "bubble" else 50.0)
    d = volume ** (1.0 / 3.0)
    grid = cartesian_grid((case["nz"], case["nx"], case["ny"]), (d, d, d),
                          nspacedims=1 if column else 3)
    zc = (np.arange(grid["ngbxs"]) % case["nz"] + 0.5) * d
    temp, press, qvap, _ = W.column_thermo(zc, rng)
    wind = W.divfree_flow(grid) if case["flow"] == "bubble" else (None, None)
    state = W.make_state(grid["ngbxs"], volume / VOL0, temp, press, qvap, w=wind[0], u=wind[1])
    s_ratio = press * qvap / ((Mr_ratio + qvap) * W.psat_dimless(temp))
    counts = W.lognormal_counts(grid["ngbxs"], np.random.default_rng(11), case["median"],
                                case["sigma"])
    n = int(counts.sum())
    g = torch.repeat_interleave(torch.arange(grid["ngbxs"], device="cuda"),
                                torch.from_numpy(counts).cuda())
    on_gpu = {k: torch.from_numpy(v).cuda() for k, v in (("T", temp), ("s", s_ratio))}
    supers = {"sdgbxindex": g.to(torch.int32), "sdid": torch.arange(n, device="cuda")}
    for c in ("coord3", "coord1", "coord2"):
        lo = torch.from_numpy(grid[c + "lo"]).cuda()[g]
        hi = torch.from_numpy(grid[c + "hi"]).cuda()[g]
        x = torch.minimum(lo + torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
                          * (hi - lo), torch.nextafter(hi, lo))
        supers[c] = torch.where(lo == LLIM, torch.zeros_like(x), x)
    rdry = _dry_radii(n, gen)
    msol = _msol(rdry)
    supers["msol"] = msol
    supers["radius"] = _equilibrium(rdry, msol, on_gpu["s"][g], on_gpu["T"][g])
    xi = np.maximum(1, np.round(1.325e9 * volume / np.maximum(counts, 1))).astype(np.int64)
    supers["xi"] = torch.from_numpy(xi).cuda()[g]
    types = dict(abi.SUPERS_FIELDS)
    supers = {k: torch.empty(n, dtype=v.dtype, pin_memory=True).copy_(v).numpy().view(types[k])
              for k, v in supers.items()}
    state = {k: torch.from_numpy(v).pin_memory().numpy() for k, v in state.items()}
    return grid, state, supers


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def _droplets(n, seed):
    """Independent droplets for condensation solves, as workloads.condsolve draws them."""
    gen = _gen(seed)
    rdry = _dry_radii(n, gen)
    low = rdry.clamp(min=0.01).log()
    r = (low + _uniform(n, 0.0, 1.0, gen) * (math.log(100.0) - low)).exp()
    delt = torch.tensor([0.5, 1.0, 2.0], dtype=torch.float64, device="cuda") / TIME0
    return dict(radius=torch.maximum(r, rdry), msol=_msol(rdry),
                temp=_uniform(n, 250.0, 305.0, gen) / TEMP0,
                press=_uniform(n, 50e3, 101e3, gen) / P0,
                s_ratio=1.0 + _uniform(n, -0.05, 0.02, gen),
                delt=delt[torch.randint(0, 3, (n,), device="cuda", generator=gen)])


def _weights(seed):
    """A surrogate's parameters (Glorot-uniform) as float32."""
    rng = np.random.default_rng([7, seed])
    uni = lambda fan, *shape: rng.uniform(-1, 1, shape) * math.sqrt(6.0 / fan)  # noqa: E731
    return np.concatenate([uni(71, 64 * 7), np.zeros(64), uni(128, 64 * 64), np.zeros(64),
                           uni(65, 64), np.zeros(1)]).astype(np.float32)


def _features(d):
    a, b = _kohler(d["msol"], d["temp"])
    x = (torch.log(d["radius"]), torch.log(d["msol"]), d["s_ratio"] - 1.0, d["temp"], d["press"],
         d["delt"], torch.log(3.0 * b / a))
    return torch.stack(x, dim=1).float().contiguous()


def _normalisation(feats, target):
    f, t = feats.double(), target.double()
    out = torch.cat([f.mean(0), 1.0 / f.std(0), t.mean()[None], t.std()[None]])
    return out.float().cpu().numpy()


def _training_pairs(n, seed):
    """Features and targets of n droplets whose solve needs no sub-steps."""
    d = _droplets(int(3.6 * n) + 4096, seed)
    direct = torch.nonzero(_implicit_euler(d, 0.001 / TIME0, branch_only=True))[:n, 0]
    assert direct.numel() == n
    d = {k: v[direct] for k, v in d.items()}
    r, _ = _implicit_euler(d, 0.001 / TIME0)
    return _features(d), (2.0 * torch.log(r / d["radius"])).float()


def _settled(d, ok, n):
    """The first n droplets whose solve converged (a droplet in a million's does not, and CLEO
    aborts on it)."""
    keep = torch.nonzero(ok)[:n, 0]
    return {k: v[keep] for k, v in d.items()}


# ------------------------------------------------------------------------------------------
# the calls
# ------------------------------------------------------------------------------------------
_TRAINED = []


def _trained_surrogate():
    """A surrogate trained once per process, as a user's program loads or trains one."""
    if not _TRAINED:
        solver = _solver()
        sur, _ = train_surrogate(solver, n_pairs=1 << 18, steps=2000, chunk=1 << 20)
        _TRAINED.append(sur)
    return _TRAINED[0]


def _solver():
    grid = cartesian_grid((1, 1, 1), (100.0, 100.0, 100.0), nspacedims=0)
    return SDM(make_params(condtstep=1.0, **CONVERGED), grid, 1)


def _output(n):
    """Pinned host arrays of one observation and the C structure over them."""
    dt = {np.uint32: torch.int32, np.uint64: torch.int64, np.float32: torch.float32}
    out = {v: _pinned(n, dt[t]) for v, (_, t) in abi.OBS_VARS.items()}
    return out, abi.obs_struct({v: out[v].numpy().view(t) for v, (_, t) in abi.OBS_VARS.items()})


def prepare(case, seed):
    kind, lib = case["kind"], abi.load_library()
    if kind == "box":
        w = W.box_golovin(n_sd=case["n"], seed=seed)
        sdm = SDM(w["params"], w["grid"], case["n"])
        sdm.upload_state(w["state"])
        out, struct = _output(case["n"])
        return dict(case=case, sdm=sdm, supers=w["supers"], out=out, struct=struct)
    if kind == "steps":
        grid, state, supers = _domain(case, seed)
        column = case["flow"] == "column"
        params = make_params(
            condtstep=1.0, colltstep=1.0, motiontstep=1.0, minsubtstep=0.001,
            coll_prob=abi.PROB_LONG, seed=seed, motion_tv=abi.TV_ROGERSGK,
            coll_enact=abi.ENACT_COALESCENCE if column else abi.ENACT_COALBURE,
            nfrags_kind=abi.NFRAGS_CONST, nfrags=5.0, flag_kind=abi.FLAG_STRAUB,
            flag_tv=abi.TV_ROGERSGK, monitors=7 if case["monitors"] else 0,
            do_alter_thermo=case["feedback"],
            nr_seed=abi.NRSEED_MLP if case["seeded"] else abi.NRSEED_REFERENCE,
            **(TIGHT if case["tight"] else NORMAL))
        n = len(supers["xi"])
        sdm = SDM(params, grid, n)
        s = dict(case=case, sdm=sdm, n=n, state=state, supers=supers)
        s["out"], s["struct"] = _output(n)
        if case["coupled"]:
            s["mass"] = _pinned(grid["ngbxs"], torch.float64).numpy()
            s["iters"] = _pinned(grid["ngbxs"], torch.int64).numpy().view(np.uint64)
        if case["seeded"]:
            s["model"] = _trained_surrogate()
            assert lib.cleo_b200_set_surrogate(sdm.ctx, s["model"].handle) == 0
        if case["tuned"]:
            sdm.upload_state(state)
            sdm.upload_supers(supers)
            assert lib.cleo_b200_autotune(sdm.ctx, 2) == 0
            for k in range(8):
                sdm.run_step(k * STEP, (k + 1) * STEP)
            sdm.check()
        return s
    if kind == "solve":
        sdm, d = _solver(), _droplets(case["n"] + 512, seed)
        _, niters = condensation_solve(sdm, d, allow=("CLEO_ERR_NR_NOCONVERGE",))
        lib.cleo_b200_clear_status(sdm.ctx)
        return dict(case=case, sdm=sdm, inputs=_settled(d, niters >= 0, case["n"]))
    if kind == "sort":
        n, ng = case["n"], case["ngbxs"]
        gen = _gen(seed)
        g = torch.sort(torch.randint(0, ng, (n,), device="cuda", generator=gen))[0]
        # after a motion step: a few have crossed into a neighbour, some left at the bottom
        move = torch.rand(n, device="cuda", generator=gen)
        g = torch.where(move < 0.05, g - 1, g)
        g = torch.where((move < 0.001) | (g < 0), torch.full_like(g, 0x7FFFFFFF), g)
        assert lib.cleo_b200_sort_by_gridbox_static(None, 0, 0, None, None, None) == 0
        new = lambda k: torch.empty(k, dtype=torch.int32, device="cuda")  # noqa: E731
        return dict(case=case, keys=g.to(torch.int32), order=new(n), start=new(ng + 2), lib=lib)
    sur = Surrogate(seed=1)
    if kind == "train":
        feats, target = _training_pairs(case["n"], seed)
        sur.set_params(_weights(seed), _normalisation(feats, target))
        return dict(case=case, model=sur, feats=feats, target=target)
    feats = _features(_droplets(case["n"], seed))
    sur.set_params(_weights(seed), _normalisation(feats, 0.1 * feats[:, 0]))
    return dict(case=case, model=sur, feats=feats)


def _observe(s, cap):
    n = C.c_size_t()
    sdm = s["sdm"]
    rc = sdm.lib.cleo_b200_gather_supers(sdm.ctx, abi.OBS_ALL, C.byref(s["struct"]), cap,
                                         C.byref(n))
    if rc != 0:
        raise CleoError(rc, where="in gather_supers")
    return {**s["out"], "count": n.value}


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "box":
        s["sdm"].upload_supers(s["supers"])
        for k in range(case["steps"]):
            s["sdm"].run_step(k * STEP, (k + 1) * STEP)
        return _observe(s, case["n"])
    if kind == "steps":
        sdm = s["sdm"]
        sdm.upload_state(s["state"])
        sdm.upload_supers(s["supers"])
        if case["monitors"]:
            sdm.monitors_begin()
        for k in range(case["steps"]):
            if case["coupled"]:
                sdm.upload_state_async(s["state"])
            sdm.run_step(k * STEP, (k + 1) * STEP)
            if case["coupled"]:
                sdm.download_budgets_async(s["mass"], s["iters"])
        out = _observe(s, s["n"])
        if case["coupled"]:
            sdm.synchronize()
            mass, iters = s["mass"], s["iters"]
        else:
            mass, iters = sdm.download_budgets()
        out["condensed_mass"] = mass
        # with a surrogate the iterations tell how good its seeds are, not what was solved
        if not case["seeded"]:
            out["newton_iterations"] = iters.view(np.int64)
        if case["monitors"]:
            mon = sdm.download_monitors(reset=True)
            out["monitors"] = {k: v.view(np.int64) if v.dtype == np.uint64 else v
                               for k, v in mon.items()}
        return out
    if kind == "solve":
        r, niters = condensation_solve(s["sdm"], s["inputs"])
        return {"radius": r, "iterations": niters}
    if kind == "train":
        loss = s["model"].train(s["feats"], s["target"], steps=case["steps"], batch=case["batch"])
        return {"params": s["model"].get_params()[0], "loss": loss}
    if kind == "infer":
        return s["model"].infer(s["feats"])
    p = [C.c_void_p(s[k].data_ptr()) for k in ("keys", "order", "start")]
    rc = s["lib"].cleo_b200_sort_by_gridbox_static(
        p[0], case["n"], case["ngbxs"], p[1], p[2],
        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise CleoError(rc, where="in sort_by_gridbox_static")
    return {"order": s["order"], "start": s["start"]}


def work(case):
    """Bytes: every superdroplet's 60 bytes read and written once a step (collisions put each
    gridbox in a new order), uploaded once (60) and read once into 36 bytes of output."""
    kind = case["kind"]
    if kind == "box":
        return dict(bytes=case["n"] * (120.0 * case["steps"] + 96.0 + 60.0),
                    flops=case["n"] * case["steps"] * 20.0)
    if kind == "steps":
        n = case["nz"] * case["nx"] * case["ny"] * case["median"] * math.exp(case["sigma"] ** 2 / 2)
        # motion, two Newton iterations and a pair's probability: some 200 operations
        return dict(bytes=n * (120.0 * case["steps"] + 156.0), flops=n * case["steps"] * 200.0)
    n = case["n"]
    if kind == "solve":  # 68 Newton iterations in the mean, about 30 operations each
        return dict(bytes=n * 60.0, flops=n * 68.0 * 30.0)
    if kind == "train":
        rows = float(case["batch"] * case["steps"])
        return dict(bytes=rows * 32.0 + 4 * 4737, flops=rows * 6 * 4608)
    if kind == "infer":
        return dict(bytes=n * 32.0, flops=n * 2.0 * 4608)
    return dict(bytes=n * 8.0 + (case["ngbxs"] + 2) * 4.0, flops=0.0)


# ------------------------------------------------------------------------------------------
# the same in 64 bits, with torch and numpy alone
# ------------------------------------------------------------------------------------------
def _implicit_euler(d, minsubdelt, branch_only=False):
    """One implicit-Euler condensation step of each droplet: the radii and whether Newton's
    iterations converged; with branch_only, whether each step is taken without sub-steps."""
    r, T, s = d["radius"], d["temp"] * TEMP0, d["s_ratio"]
    latent, rgas_v, rho_l = 2500930.0, 8.314462618 / 0.01801528, 998.203 / RHO0
    f0 = TIME0 / (RHO0 * R0 * R0)
    psat = 611.655 * torch.exp(17.4146 * (T - 273.16) / (T - 33.639))
    thermk = 7.11756e-5 * T * T + T * 4.38127686e-3
    diffuse = 4.012182971e-5 / (d["press"] * P0) * T ** 1.94 / rgas_v
    ff = rho_l * ((latent / rgas_v / T - 1.0) * latent / (thermk * f0) + T / (diffuse * psat) / f0)
    vent = 1.0 + 1.0 / (1.0 / (6.954e7 * (r * R0) ** 1.963) + 1.0 / (1.069e3 * (r * R0) ** 0.702))
    ff = ff / vent.clamp(max=20.0)
    a, b = _kohler(d["msol"], d["temp"])
    s_act = 1.0 + torch.sqrt(4.0 * a ** 3 / 27.0 / b)
    z = torch.where(s > s_act, torch.clamp(r, min=1e-3 / R0) ** 2, r * r)
    rcrit2 = 3.0 * b / a
    crit = 2.5 * ff / a * (5.0 * b / a) ** 1.5
    direct = ((r * r < rcrit2) & (z < rcrit2) & (s <= s_act)) | (d["delt"] <= crit)
    if branch_only:
        return direct
    whole = torch.where(direct, d["delt"], torch.clamp(crit, min=minsubdelt))
    out, ok = torch.empty_like(r), torch.ones_like(direct)
    live = torch.arange(r.numel(), device=r.device)
    prev, left, sm1 = r.clone(), d["delt"].clone(), s - 1.0

    def residual(w, p2, h, sm1, a, b, f):  # g and its derivative times w
        q = torch.sqrt(w)
        aq, bq, hf = a / q, b / (q * w), h / (w * f)
        return 1.0 - p2 / w - 2.0 * hf * (sm1 - aq + bq), 1.0 - hf * (aq - 3.0 * bq)

    while live.numel():  # a sub-step of every droplet that has time left
        dt = torch.minimum(whole, left)
        args, w = (prev * prev, dt, sm1, a, b, ff), z
        before, slope = residual(w, *args)
        open_ = torch.ones_like(w, dtype=torch.bool)
        for it in range(CONVERGED["maxniters"]):
            new = torch.clamp(w * (1.0 - before / slope), min=1e-8)
            w = torch.where(open_, new, w)
            after, slope = residual(w, *args)
            if it >= 1:
                open_ = open_ & ((after - before).abs() >= CONVERGED["atol"])
                if not open_.any():
                    break
            before = after
        z = w
        ok[live[open_]] = False
        prev = torch.sqrt(z)
        left = left - dt
        done = (left <= 0.0) | open_
        if done.any():
            out[live[done]] = prev[done]
            keep = ~done
            live, z, prev, left, whole, sm1, a, b, ff = (
                v[keep] for v in (live, z, prev, left, whole, sm1, a, b, ff))
    rdry = (3.0 / (4.0 * math.pi) * d["msol"] / Rho_sol) ** (1.0 / 3.0)
    return torch.maximum(out, rdry), ok


def _mix64(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _minibatch(seed, step, batch, n):
    """The samples of a training step: counter-based draws from [0, n)."""
    golden = np.uint64(0x9E3779B97F4A7C15)
    with np.errstate(over="ignore"):
        key = _mix64(_mix64(np.uint64(seed) + golden) ^ np.uint64((step << 32) | 0x4D4C50))
        u = _mix64(key + (np.arange(batch, dtype=np.uint64) + np.uint64(1)) * golden)
    low = ((u & np.uint64(0xFFFFFFFF)) * np.uint64(n)) >> np.uint64(32)
    return (((u >> np.uint64(32)) * np.uint64(n) + low) >> np.uint64(32)).astype(np.int64)


def _unpack(p):
    w1, b1, w2, b2, w3, b3 = torch.split(p, [448, 64, 4096, 64, 64, 1])
    return w1.view(64, 7), b1, w2.view(64, 64), b2, w3, b3


def _network(p, x):
    w1, b1, w2, b2, w3, b3 = _unpack(p)
    gelu = torch.nn.functional.gelu
    return gelu(gelu(x @ w1.T + b1) @ w2.T + b2) @ w3 + b3


def exact(case, seed):
    """None for box and steps: a whole engine's random collisions."""
    kind = case["kind"]
    if kind == "solve":
        d = _droplets(case["n"] + 512, seed)
        d["r"], ok = _implicit_euler(d, 0.001 / TIME0)
        return {"radius": _settled(d, ok, case["n"])["r"], "iterations": None}
    if kind == "infer":  # BF16 weights, as the model holds them
        feats = _features(_droplets(case["n"], seed))
        norm = torch.from_numpy(_normalisation(feats, 0.1 * feats[:, 0])).cuda().double()
        p = torch.from_numpy(_weights(seed)).cuda()
        for part in (slice(0, 448), slice(512, 4608), slice(4672, 4736)):
            p[part] = p[part].bfloat16().float()
        return torch.cat([norm[14] + norm[15] * _network(p.double(), (x.double() - norm[:7])
                                                          * norm[7:14])
                          for x in feats.split(1 << 20)])
    if kind != "train":
        return None
    feats, target = _training_pairs(case["n"], seed)
    norm = torch.from_numpy(_normalisation(feats, target)).cuda().double()
    p = torch.from_numpy(_weights(seed)).cuda().double().requires_grad_()
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    steps, warm = case["steps"], case["steps"] // 50 + 1
    for k in range(steps):
        idx = torch.from_numpy(_minibatch(1, k, case["batch"], case["n"])).cuda()
        x = (feats[idx].double() - norm[:7]) * norm[7:14]
        t = (target[idx].double() - norm[14]) / norm[15]
        loss = ((_network(p, x) - t) ** 2).mean()
        g, = torch.autograd.grad(loss, p)
        lr = 2e-3 * (0.02 + 0.98 * 0.5 * (1.0 + math.cos(math.pi * k / steps)))
        lr *= min(1.0, (k + 1) / warm)
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        with torch.no_grad():
            p -= lr * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
        losses.append(loss.detach())
    return {"params": p.detach(), "loss": torch.stack(losses)}
