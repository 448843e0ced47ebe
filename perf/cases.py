"""The work that users of das_gb300 have it do, as measurable cases.

Kinds (``case["kind"]``), each through the public entry point a program calls:

* ``model``     WaveSolver2D.forward_propagate_acoustic: modelling of an observed gather
* ``shot``      TSWRTMEngine.migrate_shot: forward with illumination, backward with imaging
* ``survey``    TSWRTMEngine.migrate_multiple_shots: every shot of a line, stacked and filtered
* ``batch``     BatchEngine.run: uneven virtual-source gathers admitted by memory budget
* ``gradient``  autograd.model_traces and its backward: acoustic velocity gradient
* ``elastic``   elastic.elastic_traces and its backward: shear-velocity gradient
* ``stack``     CrossCorrelationStack: noise windows correlated for many virtual sources
* ``gather``    compute_cross_correlation .. resample_gather_to_sim_dt: one virtual gather

Sizes are those of the benchmark configurations (150 x 400 and 1000 x 4000 acoustic grids,
uneven 200-600 x 400-2000 gathers, the 1024 x 2048 elastic grid, 3000-sample windows of 600
channels), runs cut in length where the whole would take longer than a pass may, and odd
sizes between them.  Models, wavelets and data are synthetic: layered, faulted, smoothed
velocities; Ricker sources; gathers of hyperbolic arrivals; band-limited noise windows.
"""
from __future__ import annotations

import math

import numpy as np
import torch

SPONGE_ALPHA = 0.0015


def listed():
    return [
        # one virtual gather of the pipeline: the smallest call, host arrays in and out
        dict(name="virtual_gather", kind="gather", nt=3000, nch=120, n_rec=95, lag_s=1.75,
             dt=0.01, dt_sim=0.002, nt_sim=1000, branch="symmetric"),
        # observed gather of the example line: few points a step, many steps
        dict(name="model_example", kind="model", nz=150, nx=400, nt=2000, rec_step=1, fs=True,
             n_sponge=40),
        # the example survey, all shots of the line in one call
        dict(name="survey_example", kind="survey", nz=150, nx=400, nt=2000, n_shots=20,
             rec_step=1, n_sponge=40, interval=2),
        # a mid-size shot with odd sides, sparse receivers and every third step imaged
        dict(name="shot_odd", kind="shot", nz=301, nx=1203, nt=1500, rec_step=3, fs=True,
             n_sponge=30, interval=3, storage="auto"),
        # a shot whose forward field is checkpointed, no free surface
        dict(name="shot_checkpoint", kind="shot", nz=607, nx=2410, nt=1200, rec_step=2, fs=False,
             iz=44, n_sponge=40, interval=2, storage="checkpoint"),
        # the production grid: one shot with a receiver in every column
        dict(name="shot_large", kind="shot", nz=1000, nx=4000, nt=3000, rec_step=1, fs=True,
             n_sponge=40, interval=2, storage="auto"),
        # uneven gathers, admitted as memory allows
        dict(name="batch_gathers", kind="batch", n_jobs=20, nz0=200, nz1=600, nx0=400, nx1=2000,
             nt0=1500, nt1=3000, arena_gb=24.0),
        # velocity gradients: a small odd grid and the production grid
        dict(name="gradient_odd", kind="gradient", nz=211, nx=517, nt=900, rec_step=2, fs=True,
             n_sponge=30),
        dict(name="gradient_large", kind="gradient", nz=1000, nx=4000, nt=600, rec_step=1,
             fs=True, n_sponge=40),
        # elastic gradients: a job of several shots on one model, and the survey grid
        dict(name="elastic_job", kind="elastic", nz=363, nx=725, nt=700, n_shots=4, fs=True,
             n_sponge=30),
        dict(name="elastic_large", kind="elastic", nz=1024, nx=2048, nt=500, n_shots=1, fs=True,
             n_sponge=40),
        # the correlation stack of the pipeline
        dict(name="correlation_stack", kind="stack", nt=3000, nch=600, n_src=16, n_rec=95,
             lag_s=1.75, dt=0.01, n_win=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "shot", "shot", "survey", "batch", "gradient", "elastic", "stack",
                       "gather"])
    fs, n_sp = rng.random() < 0.75, rng.randint(10, 40)
    # near the surface, or below the upper sponge where there is no free surface
    iz = rng.choice([2, 3]) if fs or kind == "survey" else n_sp + rng.randint(1, 6)
    if kind == "gather":
        nt = _log_int(rng, 400, 4000)
        return dict(kind=kind, nt=nt, nch=rng.randint(30, 600), n_rec=rng.randint(8, 200),
                    lag_s=round(min(2.5, 0.004 * nt) * rng.uniform(0.3, 1.0), 2), dt=0.01,
                    dt_sim=rng.choice([0.001, 0.002, 0.0033]), nt_sim=_log_int(rng, 200, 2000),
                    branch=rng.choice(["causal", "anticausal", "symmetric"]))
    if kind == "stack":
        nt = _log_int(rng, 500, 4000)
        return dict(kind=kind, nt=nt, nch=rng.randint(100, 600), n_src=rng.randint(1, 16),
                    n_rec=rng.randint(10, 200), lag_s=round(rng.uniform(0.3, 1.75), 2), dt=0.01,
                    n_win=rng.randint(1, 6))
    if kind == "batch":
        nt = rng.randint(400, 1500)
        return dict(kind=kind, n_jobs=rng.randint(3, 20), nz0=rng.randint(60, 250),
                    nz1=rng.randint(250, 600), nx0=rng.randint(120, 500),
                    nx1=rng.randint(500, 1800), nt0=nt, nt1=2 * nt, arena_gb=16.0)
    if kind == "elastic":
        nz, nx = _log_int(rng, 90, 1024), _log_int(rng, 150, 2048)
        shots = rng.randint(1, max(1, min(6, 1500000 // (nz * nx))))
        nt = _log_int(rng, 150, max(160, min(900, int(1.0e9 / (nz * nx * shots)))))
        return dict(kind=kind, nz=nz, nx=nx, nt=nt, n_shots=shots, fs=fs,
                    n_sponge=rng.randint(10, 40))
    if kind == "gradient":
        nz, nx = _log_int(rng, 90, 1000), _log_int(rng, 130, 4000)
        nt = _log_int(rng, 150, max(160, min(2000, int(2.0e9 / (nz * nx)))))
        return dict(kind=kind, nz=nz, nx=nx, nt=nt, rec_step=rng.randint(1, 4), fs=fs,
                    iz=iz, n_sponge=n_sp)
    if kind == "survey":
        nz, nx = _log_int(rng, 80, 400), _log_int(rng, 150, 1200)
        n = rng.randint(2, 16)
        nt = _log_int(rng, 200, max(220, min(2000, int(3.0e9 / (nz * nx * n)))))
        return dict(kind=kind, nz=nz, nx=nx, nt=nt, n_shots=n, rec_step=rng.randint(1, 4),
                    iz=iz, n_sponge=n_sp,
                    interval=rng.randint(1, 4))
    # single shots and gathers: from small grids to the production one and just beyond
    nz, nx = _log_int(rng, 60, 1024), _log_int(rng, 100, 4096)
    nt = _log_int(rng, 200, max(220, min(3000, int(8.0e9 / (nz * nx)))))
    if kind == "model":
        return dict(kind=kind, nz=nz, nx=nx, nt=nt, rec_step=rng.randint(1, 4), fs=fs,
                    iz=iz, n_sponge=n_sp)
    return dict(kind=kind, nz=nz, nx=nx, nt=nt, rec_step=rng.randint(1, 4), fs=fs,
                iz=iz, n_sponge=n_sp,
                interval=rng.randint(1, 4), storage=rng.choice(["auto", "checkpoint"]))


# ---- inputs --------------------------------------------------------------------

DX = 5.0
V0, V1 = 1500.0, 3000.0
DT = 0.4 * DX / 3500.0  # CFL about 0.57 at the fastest cell


def _ricker(f0, dt, nt):
    a = (np.pi * f0 * (np.arange(nt) * dt - 1.0 / f0)) ** 2
    return ((1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _smooth(v, sigma):
    """Gaussian smoothing of a (nz, nx) float64 CUDA tensor, edges repeated."""
    r = int(3 * sigma)
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=v.device, dtype=v.dtype) / sigma) ** 2)
    k = k / k.sum()
    for dim in (0, 1):
        n = v.shape[dim]
        idx = torch.arange(-r, n + r, device=v.device).clamp(0, n - 1)
        p = v.index_select(dim, idx)
        acc = torch.zeros_like(v)
        for i in range(2 * r + 1):
            acc += k[i] * p.narrow(dim, i, n)
        v = acc
    return v


def _velocity(rng, nz, nx, v0=V0, v1=V1, jump=400.0):
    """Velocity rising with depth plus a layer cut by two faults, smoothed; float32 numpy."""
    z = torch.arange(nz, device="cuda", dtype=torch.float64)[:, None] / max(1, nz - 1)
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[None, :] / max(1, nx - 1)
    top = torch.full((nz, nx), float(rng.uniform(0.3, 0.6)), device="cuda", dtype=torch.float64)
    for _ in range(2):
        trace = float(rng.uniform(0.15, 0.85)) + float(rng.uniform(-0.3, 0.3)) * z
        top = top + torch.where(x > trace, float(rng.uniform(-0.1, 0.1)), 0.0)
    v = v0 + (v1 - v0) * z + 0.0 * x
    v = v + torch.where((z >= top) & (z < top + float(rng.uniform(0.08, 0.2))), jump, 0.0)
    return _smooth(v, 3.0).float().cpu().numpy()


def _gather(rng, nt, dt, f0, cols, src, dx, v=1800.0, amp=1.0):
    """A direct arrival and two reflections recorded at grid columns ``cols``, weak noise."""
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    t = torch.arange(nt, device="cuda", dtype=torch.float32)[:, None] * dt - 1.0 / f0
    off = (torch.as_tensor(np.asarray(cols), device="cuda").float()[None, :] - float(src)) * dx
    out = 1e-3 * torch.randn((nt, len(cols)), device="cuda", generator=g)
    for k in range(3):
        t0 = 0.0 if k == 0 else float(rng.uniform(0.15, 0.7)) * nt * dt
        a = (math.pi * f0 * (t - torch.sqrt(t0 * t0 + (off / (v * (1.0 + 0.2 * k))) ** 2))) ** 2
        out += (1.0, 0.4, -0.25)[k] * (1.0 - 2.0 * a) * torch.exp(-a)
    return (amp * out).cpu().numpy()


def _acoustic_inputs(case, seed):
    rng = np.random.default_rng([seed, 11])
    nz, nx, nt = case["nz"], case["nx"], case["nt"]
    f0 = V0 / (12.0 * DX)
    base = _velocity(rng, nz, nx)
    rec = np.arange(0, nx, case["rec_step"])
    d = dict(vel=base, rec=rec, w=_ricker(f0, DT, nt), iz=case.get("iz", 2))
    n = case.get("n_shots", 1)
    d["src"] = [int(s) for s in rng.integers(4, nx - 4, n)] if n == 1 else \
        [int(4 + (2 * k + 1) * (nx - 8) // (2 * n)) for k in range(n)]
    if case["kind"] in ("shot", "survey"):
        # flood models: the columns beyond a line either side of a fault repeat the line's
        fault = int(rng.integers(nx // 3, 2 * nx // 3 + 1))
        ls, lr = max(0, fault - 15), min(nx - 1, fault + 15)
        d["sed"] = np.ascontiguousarray(base[:, np.minimum(np.arange(nx), ls)])
        d["rock"] = np.ascontiguousarray(base[:, np.maximum(np.arange(nx), lr)])
        d["data"] = [_gather(rng, nt, DT, f0, rec, s, DX) for s in d["src"]]
    if case["kind"] == "gradient":
        d["data"] = [_gather(rng, nt, DT, f0, rec, d["src"][0], DX, amp=DT * DT)]
    return d


def _batch_inputs(case, seed):
    rng = np.random.default_rng([seed, 12])
    size = np.random.default_rng([case["n_jobs"], case["nt0"], case["nx1"]])  # sizes: the case's own
    jobs = []
    for _ in range(case["n_jobs"]):
        nz = int(size.integers(case["nz0"], case["nz1"] + 1))
        nx = int(size.integers(case["nx0"], case["nx1"] + 1))
        nt = int(size.integers(case["nt0"], case["nt1"] + 1))
        f0 = V0 / (float(rng.uniform(10.0, 14.0)) * DX)
        vel = _velocity(rng, nz, nx)
        rec = np.arange(nx)
        src = int(rng.integers(4, nx - 4))
        jobs.append(dict(nz=nz, nx=nx, nt=nt, vel=vel, rec=rec, src=src, w=_ricker(f0, DT, nt),
                         data=_gather(rng, nt, DT, f0, rec, src, DX)))
    return jobs


EL_DX, EL_DT = 2.0, 2e-4


def _elastic_inputs(case, seed):
    rng = np.random.default_rng([seed, 13])
    nz, nx, nt, n = case["nz"], case["nx"], case["nt"], case["n_shots"]
    vs = _velocity(rng, nz, nx, 300.0, 1200.0, 150.0)
    f0 = 20.0 if nt * EL_DT > 0.1 else 40.0
    src = [int(4 + (2 * k + 1) * (nx - 8) // (2 * n)) for k in range(n)]
    rec = np.arange(2, nx - 2)
    data = np.stack([_gather(rng, nt, EL_DT, f0, rec, s, EL_DX, v=500.0, amp=1e-5) for s in src])
    return dict(vs=vs, src=src, rec=rec, w=_ricker(f0, EL_DT, nt), data=data)


def _noise(rng, nt, nch):
    """Band-limited noise crossing the array: a common signal with moveout plus local noise."""
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    common = torch.randn(nt + 2 * nch, device="cuda", generator=g)
    idx = torch.arange(nt, device="cuda")[:, None] + torch.arange(nch, device="cuda")[None, :] // 3
    d = common[idx] + 0.5 * torch.randn((nt, nch), device="cuda", generator=g)
    return (0.25 * d[:-2] + 0.5 * d[1:-1] + 0.25 * d[2:]).cpu().numpy()


def _noise_inputs(case, seed):
    rng = np.random.default_rng([seed, 14])
    nch = case["nch"]
    n_win = case.get("n_win", 1)
    wins = [_noise(rng, case["nt"] + 2, nch) for _ in range(n_win)]
    n_src = case.get("n_src", 1)
    src = [int((2 * k + 1) * nch // (2 * n_src)) for k in range(n_src)]
    rec = np.unique(np.linspace(0, nch - 1, case["n_rec"]).astype(int))
    return dict(wins=wins, src=src, rec=rec)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("model", "shot", "survey", "gradient"):
        from das_gb300.rtm_engine import FloodModels, TSWRTMEngine
        from das_gb300.wave_solver import WaveSolver2D
        d = _acoustic_inputs(case, seed)
        st["d"] = d
        st["solver"] = WaveSolver2D(case["nx"], case["nz"], DX, DX, DT,
                                    n_sponge=case["n_sponge"], sponge_alpha=SPONGE_ALPHA,
                                    free_surface_top=case.get("fs", True))
        if kind in ("shot", "survey"):
            st["flood"] = FloodModels(d["vel"], d["sed"], d["rock"], 0, 0)
            st["engine"] = TSWRTMEngine(st["solver"], storage=case.get("storage", "auto"))
        if kind == "gradient":
            st["vel"] = torch.tensor(d["vel"], device="cuda")
            st["obs"] = torch.tensor(d["data"][0], device="cuda")
    elif kind == "batch":
        from das_gb300.batch import BatchEngine, ShotJob
        st["jobs"] = [ShotJob(j["nx"], j["nz"], DX, DX, DT, j["vel"], j["vel"], j["w"], j["data"],
                              j["rec"], j["src"], 2) for j in _batch_inputs(case, seed)]
        st["engine"] = BatchEngine(arena_bytes=int(case["arena_gb"] * (1 << 30)), max_shots=64,
                                   tile=(4, 4))
    elif kind == "elastic":
        from das_gb300.elastic import ElasticSolver2D
        d = _elastic_inputs(case, seed)
        st["d"] = d
        st["solver"] = ElasticSolver2D(case["nx"], case["nz"], EL_DX, EL_DX, EL_DT,
                                       n_sponge=case["n_sponge"], sponge_alpha=SPONGE_ALPHA,
                                       free_surface_top=case["fs"])
        vs = torch.tensor(d["vs"], device="cuda")
        st["vs"] = vs if case["n_shots"] == 1 else vs.expand(case["n_shots"], -1, -1).contiguous()
        st["obs"] = torch.tensor(d["data"] if case["n_shots"] > 1 else d["data"][0],
                                 device="cuda")
    elif kind in ("stack", "gather"):
        st["d"] = _noise_inputs(case, seed)
    else:
        raise ValueError(kind)
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "model":
        d = state["d"]
        rec, _ = state["solver"].forward_propagate_acoustic(d["vel"], d["w"], d["src"][0], d["iz"],
                                                            d["rec"], d["iz"])
        return rec
    if kind == "shot":
        d = state["d"]
        img, ill = state["engine"].migrate_shot(state["flood"], d["w"], d["src"][0], d["iz"],
                                                d["data"][0], d["rec"], d["iz"],
                                                case["interval"])
        return {"image": img, "illumination": ill}
    if kind == "survey":
        d = state["d"]
        n = len(d["src"])
        r = state["engine"].migrate_multiple_shots(state["flood"], [d["w"]] * n, d["src"],
                                                   [d["iz"]] * n, d["data"], d["rec"], d["iz"],
                                                   case["interval"])
        return {"raw": r.raw_image, "laplacian": r.laplacian_image,
                "normalized": r.normalized_image}
    if kind == "batch":
        results, _ = state["engine"].run(state["jobs"])
        return [x for pair in results for x in pair]
    if kind == "gradient":
        from das_gb300.autograd import model_traces
        d = state["d"]
        v = state["vel"].detach().requires_grad_(True)
        tr = model_traces(v, state["solver"], d["w"], d["src"][0], d["iz"],
                          d["rec"][_inside(d, case)], d["iz"])
        (0.5 * ((tr - state["obs"][:, _inside(d, case)]) ** 2).sum()).backward()
        return {"traces": tr.detach(), "gradient": v.grad}
    if kind == "elastic":
        from das_gb300.elastic import elastic_traces
        d = state["d"]
        vs = state["vs"].detach().requires_grad_(True)
        src = d["src"] if case["n_shots"] > 1 else d["src"][0]
        iz = [2] * case["n_shots"] if case["n_shots"] > 1 else 2
        tr = elastic_traces(vs, state["solver"], d["w"], src, iz, d["rec"], 4)
        (0.5 * ((tr - state["obs"]) ** 2).sum()).backward()
        return {"traces": tr.detach(), "gradient": vs.grad}
    if kind == "stack":
        from das_gb300.interferometry import CrossCorrelationStack
        d = state["d"]
        st = CrossCorrelationStack(case["nt"], case["nch"], d["src"], d["rec"], case["lag_s"],
                                   case["dt"])
        try:
            for w in d["wins"]:
                st.add(w)
            out = st.result()
        finally:
            st.close()
        return {str(s): out[s][0] for s in d["src"]}
    from das_gb300.interferometry import (build_virtual_shot_gather, compute_cross_correlation,
                                          resample_gather_to_sim_dt)
    d = state["d"]
    ccfs, lags = compute_cross_correlation(d["wins"][0], d["src"][0], case["lag_s"], case["dt"],
                                           d["rec"])
    g = build_virtual_shot_gather(ccfs, lags, 0, d["src"][0], np.arange(case["nch"]) * 10.0,
                                  d["rec"], branch=case["branch"])
    sim = resample_gather_to_sim_dt(g.shot_gather, case["dt"], case["dt_sim"], case["nt_sim"])
    return {"ccfs": ccfs, "gather": g.shot_gather, "resampled": sim}


def _inside(d, case):
    """Receivers of the gradient path sit on updated cells: the first and last two columns out."""
    return np.flatnonzero((d["rec"] >= 2) & (d["rec"] < case["nx"] - 2))


def work(case):
    """Inputs read once, outputs written once; arithmetic of the time steps or correlations."""
    kind = case["kind"]
    if kind in ("model", "shot", "survey", "gradient"):
        p, nt, n = case["nz"] * case["nx"], case["nt"], case.get("n_shots", 1)
        nr = len(range(0, case["nx"], case["rec_step"]))
        passes = {"model": 1, "shot": 2, "survey": 2, "gradient": 2}[kind]
        models = {"model": 1, "shot": 2, "survey": 2, "gradient": 1}[kind]
        outs = {"model": 0, "shot": 2, "survey": 3, "gradient": 1}[kind]
        per = {"model": 20, "shot": 21, "survey": 21, "gradient": 31}[kind]
        gathers = (2 if kind == "gradient" else 1) * n * nt * nr
        return {"bytes": 4.0 * ((models + outs) * p + gathers + nt),
                "flops": float(per * passes * p * nt * n)}
    if kind == "batch":
        size = np.random.default_rng([case["n_jobs"], case["nt0"], case["nx1"]])
        b = f = 0.0
        for _ in range(case["n_jobs"]):
            nz = int(size.integers(case["nz0"], case["nz1"] + 1))
            nx = int(size.integers(case["nx0"], case["nx1"] + 1))
            nt = int(size.integers(case["nt0"], case["nt1"] + 1))
            b += 4.0 * (4 * nz * nx + nt * nx + nt)
            f += 42.0 * nz * nx * nt
        return {"bytes": b, "flops": f}
    if kind == "elastic":
        p, nt, n = case["nz"] * case["nx"], case["nt"], case["n_shots"]
        return {"bytes": 4.0 * (2 * n * p + 2 * n * nt * (case["nx"] - 4)),
                "flops": float(170 * p * nt * n)}
    nr, ns, nw = case["n_rec"], case.get("n_src", 1), case.get("n_win", 1)
    rows = 2 * int(round(case["lag_s"] / case["dt"])) + 1
    b = 4.0 * (nw * case["nt"] * (nr + ns) + ns * rows * nr)
    if kind == "gather":
        b += 4.0 * nr * (rows + case["nt_sim"])
    return {"bytes": b, "flops": 2.0 * nw * ns * rows * nr * case["nt"]}


# ---- the same in 64 bits, plain torch ------------------------------------------------

F64 = torch.float64


def _cerjan(nz, nx, n, fs):
    ix, iz = torch.arange(nx, device="cuda")[None, :], torch.arange(nz, device="cuda")[:, None]
    d = torch.zeros((nz, nx), device="cuda", dtype=F64)
    for c in (n - ix, ix - (nx - 1 - n), iz - (nz - 1 - n)):
        d = torch.maximum(d, c.to(F64).expand(nz, nx))
    if not fs:
        d = torch.maximum(d, (n - iz).to(F64).expand(nz, nx))
    # the taper is an input of the scheme: its float32 values
    return torch.exp(-float(np.float32(SPONGE_ALPHA)) * d * d).float().to(F64)


def _lap(p):
    """4th-order Laplacian of the interior, unit spacing."""
    m = slice(2, -2)
    far = p[..., m, :-4] + p[..., m, 4:] + p[..., :-4, m] + p[..., 4:, m]
    near = p[..., m, 1:-3] + p[..., m, 3:-1] + p[..., 1:-3, m] + p[..., 3:-1, m]
    return (-1.0 / 12.0) * far + (4.0 / 3.0) * near - 5.0 * p[..., m, m]


def _interior(p, pp, c, sp):
    """The updated interior of one step from p_curr, p_prev, v^2 dt^2 and the sponge."""
    m = slice(2, -2)
    return (2.0 * p[..., m, m] - pp[..., m, m] + c[..., m, m] * _lap(p) / DX ** 2) * sp[..., m, m]


def _advance(pn, p, pp, c, sp, fs):
    pn[..., 2:-2, 2:-2] = _interior(p, pp, c, sp)
    if fs:
        pn[..., 0, :] = 0.0
        pn[..., 1, :] = -pn[..., 2, :]


def _model64(vel, w, src, rec, iz, n_sponge, fs, interval=0):
    """Traces, snapshots and illumination of shots (S sources) in one model."""
    nz, nx = vel.shape
    S, nt = len(src), len(w)
    c = torch.as_tensor(vel, device="cuda").to(F64) ** 2 * DT ** 2
    sp = _cerjan(nz, nx, n_sponge, fs)
    p = [torch.zeros((S, nz, nx), device="cuda", dtype=F64) for _ in range(3)]
    si, sx = torch.arange(S, device="cuda"), torch.as_tensor(src, device="cuda")
    rx = torch.as_tensor(rec, device="cuda")
    tr = torch.zeros((S, nt, len(rec)), device="cuda", dtype=F64)
    snaps, ill = [], torch.zeros((S, nz, nx), device="cuda", dtype=F64)
    for it in range(nt):
        pp, pc, pn = p[it % 3], p[(it + 1) % 3], p[(it + 2) % 3]
        pc[si, iz, sx] += float(w[it]) * DT * DT
        if interval and it % interval == 0:
            snaps.append(pc.clone())
            ill += pc * pc
        _advance(pn, pc, pp, c, sp, fs)
        tr[:, it] = pn[:, iz, rx]
    return tr, snaps, ill * (DT * max(1, interval))


def _image64(vel, data, rec, iz, snaps, n_sponge, fs, interval):
    nz, nx = vel.shape
    S, nt = len(data), data[0].shape[0]
    c = torch.as_tensor(vel, device="cuda").to(F64) ** 2 * DT ** 2
    sp = _cerjan(nz, nx, n_sponge, fs)
    p = [torch.zeros((S, nz, nx), device="cuda", dtype=F64) for _ in range(3)]
    rx = torch.as_tensor(rec, device="cuda")
    dd = torch.as_tensor(np.stack(data), device="cuda")
    img = torch.zeros((S, nz, nx), device="cuda", dtype=F64)
    for m in range(nt):
        it = nt - 1 - m
        pp, pc, pn = p[m % 3], p[(m + 1) % 3], p[(m + 2) % 3]
        pc[:, iz, rx] += dd[:, it].to(F64) * DT ** 2
        if it % interval == 0:
            img += snaps[it // interval] * pc * (DT * interval)
        _advance(pn, pc, pp, c, sp, fs)
    return img


def _grad_acoustic64(case, d):
    from torch.utils.checkpoint import checkpoint
    nz, nx, nt, fs = case["nz"], case["nx"], case["nt"], case["fs"]
    keep = _inside(d, case)
    vel = torch.as_tensor(d["vel"], device="cuda").to(F64).requires_grad_(True)
    sp = _cerjan(nz, nx, case["n_sponge"], fs)
    rx = torch.as_tensor(d["rec"][keep], device="cuda")
    w = [float(x) * DT * DT for x in d["w"]]
    unit = torch.zeros((nz, nx), device="cuda", dtype=F64)
    unit[d["iz"], d["src"][0]] = 1.0

    def seg(vel, pp, pc, a, b):
        c = vel * vel * DT ** 2
        out = []
        for it in range(a, b):
            pc = pc + w[it] * unit
            u = torch.nn.functional.pad(_interior(pc, pp, c, sp), (2, 2, 2, 2))
            if fs:
                u = torch.cat([u[:1], -u[2:3], u[2:]], 0)
            out.append(u[d["iz"], rx])
            pp, pc = pc, u
        return pp, pc, torch.stack(out)

    pp = torch.zeros((nz, nx), device="cuda", dtype=F64)
    pc, tr, step = pp, [], max(5, int(math.sqrt(nt)))
    for a in range(0, nt, step):
        pp, pc, t = checkpoint(seg, vel, pp, pc, a, min(nt, a + step), use_reentrant=False)
        tr.append(t)
    tr = torch.cat(tr)
    obs = torch.as_tensor(d["data"][0], device="cuda")[:, torch.as_tensor(keep, device="cuda")]
    (0.5 * ((tr - obs.to(F64)) ** 2).sum()).backward()
    return {"traces": tr.detach(), "gradient": vel.grad}


def _grad_elastic64(case, d):
    from torch.utils.checkpoint import checkpoint
    nz, nx, nt, fs, S = case["nz"], case["nx"], case["nt"], case["fs"], case["n_shots"]
    sp = _cerjan(nz, nx, case["n_sponge"], fs)
    z0 = 1 if fs else 2
    mask = torch.zeros((nz, nx), device="cuda", dtype=F64)
    mask[z0:nz - 2, 2:nx - 2] = 1.0
    sp = sp * mask
    vs = torch.as_tensor(d["vs"], device="cuda").to(F64).expand(S, nz, nx).clone()
    vs.requires_grad_(True)
    rx = torch.as_tensor(d["rec"], device="cuda")
    unit = torch.zeros((S, nz, nx), device="cuda", dtype=F64)
    for k, s in enumerate(d["src"]):
        unit[k, 2, s] = 1.0
    k1, k2 = 9.0 / 8.0, -1.0 / 24.0

    def diff(a, dim, fwd):
        """4th-order staggered difference, zero outside the grid."""
        q = torch.nn.functional.pad(a, (2, 2, 0, 0) if dim == -1 else (0, 0, 2, 2))
        n = a.shape[dim]
        s = lambda k: q.narrow(dim, 2 + k, n)  # noqa: E731
        if fwd:
            return (k1 * (s(1) - s(0)) + k2 * (s(2) - s(-1))) / EL_DX
        return (k1 * (s(0) - s(-1)) + k2 * (s(1) - s(-2))) / EL_DX

    def seg(vs, st, a, b):
        vp = 1.73 * vs
        rho = 310.0 * vp ** 0.25
        mu = rho * vs * vs
        lam = rho * vp * vp - 2.0 * mu
        bu = EL_DT / rho
        l2m = (lam + 2.0 * mu) * EL_DT
        lam, mu = lam * EL_DT, mu * EL_DT
        vx, vz, xx, zz, xz = st
        out = []
        for n in range(a, b):
            vz = vz + (float(d["w"][n]) * EL_DT) * unit
            vx = (vx + bu * (diff(xx, -1, True) + diff(xz, -2, False))) * sp
            vz = (vz + bu * (diff(xz, -1, False) + diff(zz, -2, True))) * sp
            ex, ez = diff(vx, -1, False), diff(vz, -2, False)
            xx = (xx + l2m * ex + lam * ez) * sp
            zz = (zz + lam * ex + l2m * ez) * sp
            xz = (xz + mu * (diff(vz, -1, True) + diff(vx, -2, True))) * sp
            out.append(ez[:, 4, rx])
        return (vx, vz, xx, zz, xz), torch.stack(out, 1)

    st = tuple(torch.zeros((S, nz, nx), device="cuda", dtype=F64) for _ in range(5))
    tr, step = [], max(4, int(0.7 * math.sqrt(nt)))
    for a in range(0, nt, step):
        st, t = checkpoint(seg, vs, st, a, min(nt, a + step), use_reentrant=False)
        tr.append(t)
    tr = torch.cat(tr, 1)
    obs = torch.as_tensor(d["data"], device="cuda").to(F64)
    (0.5 * ((tr - obs) ** 2).sum()).backward()
    if S == 1:
        return {"traces": tr.detach()[0], "gradient": vs.grad[0]}
    return {"traces": tr.detach(), "gradient": vs.grad}


def _xcorr64(win, src, rec, n_lags):
    """(rows, n_rec): sum_t s[t] r[t + l], l = -n_lags..n_lags."""
    nt = win.shape[0]
    a = torch.as_tensor(win, device="cuda").to(F64)
    n = 1 << (nt + n_lags).bit_length()
    f = torch.fft.rfft(a[:, torch.as_tensor(rec, device="cuda")], n=n, dim=0)
    c = torch.fft.irfft(f * torch.fft.rfft(a[:, src], n=n).conj()[:, None], n=n, dim=0)
    return torch.cat([c[n - n_lags:], c[:n_lags + 1]])


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("model", "shot", "survey"):
            d, fs, n_sp = _acoustic_inputs(case, seed), case.get("fs", True), case["n_sponge"]
            if kind == "model":
                return _model64(d["vel"], d["w"], d["src"], d["rec"], d["iz"], n_sp, fs)[0][0]
            if case.get("n_shots", 1) * case["nz"] * case["nx"] * \
                    (case["nt"] // case["interval"] + 1) * 8.0 > 1.0e11:
                return None
            _, snaps, ill = _model64(d["sed"], d["w"], d["src"], d["rec"], d["iz"], n_sp, fs,
                                     case["interval"])
            img = _image64(d["rock"], d["data"], d["rec"], d["iz"], snaps, n_sp, fs,
                           case["interval"])
            if kind == "shot":
                return {"image": img[0], "illumination": ill[0]}
            img, ill = img.sum(0), ill.sum(0)
            mute = _cerjan(case["nz"], case["nx"], n_sp, fs) < 0.99
            img[mute] = 0.0
            ill[mute] = 0.0
            p = torch.nn.functional.pad(img[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
            lap = (p[1:-1, :-2] + p[1:-1, 2:] + p[:-2, 1:-1] + p[2:, 1:-1] - 4.0 * img) / DX ** 2
            lap[mute] = 0.0
            return {"raw": img, "laplacian": lap,
                    "normalized": img / (ill.sqrt() + 1e-4 * ill.max())}
        if kind in ("stack", "gather"):
            d = _noise_inputs(case, seed)
            n_lags = int(round(case["lag_s"] / case["dt"]))
            if 2 * n_lags + 1 >= case["nt"]:
                return None
            if kind == "stack":
                return {str(s): sum(_xcorr64(w, s, d["rec"], n_lags) for w in d["wins"]) /
                        len(d["wins"]) for s in d["src"]}
            c = _xcorr64(d["wins"][0], d["src"][0], d["rec"], n_lags)
            lags = np.arange(-n_lags, n_lags + 1) * case["dt"]
            g = torch.gradient(c, spacing=float(lags[1] - lags[0]), dim=0)[0]
            pos, neg = g[n_lags:], g[:n_lags + 1].flip(0)
            b = {"causal": pos, "anticausal": neg, "symmetric": 0.5 * (pos + neg)}[case["branch"]]
            x = np.arange(case["nt_sim"]) * case["dt_sim"]
            t = np.arange(b.shape[0]) * case["dt"]
            hi = np.clip(np.searchsorted(t, x), 1, len(t) - 1)
            wt = torch.as_tensor((x - t[hi - 1]) / (t[hi] - t[hi - 1]), device="cuda")[:, None]
            hi = torch.as_tensor(hi, device="cuda")
            r = b[hi] * wt + b[hi - 1] * (1.0 - wt)
            r[torch.as_tensor(x > t[-1], device="cuda")] = 0.0
            return {"ccfs": c, "gather": b, "resampled": r}
    if kind == "gradient":
        return _grad_acoustic64(case, _acoustic_inputs(case, seed))
    if kind == "elastic":
        return _grad_elastic64(case, _elastic_inputs(case, seed))
    return None  # batch: too many steps in 64 bits for the time allowed
