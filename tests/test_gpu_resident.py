"""The time loop with its wavefields kept on chip (the default where a grid fits) against
one launch per step: traces, snapshots, images and illumination bit-identical.

Sizes: the smallest grid, every remainder of nx by the four-point unit, one tile, many
tiles, tiles of the least height, the production grid; calls that keep the step kernels
(receivers sharing a column, sources and receivers off the interior rows) are among them.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# nz, nx, free surface, sponge, receiver row, receivers, interval, steps
CASES = [
    (5, 5, True, 0, 2, "all", 1, 7),
    (8, 6, False, 2, 3, "all", 2, 9),
    (9, 37, True, 3, 2, "all", 1, 1),
    (33, 130, True, 6, 2, "all", 2, 41),
    (34, 131, True, 6, 3, "third", 3, 40),
    (35, 129, False, 6, 20, "shuffled", 2, 40),
    (61, 260, True, 10, 58, "all", 1, 33),
    (61, 261, True, 10, 2, "shared", 2, 33),
    (61, 262, False, 10, 1, "all", 2, 33),
    (150, 403, True, 40, 2, "all", 4, 120),
    (607, 1203, False, 30, 36, "third", 2, 90),
    (1000, 4000, True, 40, 2, "all", 2, 60),
    (1024, 4096, True, 40, 2, "all", 2, 12),  # beyond the chip
]


@pytest.mark.parametrize("nz,nx,fs,n_sponge,riz,kind,interval,nt", CASES)
def test_resident_equals_steps(nz, nx, fs, n_sponge, riz, kind, interval, nt):
    from das_gb300.rtm_engine import TSWRTMEngine
    from das_gb300.velocity_flood import FloodModels
    from das_gb300.wave_solver import WaveSolver2D
    rng = np.random.default_rng(nz * 5000 + nx)
    v = rng.uniform(1500, 3000, (nz, nx)).astype(np.float32)
    v2 = (v * np.float32(1.01)).astype(np.float32)
    w = rng.standard_normal(nt).astype(np.float32)
    rix = {"all": np.arange(nx), "third": np.arange(1, nx, 3),
           "shuffled": rng.permutation(nx)[: nx // 2],
           "shared": np.sort(rng.integers(0, nx, nx // 2))}[kind]
    data = rng.standard_normal((nt, len(rix))).astype(np.float32)
    out = []
    for pdl in (True, False):  # the default launch mode, and the step kernels
        s = WaveSolver2D(nx, nz, 5.0, 5.0, 5e-4, n_sponge=n_sponge, free_surface_top=fs)
        s.set_launch("grid", pdl)
        six, siz = max(2, nx // 3), min(max(riz, 2), nz - 3)
        res = []
        for _ in range(2):  # a second run finds the first one's packets and planes
            rec, snaps = s.forward_propagate_acoustic(v, w, six, siz, rix, riz, nz * nx < 1 << 20,
                                                      interval)
            res.append((rec, snaps))
        for storage in ("all", "checkpoint"):
            res.append(TSWRTMEngine(s, storage).migrate_shot(FloodModels(v, v, v2, 0, 0), w, six,
                                                             siz, data, rix, riz, interval))
        if nz * nx < 1 << 20:
            fw = res[0][1]
            img = np.ones((nz, nx), np.float32)
            s.backward_propagate_and_correlate(v2, data, rix, riz, fw, img, interval)
            res.append((img, None))
        out.append(res)
        s.close()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            if x is not None:
                np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(out[0][0][0], out[0][1][0])


def test_batch_waves_equal_steps():
    """A batch whose shots advance on chip, several to a launch and over more than one
    launch, beside shots that keep the step kernels; modelling jobs among them."""
    from das_gb300.batch import BatchEngine, ModelJob, ShotJob
    from das_gb300.rtm_engine import TSWRTMEngine
    from das_gb300.velocity_flood import FloodModels
    from das_gb300.wave_solver import WaveSolver2D
    rng = np.random.default_rng(7)
    dx, dt, jobs = 5.0, 5e-4, []
    for k, (nz, nx, nt) in enumerate([(90, 260, 150), (600, 2000, 70), (33, 77, 64), (500, 1900, 90),
                                      (128, 301, 180), (1024, 4100, 20), (590, 1990, 75),
                                      (61, 130, 333)]):
        v = rng.uniform(1500, 3200, (nz, nx)).astype(np.float32)
        w = rng.standard_normal(nt).astype(np.float32)
        rix = np.arange(nx) if k % 2 else rng.permutation(nx)[: nx // 2]
        if k == 4:
            rix = np.zeros(9, int) + 5  # one column: the step kernels
        if k == 6:
            jobs.append(ModelJob(nx, nz, dx, dx, dt, v, w, rix, nx // 2, 2))
            continue
        data = rng.standard_normal((nt, len(rix))).astype(np.float32)
        jobs.append(ShotJob(nx, nz, dx, dx, dt, v, v * np.float32(1.01), w, data, rix, nx // 2, 2, 2,
                            1 + k % 3, 10 if k else -1, 0.0015, k != 2))
    eng = BatchEngine(arena_bytes=8 << 30, max_shots=16, tile=(4, 4), steps_per_launch=8,
                      launches_per_graph=3)
    for _ in range(2):
        results, _ = eng.run(jobs)
        for j, r in zip(jobs, results):
            s = WaveSolver2D(j.nx, j.nz, dx, dx, dt, max(j.n_sponge, 0), 0.0015, j.free_surface_top)
            s.set_launch("grid", False)
            if isinstance(j, ModelJob):
                rec, _ = s.forward_propagate_acoustic(j.vel, j.wavelet, j.source_ix, 2,
                                                      j.receiver_ix, 2)
                np.testing.assert_array_equal(r, rec)
            else:
                img, ill = TSWRTMEngine(s, "all").migrate_shot(
                    FloodModels(j.vel_fwd, j.vel_fwd, j.vel_bwd, 0, 0), j.wavelet, j.source_ix, 2,
                    j.data, j.receiver_ix, 2, j.snapshot_interval)
                np.testing.assert_array_equal(r[0], img)
                np.testing.assert_array_equal(r[1], ill)
            s.close()
    eng.close()


@pytest.mark.parametrize("nz,nx,fs,n_sponge,riz,rstep,nt,seg", [
    (8, 9, True, 2, 2, 1, 40, 0),        # one tile; the fold's rows 2 and 3 at a tile's edge
    (9, 37, True, 3, 3, 1, 30, 7),
    (61, 261, True, 10, 2, 2, 90, 0),
    (60, 262, False, 10, 13, 1, 90, 90),  # every state stored
    (150, 403, True, 40, 2, 3, 200, 0),
    (700, 1990, False, 30, 36, 1, 60, 0),
])
def test_resident_gradient_equals_adjoint_kernels(nz, nx, fs, n_sponge, riz, rstep, nt, seg):
    """The velocity gradient with the adjoint on chip against the adjoint kernels: traces
    equal, the gradient to float32 rounding (a sum of nt products, each with a few
    roundings of 6e-8: 1e-5 holds with room, as between the two adjoint kernels)."""
    import torch
    from das_gb300.autograd import model_traces
    from das_gb300.wave_solver import WaveSolver2D
    rng = np.random.default_rng(nz + nx)
    v = (2000.0 + 300.0 * rng.random((nz, nx))).astype(np.float32)
    v[nz // 2, nx // 2] = 0.0  # no gradient where the velocity is zero
    w = rng.standard_normal(nt).astype(np.float32)
    rix = np.arange(2, nx - 2, rstep)
    r = torch.tensor(rng.standard_normal((nt, len(rix))).astype(np.float32), device="cuda")
    out = []
    for pdl in (True, False):
        s = WaveSolver2D(nx, nz, 5.0, 5.0, 5e-4, n_sponge=n_sponge, free_surface_top=fs)
        s.set_launch("grid", pdl)
        if seg:
            s.set_checkpoint_segment(seg)
        g = []
        for _ in range(2):
            vt = torch.tensor(v, device="cuda", requires_grad=True)
            d = model_traces(vt, s, w, nx // 3, min(max(riz, 2), nz - 3), rix, riz)
            d.backward(r)
            g.append((d.detach().cpu().numpy(), vt.grad.cpu().numpy()))
        np.testing.assert_array_equal(g[0][1], g[1][1])
        out.append(g[0])
        s.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    a, b = (x[1].astype(np.float64) for x in out)
    assert np.isfinite(a).all() and a[nz // 2, nx // 2] == 0.0
    assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
