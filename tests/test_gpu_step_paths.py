"""The paths of one launch per step in the default launch mode: captured passes, tile shapes,
the tiled adjoint.  Two receivers in one column keep a call on them where the grid alone would
run on chip.  And several engines at once, whose launches each want the whole chip."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _line(nx, step=3):
    r = np.arange(3, nx - 3, step)
    return np.append(r, r[len(r) // 2])


def _solver(nz, nx, fs=True, **kw):
    from das_gb300.wave_solver import WaveSolver2D
    s = WaveSolver2D(nx, nz, 5.0, 5.0, 5e-4, 20, 0.0015, fs)
    for k, v in kw.items():
        setattr(s, k, v)
    return s


@pytest.mark.parametrize("storage", ["all", "checkpoint"])
def test_replayed_passes_equal_direct_launches(storage):
    """Captured passes, replayed for new sources, models, data and receiver lines of the same
    count, against launches one by one: equal bit for bit, with the same counts of steps."""
    from das_gb300.rtm_engine import TSWRTMEngine
    from das_gb300.velocity_flood import FloodModels
    nz, nx, nt = 140, 500, 150
    rng = np.random.default_rng(5)
    shots = []
    for k, n in enumerate([nt, nt, nt - 31, nt]):
        v = rng.uniform(1600, 3000, (nz, nx)).astype(np.float32)
        rix = _line(nx) + k
        shots.append((FloodModels(v, v, (v * 1.01).astype(np.float32), 0, 0),
                      rng.standard_normal(n).astype(np.float32), 60 + 90 * k, rix, 2 + k,
                      rng.standard_normal((n, len(rix))).astype(np.float32)))
    out = []
    for graphs in (True, False):
        s = _solver(nz, nx)
        s.set_graphs(graphs)
        e = TSWRTMEngine(s, storage)
        res = []
        for fm, w, six, rix, riz, d in shots:
            img, ill = e.migrate_shot(fm, w, six, 2, d, rix, riz, 2)
            st = s.last_stats()
            assert st["step_launches"] >= 2 * len(w) and st["storage"] == storage
            res.append((img, ill, st["step_launches"], st["recomputed_steps"]))
            v, corr = fm.rock_flood, img.copy()
            rec, snaps = s.forward_propagate_acoustic(v, w, six, 2, rix, riz, True, 2)
            s.backward_propagate_and_correlate(v, d, rix, riz, snaps, corr, 2)
            res.append((rec, snaps, corr))
        out.append(res)
        s.close()
    for k, (a, b) in enumerate(zip(*out)):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y, err_msg=f"call {k}")


@pytest.mark.parametrize("tile", [(4, 4), (8, 4), (4, 8), (8, 8)])
@pytest.mark.parametrize("nz,nx,fs", [(33, 130, True), (61, 261, False), (150, 403, True)])
def test_tiles_in_the_default_mode(tile, nz, nx, fs):
    """Every tile shape with programmatic dependent launches equals the plain ones."""
    from das_gb300.rtm_engine import TSWRTMEngine
    from das_gb300.velocity_flood import FloodModels
    nt = 40
    rng = np.random.default_rng(nz)
    v = rng.uniform(1500, 3000, (nz, nx)).astype(np.float32)
    w = rng.standard_normal(nt).astype(np.float32)
    rix = _line(nx, 2)
    d = rng.standard_normal((nt, len(rix))).astype(np.float32)
    out = []
    for t, pdl in ((tile, True), ((4, 4), False)):
        s = _solver(nz, nx, fs, tile=t)
        s.set_launch("grid", pdl)
        res = list(s.forward_propagate_acoustic(v, w, nx // 3, 3, rix, 2, True, 2))
        for storage in ("all", "checkpoint"):
            res += TSWRTMEngine(s, storage).migrate_shot(FloodModels(v, v, v, 0, 0), w, nx // 3,
                                                         3, d, rix, 2, 2)
        assert s.last_stats()["step_launches"] >= 2 * nt
        out.append(res)
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("nz,nx,fs", [(50, 100, True), (70, 300, True), (90, 520, False)])
def test_tiled_adjoint_equals_per_cell_adjoint_on_step_kernels(nz, nx, fs):
    """As between the two kernels elsewhere: equal to float32 rounding."""
    from das_gb300.autograd import misfit_and_gradient
    rng = np.random.default_rng(nz + nx)
    v = (1800.0 + 40.0 * rng.standard_normal((nz, nx))).astype(np.float32)
    w = rng.standard_normal(120).astype(np.float32)
    rix = _line(nx, 1)
    obs = rng.standard_normal((len(w), len(rix))).astype(np.float32)
    s = _solver(nz, nx, fs)
    g = {}
    for form in ("cells", "tiled"):
        s.set_adjoint_form(form)
        g[form] = misfit_and_gradient(s, v, w, nx // 3, 6, rix, 3, obs)[1].astype(np.float64)
        assert s.last_stats()["step_launches"] >= len(w)
    s.close()
    assert np.abs(g["cells"]).max() > 0
    assert np.linalg.norm(g["tiled"] - g["cells"]) < 1e-5 * np.linalg.norm(g["cells"])


def test_engines_and_a_batch_on_threads():
    """Resident launches of several engines and a batch, enqueued from several threads at once
    (each launch's CTAs wait for one another, and only for their own launch's): every result
    as alone."""
    from das_gb300.batch import BatchEngine, ShotJob
    from das_gb300.wave_solver import WaveSolver2D
    rng = np.random.default_rng(2)
    runs = []
    for nz, nx, nt in [(301, 1203, 200), (600, 2000, 120), (150, 400, 400), (90, 260, 300)]:
        runs.append((rng.uniform(1500, 3000, (nz, nx)).astype(np.float32),
                     rng.standard_normal(nt).astype(np.float32)))
    jobs = []
    for nz, nx, nt in [(150, 400, 200), (301, 1203, 100), (90, 260, 150)]:
        v = rng.uniform(1500, 3000, (nz, nx)).astype(np.float32)
        jobs.append(ShotJob(nx, nz, 5.0, 5.0, 5e-4, v, v, rng.standard_normal(nt).astype(np.float32),
                            rng.standard_normal((nt, nx)).astype(np.float32), np.arange(nx),
                            nx // 2, 2, 2, 2, 10, 0.0015, True))
    solvers = [WaveSolver2D(v.shape[1], v.shape[0], 5.0, 5.0, 5e-4, n_sponge=10) for v, _ in runs]
    batch = BatchEngine(arena_bytes=2 << 30, max_shots=8)

    def model(i):
        v, w = runs[i]
        nx = v.shape[1]
        return [solvers[i].forward_propagate_acoustic(v, w, nx // 2, 2, np.arange(nx), 2)[0]]

    def shots(_):
        return [a for r in batch.run(jobs)[0] for a in r]

    calls = [model] * len(solvers) + [shots]
    alone = [f(i) for i, f in enumerate(calls)]
    bad = []

    def work(i):
        try:
            for k in range(8):
                if not all(np.array_equal(a, b) for a, b in zip(calls[i](i), alone[i])):
                    bad.append((i, k))
        except Exception as e:  # noqa: BLE001 (reported below)
            bad.append((i, repr(e)))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for s in solvers:
        s.close()
    batch.close()
    assert not bad
