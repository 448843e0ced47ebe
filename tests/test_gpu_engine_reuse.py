"""One engine over shots whose geometry changes from call to call -- source cell, receiver row,
first column, columns shared or not -- at equal length and receiver count, so that whatever an
engine keeps from one shot (captured passes, packets, tables) meets the next one's geometry.
Each result equals that of a fresh engine's step kernels, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NZ, NX, N_REC = 90, 330, 64
# receiver row and columns of equal count
LINES = [(2, np.arange(3, 3 + N_REC)), (7, np.arange(40, 40 + N_REC)),
         (2, np.arange(N_REC) // 2 * 3 + 10), (NZ - 4, np.arange(NX - 1, NX - 1 - N_REC, -1)),
         (1, np.arange(3, 3 + N_REC)), (5, np.arange(0, 4 * N_REC, 4)),
         (2, np.arange(3, 3 + N_REC))]


@pytest.mark.parametrize("storage", ["all", "checkpoint"])
@pytest.mark.parametrize("source", [(NX // 2, 1), (1, 6), (NX - 2, 6), (NX // 2, NZ - 2),
                                    (NX // 2, 0), (NX // 2, 2)])
@pytest.mark.parametrize("nt", [2, 60])
def test_migrations_of_changing_lines(storage, source, nt):
    from das_gb300.rtm_engine import TSWRTMEngine
    from das_gb300.velocity_flood import FloodModels
    from das_gb300.wave_solver import WaveSolver2D
    rng = np.random.default_rng(nt)
    v = rng.uniform(1500, 3000, (NZ, NX)).astype(np.float32)
    fm = FloodModels(v, v, (v * np.float32(1.02)).astype(np.float32), 0, 0)
    kept = WaveSolver2D(NX, NZ, 5.0, 5.0, 5e-4, n_sponge=12)
    eng = TSWRTMEngine(kept, storage)
    for k, (row, cols) in enumerate(LINES + LINES):
        w = rng.standard_normal(nt).astype(np.float32)
        d = rng.standard_normal((nt, N_REC)).astype(np.float32)
        got = eng.migrate_shot(fm, w, *source, d, cols, row, 2)
        fresh = WaveSolver2D(NX, NZ, 5.0, 5.0, 5e-4, n_sponge=12)
        fresh.set_launch("grid", False)
        fresh.set_graphs(False)
        ref = TSWRTMEngine(fresh, storage).migrate_shot(fm, w, *source, d, cols, row, 2)
        fresh.close()
        np.testing.assert_array_equal(got[0], ref[0], err_msg=f"image, shot {k}")
        np.testing.assert_array_equal(got[1], ref[1], err_msg=f"illumination, shot {k}")
    kept.close()


@pytest.mark.parametrize("source", [(NX // 2, 1), (1, 6), (NX // 2, 2)])
def test_modelling_and_correlation_of_changing_lines(source):
    from das_gb300.wave_solver import WaveSolver2D
    nt = 50
    rng = np.random.default_rng(3)
    v = rng.uniform(1500, 3000, (NZ, NX)).astype(np.float32)
    kept = WaveSolver2D(NX, NZ, 5.0, 5.0, 5e-4, n_sponge=12)
    for k, (row, cols) in enumerate(LINES + LINES):
        w = rng.standard_normal(nt).astype(np.float32)
        d = rng.standard_normal((nt, N_REC)).astype(np.float32)
        fresh = WaveSolver2D(NX, NZ, 5.0, 5.0, 5e-4, n_sponge=12)
        fresh.set_launch("grid", False)
        fresh.set_graphs(False)
        res = []
        for s in (kept, fresh):
            rec, snaps = s.forward_propagate_acoustic(v, w, *source, cols, row, True, 2)
            img = np.zeros((NZ, NX), np.float32)
            s.backward_propagate_and_correlate(v, d, cols, row, snaps, img, 2)
            res.append((rec, snaps, img))
        fresh.close()
        for a, b in zip(*res):
            np.testing.assert_array_equal(a, b, err_msg=f"call {k}")
    kept.close()


def test_gradient_after_its_states_were_given_back():
    """The states kept for a gradient, given back before it (a budget below them), and a second
    gradient of one forward run: the same bit for bit."""
    import torch
    from das_gb300.autograd import model_traces
    from das_gb300.wave_solver import WaveSolver2D
    nt = 200
    rng = np.random.default_rng(8)
    v = rng.uniform(1500, 3000, (NZ, NX)).astype(np.float32)
    w = rng.standard_normal(nt).astype(np.float32)
    rix = np.arange(2, NX - 2, 2)
    r = torch.tensor(rng.standard_normal((nt, len(rix))).astype(np.float32), device="cuda")
    s = WaveSolver2D(NX, NZ, 5.0, 5.0, 5e-4, n_sponge=12)
    grads = []
    for give_back in (False, True):
        vt = torch.tensor(v, device="cuda", requires_grad=True)
        d = model_traces(vt, s, w, NX // 3, 2, rix, 2)
        if give_back:
            assert s._lib.w2d_engine_set_memory_budget(s._eng(), 8 << 20) == 0
        for _ in range(2):
            grads.append(torch.autograd.grad(d, vt, r, retain_graph=True)[0].cpu().numpy())
    s.close()
    assert np.abs(grads[0]).max() > 0
    for g in grads[1:]:
        np.testing.assert_array_equal(grads[0], g)


@pytest.mark.parametrize("pdl", [True, False])
@pytest.mark.parametrize("segment", [0, 25, 1000])
def test_gradient_after_other_calls(pdl, segment):
    """Calls with other models, lengths and receivers between a forward run and its gradient:
    the gradient is that of its own run, bit for bit."""
    import torch
    from das_gb300.autograd import model_traces
    from das_gb300.rtm_engine import TSWRTMEngine
    from das_gb300.velocity_flood import FloodModels
    from das_gb300.wave_solver import WaveSolver2D
    nt = 120
    rng = np.random.default_rng(9)
    v, v2 = (rng.uniform(1500, 3000, (NZ, NX)).astype(np.float32) for _ in range(2))
    w, w2 = (rng.standard_normal(n).astype(np.float32) for n in (nt, 40))
    rix = np.arange(4, NX - 4, 9)
    r = torch.tensor(rng.standard_normal((nt, len(rix))).astype(np.float32), device="cuda")
    d2 = rng.standard_normal((40, NX)).astype(np.float32)
    s = WaveSolver2D(NX, NZ, 5.0, 5.0, 5e-4, n_sponge=12)
    s.set_launch("grid", pdl)
    s.set_checkpoint_segment(segment)
    grads = []
    for between in (0, 1, 2, 3):
        vt = torch.tensor(v, device="cuda", requires_grad=True)
        d = model_traces(vt, s, w, NX // 3, 2, rix, 3)
        if between & 1:
            s.forward_propagate_acoustic(v2, w2, 50, 1, np.arange(NX), 2)
        if between & 2:
            TSWRTMEngine(s, "checkpoint").migrate_shot(FloodModels(v2, v2, v2, 0, 0), w2, 70, 4,
                                                       d2, np.arange(NX), 5, 2)
        d.backward(r)
        grads.append(vt.grad.cpu().numpy())
    s.close()
    assert np.abs(grads[0]).max() > 0
    for g in grads[1:]:
        np.testing.assert_array_equal(grads[0], g)
