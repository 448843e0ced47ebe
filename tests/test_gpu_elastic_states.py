"""Which forward states an elastic solver keeps, and that results do not depend on it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NZ, NX, NT, S = 120, 260, 300, 2


def _setup():
    import torch
    from das_gb300.elastic import ElasticSolver2D
    rng = np.random.default_rng(4)
    vs = torch.tensor((1000.0 + 300.0 * rng.random((S, NZ, NX))).astype(np.float32),
                      device="cuda")
    w = rng.standard_normal(NT).astype(np.float32)
    return ElasticSolver2D(NX, NZ, 5.0, 5.0, 5e-4, n_sponge=10), vs, w


def _run(solver, vs, w, grad):
    from das_gb300.elastic import elastic_traces
    v = vs.clone().requires_grad_(grad)
    d = elastic_traces(v, solver, w, [NX // 2, NX // 3], [2, 5], np.arange(2, NX - 2), 4)
    if grad:
        d.square().sum().backward()
    return d.detach().cpu().numpy(), v.grad.cpu().numpy() if grad else None


def test_a_forward_run_without_gradient_keeps_no_states():
    import torch
    states = (NT + 1) * S * 5 * NZ * 288 * 4  # bytes, rows of 288 floats
    solver, vs, w = _setup()
    _run(solver, vs, w[:4], False)  # what the first call loads and allocates
    free0 = torch.cuda.mem_get_info()[0]
    tr0, _ = _run(solver, vs, w, False)
    free1 = torch.cuda.mem_get_info()[0]
    assert free0 - free1 < states // 2
    tr1, g1 = _run(solver, vs, w, True)
    free2 = torch.cuda.mem_get_info()[0]
    assert free1 - free2 > states // 2  # (the states, kept for the gradient)
    tr2, _ = _run(solver, vs, w, False)
    tr3, g3 = _run(solver, vs, w, True)
    solver.close()
    for t in (tr1, tr2, tr3):
        np.testing.assert_array_equal(tr0, t)
    np.testing.assert_array_equal(g1, g3)


def test_results_do_not_depend_on_the_budget():
    """States kept, kept again after they were given up, and checkpoints: the same traces and
    gradients, also over runs of other lengths and batches on one solver."""
    solver, vs, w = _setup()
    ref = _run(solver, vs, w, True)
    short = _run(solver, vs[:1].repeat(2, 1, 1), w[:90], True)
    for budget in (1 << 20, 1 << 33, 0, 1 << 20, 0):
        solver.set_memory_budget(budget)
        got = _run(solver, vs, w, True)
        np.testing.assert_array_equal(got[0], ref[0])
        np.testing.assert_array_equal(got[1], ref[1])
        got = _run(solver, vs[:1].repeat(2, 1, 1), w[:90], True)
        np.testing.assert_array_equal(got[0], short[0])
        np.testing.assert_array_equal(got[1], short[1])
    solver.close()
