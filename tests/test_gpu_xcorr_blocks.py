"""Correlations in a block that another handle used before: same results as the float64
correlation, whatever the block held, its size and the thread that takes it."""
import threading

import numpy as np
import pytest

from oracle import interferometry_oracle as io

pytestmark = pytest.mark.gpu

# samples, channels, receivers, lag seconds: larger and smaller than the one before, sizes
# beside a round of lags and a chunk of samples, one too large to be kept
SIZES = [(1500, 64, 64, 2.0), (37, 8, 3, 0.1), (1025, 40, 33, 0.8), (300, 12, 12, 5.0),
         (6000, 900, 4, 0.3), (1024, 16, 1, 0.07)]


def _one(nt, nch, nr, lag, seed):
    from das_gb300.interferometry import CrossCorrelationStack
    w = np.random.default_rng(seed).standard_normal((nt, nch)).astype(np.float32)
    rec = np.arange(nr)
    st = CrossCorrelationStack(nt, nch, [nch // 2], rec, lag, 0.01)
    st.add(w)
    got = st.result()[nch // 2][0]
    st.close()
    ex = io.correlation_exact(w, nch // 2, lag, 0.01, rec)
    # one rounding to float32 of a sum exact to 44 bits
    return np.linalg.norm(got - ex) / np.linalg.norm(ex)


@pytest.mark.parametrize("order", [1, -1])
def test_reused_blocks(order):
    for k, size in enumerate(SIZES[::order] + SIZES):
        assert _one(*size, seed=k) < 1e-7, size


def test_reused_blocks_from_threads():
    errs = {}

    def work(i):
        for k in range(6):
            errs[i, k] = _one(*SIZES[(i + k) % 4], seed=10 * i + k)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert len(errs) == 24 and max(errs.values()) < 1e-7
