"""What the engines' host code launches, captures and allocates, on a stand-in CUDA runtime
(no GPU, no arithmetic)."""
import numpy as np
import pytest

import fake_device


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    return fake_device.load(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def fake(fake_lib, monkeypatch):
    """The library as the package's own for one test, on a device of 288 GB."""
    from das_gb300 import _lib
    monkeypatch.setattr(_lib, "_LIB", fake_lib)
    fake_lib.fake_set_total(288 << 30)
    fake_device.counts(fake_lib)
    return fake_lib


def _vel(nz, nx):
    return np.full((nz, nx), 2000.0, np.float32)


# source cells (ix, iz) of a 180 x 700 grid: interior; rows and columns that the resident loop
# does not take as a source's
SOURCES = [(350, 2), (350, 0), (350, 1), (350, 178), (350, 179), (0, 5), (1, 5), (698, 5), (699, 5)]


@pytest.mark.parametrize("storage", ["all", "checkpoint"])
@pytest.mark.parametrize("source", SOURCES)
@pytest.mark.parametrize("line", ["all", "shared column", "row 1"])
def test_no_resident_launch_is_captured(fake, storage, source, line):
    """A captured pass is replayed for other shots: a launch that holds its shot's geometry by
    value must not be in it, whatever form the passes of a migration take."""
    from das_gb300.rtm_engine import TSWRTMEngine
    from das_gb300.velocity_flood import FloodModels
    from das_gb300.wave_solver import WaveSolver2D
    nz, nx, nt = 180, 700, 60
    rix = np.zeros(nx, int) + 5 if line == "shared column" else np.arange(nx)
    s = WaveSolver2D(nx, nz, 5.0, 5.0, 5e-4, n_sponge=20)
    e = TSWRTMEngine(s, storage)
    v, w, d = _vel(nz, nx), np.zeros(nt, np.float32), np.zeros((nt, nx), np.float32)
    for _ in range(2):
        e.migrate_shot(FloodModels(v, v, v, 0, 0), w, *source, d, rix, 1 if line == "row 1" else 2,
                       2)
    s.close()
    n = fake_device.counts(fake)
    assert n["captured_cooperative"] == 0
    if line == "all" and source == SOURCES[0]:
        assert n["cooperative"] >= 4 and n["captures"] == 0
    if line != "all":
        assert n["cooperative"] == 0 and n["captures"] == 2 and n["graph"] == 4


class _Fetched:
    """The C entry that copies results back, as calls that reached it."""

    def __init__(self):
        self.calls = 0

    def w2d_batch_fetch(self, *args):
        self.calls += 1
        return 0


@pytest.mark.parametrize("make", [
    lambda: np.empty((4, 6), np.float32),                    # smaller
    lambda: np.empty((6, 5), np.float32),                    # transposed
    lambda: np.empty((5, 6), np.float64),
    lambda: np.empty((5, 6), np.float16),
    lambda: np.empty((5, 12), np.float32)[:, ::2],           # strided
    lambda: np.empty((6, 5), np.float32).T,                  # other order
    lambda: np.empty(30, np.float32),                        # one dimension
    lambda: np.broadcast_to(np.float32(0), (5, 6)),          # read-only
    lambda: [[0.0] * 6] * 5,
])
@pytest.mark.parametrize("place", [0, 1])
def test_fetch_refuses_arrays_that_the_copy_would_overrun(make, place):
    from das_gb300.batch import BatchEngine
    eng = object.__new__(BatchEngine)
    eng._lib, eng._h = _Fetched(), None
    ok = [np.empty((5, 6), np.float32), np.empty((5, 6), np.float32)]
    out = list(ok)
    out[place] = make()
    with pytest.raises(ValueError):
        eng.fetch(0, 5, 6, out)
    assert eng._lib.calls == 0
    got = eng.fetch(0, 5, 6, ok)
    assert got[0] is ok[0] and got[1] is ok[1] and eng._lib.calls == 1
    assert eng.fetch(0, 5, 6)[0].shape == (5, 6)


def test_batch_without_memory_for_the_waves_runs_step_kernels(fake):
    """The waves' packet table is wanted when jobs run, after the arena took its memory:
    without it every shot advances by step kernels, and on chip again when there is room."""
    from das_gb300.batch import BatchEngine, ShotJob
    nz, nx, nt = 600, 2000, 40
    v, w, d = _vel(nz, nx), np.zeros(nt, np.float32), np.zeros((nt, nx), np.float32)
    jobs = [ShotJob(nx, nz, 5.0, 5.0, 5e-4, v, v, w, d, np.arange(nx), nx // 2, 2, 2, 2, 10,
                    0.0015, True) for _ in range(3)]
    eng = BatchEngine(arena_bytes=4 << 30, max_shots=8)
    fake.fake_set_total(fake.fake_used() + (1 << 20))
    fake_device.counts(fake)
    res, _ = eng.run(jobs)
    n = fake_device.counts(fake)
    assert len(res) == 3 and n["cooperative"] == 0 and n["graph"] > 0 and n["captures"] > 0
    fake.fake_set_total(288 << 30)
    res, _ = eng.run(jobs)
    n = fake_device.counts(fake)
    assert len(res) == 3 and n["cooperative"] > 0 and n["captured_cooperative"] == 0
    eng.close()
