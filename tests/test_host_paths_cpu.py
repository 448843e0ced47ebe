"""What the engines' host code launches, captures and allocates, on a stand-in CUDA runtime
(no GPU, no arithmetic)."""
import ctypes

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


def _elastic_forward(lib, h, nz, nx, nt, n_shots):
    """One forward call on stand-in device arrays."""
    p = np.zeros(1, np.float32)
    w = np.zeros((n_shots, nt), np.float32)
    six, siz = np.full(n_shots, nx // 2, np.int32), np.full(n_shots, 2, np.int32)
    rix = np.arange(2, nx - 2, dtype=np.int32)
    return lib.w2d_elastic_forward_batch(h, n_shots, *[p.ctypes.data] * 4, w.ctypes.data, nt,
                                         six.ctypes.data, siz.ctypes.data, rix.ctypes.data,
                                         len(rix), 4, p.ctypes.data)


def test_elastic_executor_stays_within_its_budget(fake):
    """A worker's solver holds no more than the budget its batches are sized by, over batches
    of one to four shots and of several lengths, whatever memory is free."""
    from types import SimpleNamespace
    from das_gb300.elastic import ElasticExecutor
    nz, nx = 363, 725
    ex = object.__new__(ElasticExecutor)
    ex.budget, ex._solvers = 2 << 30, {}
    s = ex._solver(SimpleNamespace(nx=nx, nz=nz, dx=5.0, dz=5.0, dt=5e-4, n_sponge=30,
                                   sponge_alpha=0.0015, free_surface_top=True))
    base = fake.fake_used()
    for n_shots, nt in [(1, 100), (4, 700), (1, 250), (1, 3000), (2, 100), (4, 700), (1, 100)]:
        per = fake.w2d_elastic_shot_bytes(nx, nz, nt, nx - 4)
        assert n_shots * per <= ex.budget
        fake_device.counts(fake)
        assert _elastic_forward(fake, s._h, nz, nx, nt, n_shots) == 0
        # (tables of columns and checkpoints of other lengths beside it)
        assert fake.fake_used() - base <= ex.budget + (600 << 20), (n_shots, nt)
    s.close()


def test_elastic_states_go_back(fake):
    """Kept states are bounded and given back: by a budget below them, by a run whose states
    do not fit, and with the solver."""
    from das_gb300.elastic import ElasticSolver2D
    nz, nx, nt = 363, 725, 700
    states = (nt + 1) * 5 * nz * 736 * 4
    start = fake.fake_used()
    s = ElasticSolver2D(nx, nz, 5.0, 5.0, 5e-4)
    assert _elastic_forward(fake, s._h, nz, nx, nt, 1) == 0
    assert fake.fake_used() - start > states
    s.set_memory_budget(1 << 30)
    assert fake.fake_used() - start < states // 8
    assert _elastic_forward(fake, s._h, nz, nx, nt, 1) == 0
    assert fake.fake_used() - start <= 1 << 30
    s.set_memory_budget(0)
    assert _elastic_forward(fake, s._h, nz, nx, nt, 1) == 0
    assert fake.fake_used() - start > states
    assert _elastic_forward(fake, s._h, nz, nx, 20000, 1) == 0  # 107 GB of states
    assert fake.fake_used() - start < states
    s.close()
    assert fake.fake_used() == start


def _fwi_forward(lib, solver, nt, n_rec=4):
    """One forward call of the gradient path on stand-in device arrays."""
    p, w = np.zeros(1, np.float32), np.zeros(nt, np.float32)
    rix = np.arange(2, 2 + n_rec, dtype=np.int32)
    return lib.w2d_fwi_forward(solver._eng(), p.ctypes.data, w.ctypes.data, nt, solver.nx // 2, 2,
                               rix.ctypes.data, n_rec, 2, p.ctypes.data)


def test_kept_states_make_room_for_snapshots(fake):
    """The forward states that the gradient path keeps by its own choice do not count against
    a migration's snapshots on the same engine: what fits an engine without them still runs,
    and a gradient asked for afterwards recomputes its states."""
    from das_gb300.rtm_engine import TSWRTMEngine
    from das_gb300.velocity_flood import FloodModels
    from das_gb300.wave_solver import WaveSolver2D
    nz, nx, nt = 1000, 4000, 1500
    s = WaveSolver2D(nx, nz, 5.0, 5.0, 5e-4)
    v = _vel(nz, nx)
    s.forward_propagate_acoustic(v, np.zeros(10, np.float32), nx // 2, 2, np.arange(4), 2)
    base = fake.fake_used()
    assert _fwi_forward(fake, s, nt) == 0
    assert fake.fake_used() - base > nt * nz * nx * 4  # 24 GB
    n = 13800  # 221 GB of snapshots: 80 % of the memory beside the states is 211 GB, of all 230
    w, d = np.zeros(n, np.float32), np.zeros((n, 4), np.float32)
    for storage in ("all", "auto"):
        TSWRTMEngine(s, storage).migrate_shot(FloodModels(v, v, v, 0, 0), w, nx // 2, 2, d,
                                              np.arange(4), 2, 1)
        assert s.last_stats()["storage"] == "all"
    s.close()

    # and a gradient after the states were given back
    assert _fwi_forward(fake, s, nt) == 0
    kept = fake.fake_used()
    _lib_check(fake, fake.w2d_engine_set_memory_budget(s._eng(), 1 << 30))
    assert kept - fake.fake_used() >= nt * nz * nx * 4
    p = np.zeros(1, np.float32)
    fake_device.counts(fake)
    _lib_check(fake, fake.w2d_fwi_gradient(s._eng(), p.ctypes.data, p.ctypes.data))
    assert fake_device.counts(fake)["cooperative"] > 2
    assert fake.fake_used() - base < nt * nz * nx * 4 // 2
    # the budget bounds the next forward call too, and a run that does not fit keeps none
    assert _fwi_forward(fake, s, nt) == 0 and fake.fake_used() - base < nt * nz * nx * 4 // 2
    _lib_check(fake, fake.w2d_engine_set_memory_budget(s._eng(), 0))
    assert _fwi_forward(fake, s, nt) == 0 and fake.fake_used() - base > nt * nz * nx * 4
    assert _fwi_forward(fake, s, 8000) == 0 and fake.fake_used() - base < nt * nz * nx * 4 // 2
    s.close()


def _lib_check(lib, rc):
    assert rc == 0, lib.w2d_last_error()


class _ShotHead(ctypes.Structure):
    """The first fields of the resident kernel's RsShot."""
    _fields_ = [(n, ctypes.c_int) for n in ("nx", "nz", "ldx", "gx", "gz", "maxc", "maxr")] + \
               [("inv_dx2", ctypes.c_float), ("inv_dz2", ctypes.c_float), ("fs", ctypes.c_int),
                ("n_sponge", ctypes.c_int), ("lut", ctypes.c_void_p)] + \
               [(n, ctypes.c_int) for n in ("src_ix", "src_iz", "rec_iz", "n_rec", "rec_c0")]


@pytest.mark.parametrize("segment", [0, 25, 1000])
def test_gradient_after_other_calls_uses_its_own_receivers(fake, segment):
    """The residuals of a gradient are (nt, n_rec) of its own forward run: with the receivers
    of a call in between, the adjoint would index them past their end."""
    from das_gb300.wave_solver import WaveSolver2D
    nz, nx, nt = 150, 700, 300
    s = WaveSolver2D(nx, nz, 5.0, 5.0, 5e-4)
    s.set_checkpoint_segment(segment)
    assert _fwi_forward(fake, s, nt) == 0
    s.forward_propagate_acoustic(_vel(nz, nx), np.zeros(10, np.float32), 100, 7, np.arange(nx), 9)
    head, p = _ShotHead(), np.zeros(1, np.float32)
    for _ in range(2):
        _lib_check(fake, fake.w2d_fwi_gradient(s._eng(), p.ctypes.data, p.ctypes.data))
        fake.fake_last_cooperative(ctypes.byref(head), ctypes.sizeof(head))
        assert (head.nx, head.nz, head.n_rec, head.rec_iz, head.rec_c0) == (nx, nz, 4, 2, 2)
    s.close()


def test_tune_plain_times_the_step_kernels(fake, tmp_path, monkeypatch):
    """A grid that fits the chip ignores the tile unless the call runs one launch per step:
    the tiles are timed on such a call."""
    from das_gb300 import autotune
    from das_gb300.wave_solver import WaveSolver2D
    monkeypatch.setenv("DAS_GB300_TUNE_CACHE", str(tmp_path / "tune.json"))
    s = WaveSolver2D(400, 150, 5.0, 5.0, 5e-4)
    autotune.tune_plain(s, _vel(150, 400), nt_sample=50)
    n = fake_device.counts(fake)
    assert n["cooperative"] == 0 and n["graph"] == 2 * len(autotune.PLAIN_TILES)
    s.close()


def test_tune_batch_compares_tiles_on_step_kernels(tmp_path, monkeypatch):
    """Where the shots run on chip in the grid form (no two receivers in a column) the times of
    its tiles differ by noise alone: the tile is the one that is fastest in step kernels."""
    import das_gb300.batch as batch
    from das_gb300 import autotune
    from das_gb300.batch import ShotJob
    monkeypatch.setenv("DAS_GB300_TUNE_CACHE", str(tmp_path / "tune.json"))
    noise = iter([1.0, 1.02, 1.01] + [1.0] * 100)

    class StandIn:
        def __init__(self, arena_bytes, max_shots, tile, steps_per_launch, launches_per_graph,
                     form):
            self.form, self.tile = form, tuple(tile)

        def run(self, jobs):
            shared = any(len(set(np.asarray(j.receiver_ix).tolist())) < len(j.receiver_ix)
                         for j in jobs)
            for j in jobs:
                assert j.data.shape == (len(j.wavelet), len(j.receiver_ix))
            if self.form == "queue":
                ms = 9.0
            elif shared:
                ms = {(4, 4): 3.0, (8, 4): 2.5, (4, 8): 4.0}[self.tile]
            else:
                ms = next(noise) if len(jobs) > 2 else 1.0
            return [], {"counted_points": 1e6 * len(jobs), "device_ms": ms}

        def close(self):
            pass

    monkeypatch.setattr(batch, "BatchEngine", StandIn)
    v = _vel(40, 60)
    for n_rec in (60, 0):
        jobs = [ShotJob(60, 40, 5.0, 5.0, 5e-4, v, v, np.zeros(99, np.float32),
                        np.zeros((99, n_rec), np.float32), np.arange(n_rec), 30, 2, 2, 2, 10,
                        0.0015, True) for _ in range(5)]
        cfg, table = autotune.tune_batch(jobs, use_cache=False)
        assert cfg == ((8, 4), 16, 16, "grid") and len(table) == len(autotune.BATCH_CANDIDATES)


@pytest.mark.parametrize("nt", [1, 2, 5, 6, 40])
def test_short_passes_keep_the_step_kernels(fake, nt):
    """Loading a grid onto the chip costs more than a few launches."""
    from das_gb300.rtm_engine import TSWRTMEngine
    from das_gb300.velocity_flood import FloodModels
    from das_gb300.wave_solver import WaveSolver2D
    nz, nx = 150, 400
    s = WaveSolver2D(nx, nz, 5.0, 5.0, 5e-4)
    v, w, d = _vel(nz, nx), np.zeros(nt, np.float32), np.zeros((nt, nx), np.float32)
    s.forward_propagate_acoustic(v, w, nx // 2, 2, np.arange(nx), 2)
    n = fake_device.counts(fake)
    assert (n["cooperative"], n["captures"]) == ((1, 0) if nt >= 6 else (0, 1))
    TSWRTMEngine(s, "all").migrate_shot(FloodModels(v, v, v, 0, 0), w, nx // 2, 2, d,
                                        np.arange(nx), 2, 2)
    n = fake_device.counts(fake)
    assert (n["cooperative"], n["captures"]) == ((2, 0) if nt >= 6 else (0, 2))
    _lib_check(fake, _fwi_forward(fake, s, nt))
    p = np.zeros(1, np.float32)
    _lib_check(fake, fake.w2d_fwi_gradient(s._eng(), p.ctypes.data, p.ctypes.data))
    assert (fake_device.counts(fake)["cooperative"] > 0) == (nt >= 6)
    s.close()
