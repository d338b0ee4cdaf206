"""Which step comes next: every form of the step takes it from the same place, so calls that run
different forms, and steps that the caller captured and replays, follow one another.
"""
import numpy as np
import pytest

from conftest import pkg
from stream_capture import Captured

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
STEPS = 60


def _mesh(cells, shots):
    return eng.mesh_from_setup(pkg.host.build_setup(pkg.workloads.small_square(n_cells=cells, steps=STEPS, shots=shots), full=False),
                               with_ref_ops=False)


def _load(e):
    rng = np.random.default_rng(6)
    for k, info in enumerate(e.info):
        for f in FIELDS:
            e.load(f, rng.standard_normal(info["K"] * 6) * (1e-3 if f[0] == "V" else 1e3), k, info["S"] - 1)


def _fields(e):
    return [e.fetch(f, k, eng.ALL_SHOTS) for k in range(len(e.info)) for f in FIELDS]


def _straight(meshes, precision, **kw):
    with eng.Engine(meshes, precision, **kw) as e:
        _load(e)
        e.step(STEPS)
        return _fields(e) + list(e.fetch_traces(0, STEPS, eng.ALL_MESHES))


@pytest.mark.parametrize("precision", ["fp32", "fp32_kahan"])
@pytest.mark.parametrize("how", ["cache", "environment"])
def test_timed_steps_after_resident_ones(precision, how, tmp_path, monkeypatch):
    """16 shots on a small mesh: dg_gpu_step stays on the SMs, timed, profiled and captured steps take
    the wavefront form, here the one that counts its steps by its tickets (a tuned choice)."""
    m = _mesh(10, 16)
    want = _straight(m, precision)
    kw = {}
    if how == "cache":
        cache = tmp_path / "tune.txt"
        cache.write_text("p%d_m1_K200_KS3200_w1 64 0 12\n" % eng.PRECISIONS[precision])
        kw = {"autotune": True, "tune_cache": str(cache)}
    else:
        monkeypatch.setenv("DG_WAVE_PERSISTENT", "0")
    with eng.Engine(m, precision, **kw) as e:
        assert e.stats()["kernel_family"] == 5
        _load(e)
        e.step(10)
        assert e.stats()["launches"] == 1
        e.step_timed(2)
        e.step(5)
        e.step_profiled(3)
        e.step_timed(1)
        with Captured(e) as g:
            e.step_async(4)
        g.launch()
        e.step(STEPS - 25)
        got = _fields(e) + list(e.fetch_traces(0, STEPS, eng.ALL_MESHES))
        g.close()
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
    assert np.abs(want[-1]).max() > 0


# one mesh whose own steps stay on the SMs (one shot; 16, whose captured steps are wavefronts; 3), two
# launches a step, a padded wavefront, a batch stepped mesh by mesh
REPLAYS = [([(10, 1)], "fp32", {}), ([(10, 1)], "fp64", {}), ([(10, 16)], "fp32", {}), ([(12, 3)], "fp32_kahan", {}),
           ([(10, 1)], "fp64", {"DG_RESIDENT": "0"}), ([(10, 24)], "fp32", {"DG_RESIDENT": "0", "DG_WAVE_MIN": "0"}),
           ([(9, 1), (12, 4), (5, 2)], "fp32", {"DG_BATCH_BY_MESH": "1"})]


@pytest.mark.parametrize("shapes,precision,env", REPLAYS)
@pytest.mark.parametrize("n", [1, 7])
def test_steps_after_replays(shapes, precision, env, n, monkeypatch):
    """A capture of n steps replayed three times, then steps through the engine: they go on where the
    replays ended (the host counts a captured call once)."""
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    meshes = [_mesh(*s) for s in shapes]
    with eng.Engine(meshes, precision) as e:
        _load(e)
        e.step(2 + 3 * n + 20)
        want = _fields(e)
    with eng.Engine(meshes, precision) as e:
        _load(e)
        e.step(2)
        with Captured(e) as g:
            e.step_async(n)
        g.launch(3)
        e.step(20)
        assert e.steps_done == 2 + n + 20
        got = _fields(e)
        g.close()
        # what lies past the table by the device's count is skipped there, and a reset starts anew
        e.step(STEPS - e.steps_done)
        assert all(np.isfinite(a).all() for a in _fields(e))
        e.reset()
        _load(e)
        e.step(2 + 3 * n + 20)
        again = _fields(e)
    for a, b, c in zip(want, got, again):
        assert np.array_equal(a, b) and np.array_equal(a, c)
    assert np.abs(want[0]).max() > 0


@pytest.mark.parametrize("shapes,precision,env", REPLAYS)
def test_traces_after_replays(shapes, precision, env, monkeypatch):
    """Traces of any window are to be had after a capture and its replays: of the captured call's
    steps, of those before, and of those after it."""
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    meshes, n = [_mesh(*s) for s in shapes], 7
    with eng.Engine(meshes, precision) as a, eng.Engine(meshes, precision) as e:
        _load(a)
        _load(e)
        a.step(2 + n + 20)
        e.step(2)
        with Captured(e) as g:
            e.step_async(n)
        g.launch()
        for t0, steps in ((2, n), (0, 2), (0, 2 + n)):
            for x, y in zip(a.fetch_traces(t0, steps, eng.ALL_MESHES), e.fetch_traces(t0, steps, eng.ALL_MESHES)):
                assert np.array_equal(x, y)
        e.step(20)
        for t0, steps in ((0, 2 + n), (2, n + 20), (0, 2 + n + 20)):
            for x, y in zip(a.fetch_traces(t0, steps, eng.ALL_MESHES), e.fetch_traces(t0, steps, eng.ALL_MESHES)):
                assert np.array_equal(x, y)
        g.close()
