"""A batch stepped mesh by mesh keeps the context stream's order: what a caller enqueues there (a
replayed capture of steps) comes before the calls made after it.
"""
import numpy as np
import pytest

from conftest import pkg
from stream_capture import Captured

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
SHAPES, STEPS, N = ((70, 4), (50, 2), (9, 1)), 400, 150


@pytest.fixture
def context(monkeypatch):
    """The batch after a replayed capture of N steps, nothing waited for, and the batch after N steps."""
    monkeypatch.setenv("DG_BATCH_BY_MESH", "1")
    meshes = [eng.mesh_from_setup(pkg.host.build_setup(pkg.workloads.small_square(n_cells=n, steps=STEPS, shots=s), full=False),
                                  with_ref_ops=False) for n, s in SHAPES]

    def load(e):
        rng = np.random.default_rng(7)
        for k, info in enumerate(e.info):
            for f in FIELDS:
                e.load(f, rng.standard_normal(info["K"] * 6) * (1e-3 if f[0] == "V" else 1e3), k, 0)

    with eng.Engine(meshes, "fp32") as a, eng.Engine(meshes, "fp32") as b:
        assert a.stats()["kernel_family"] == 9
        load(a)
        load(b)
        b.step(N)
        with Captured(a) as g:
            a.step_async(N)
        g.launch()
        a.synchronize()
        a.reset()
        load(a)
        with Captured(a) as g2:
            a.step_async(N)
        g2.launch()
        yield a, b
        a.synchronize()
        g.close()
        g2.close()


def _same(a, b, steps=N):
    for k in range(len(SHAPES)):
        for f in FIELDS:
            assert np.array_equal(a.fetch(f, k, 0), b.fetch(f, k, 0))
    for x, y in zip(a.fetch_traces(0, steps, eng.ALL_MESHES), b.fetch_traces(0, steps, eng.ALL_MESHES)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("mesh", range(len(SHAPES)))
def test_a_field(context, mesh):
    a, b = context
    assert np.array_equal(a.fetch("Txx", mesh, 0), b.fetch("Txx", mesh, 0))


@pytest.mark.parametrize("mesh", [eng.ALL_MESHES, 0, 2])
def test_traces(context, mesh):
    a, b = context
    for x, y in zip(a.fetch_traces(0, N, mesh), b.fetch_traces(0, N, mesh)):
        assert np.array_equal(x, y)


def test_a_loaded_field(context):
    a, b = context
    for e in (a, b):
        e.load("Txz", np.arange(e.info[0]["K"] * 6) * 1.0, 0, 0)
    _same(a, b)


@pytest.mark.parametrize("n", [20, 100])
def test_samples_that_enqueued_steps_read(context, n):
    a, b = context
    for e in (a, b):
        e.set_wavelet(10, np.full((len(SHAPES), n), 5.0), eng.ALL_MESHES)
        e.step(7)
    _same(a, b, N + 7)


def test_a_reset(context):
    a, _ = context
    a.reset()
    for k in range(len(SHAPES)):
        assert not np.any(a.fetch("Txx", k, 0))
