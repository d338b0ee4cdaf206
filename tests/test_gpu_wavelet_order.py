"""Wavelet updates take effect in the order of their calls, whichever way each travels: up to 64
samples are staged and copied behind the steps enqueued, more go over the second stream ahead of
them.
"""
import numpy as np
import pytest

from conftest import pkg
from stream_capture import Captured

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
LEAD, STEPS = 3000, 3300  # steps in flight while the updates are made, steps in all


def _mesh(cells, shots):
    m = eng.mesh_from_setup(pkg.host.build_setup(pkg.workloads.small_square(n_cells=cells, steps=STEPS, shots=shots), full=False),
                            with_ref_ops=False)
    m["wavelet"] = np.zeros(STEPS)
    return m


def _fields(e):
    return [e.fetch(f, k, eng.ALL_SHOTS) for k in range(len(e.info)) for f in FIELDS]


# (first sample, samples) of the updates, in the order they are made
@pytest.mark.parametrize("updates", [((LEAD, 10), (LEAD, 200)), ((LEAD, 200), (LEAD + 5, 10)),
                                     ((LEAD + 190, 30), (LEAD, 200)), ((LEAD, 64), (LEAD, 65), (LEAD + 3, 64)),
                                     ((LEAD - 5, 20), (LEAD, 100)), ((LEAD, 30), (LEAD + 30, 100), (LEAD, 100))])
@pytest.mark.parametrize("shapes", [((50, 1),), ((9, 1), (20, 4))])
def test_the_last_update_of_a_sample_wins(updates, shapes, monkeypatch):
    monkeypatch.setenv("DG_BATCH_BY_MESH", "1")
    meshes = [_mesh(*s) for s in shapes]
    rng = np.random.default_rng(4)
    values = [rng.standard_normal((len(meshes), n)) * 1e-2 for _, n in updates]
    table = np.zeros((len(meshes), STEPS))
    for (t0, n), v in zip(updates, values):
        table[:, t0:t0 + n] = v
    table[:, :LEAD] = 0.0  # those steps were enqueued before the updates
    with eng.Engine(meshes, "fp32") as a, eng.Engine(meshes, "fp32") as b:
        a.set_wavelet(0, table, eng.ALL_MESHES)
        a.step(STEPS)
        want = _fields(a)
        b.step(3)
        b.reset()  # everything loaded, so that the updates overtake the steps where they can
        b.step_async(LEAD)
        for (t0, n), v in zip(updates, values):
            b.set_wavelet(t0, v, eng.ALL_MESHES)
        b.step(STEPS - LEAD)
        got = _fields(b)
    for x, y in zip(want, got):
        assert np.array_equal(x, y)
    assert np.abs(want[1]).max() > 0


@pytest.mark.parametrize("n", [1, 64, 65])
def test_an_update_inside_a_capture_is_refused(n):
    """An update goes into the wavelet table once, with the call's values: it cannot be part of a
    capture, whatever its length."""
    m = _mesh(9, 1)
    with eng.Engine(m, "fp32") as e, eng.Engine(m, "fp32") as fresh:
        e.set_wavelet(0, np.zeros(1))
        with pytest.raises(eng.DGError):
            with Captured(e) as g:
                e.step_async(1)
                e.set_wavelet(1, np.ones(n))
        g.close()
        e.reset()
        for x in (e, fresh):  # the context works on
            x.set_wavelet(0, np.full(70, 1e-3))
            x.set_wavelet(3, np.full(n, 2e-3))
            x.step(80)
        for a, b in zip(_fields(e), _fields(fresh)):
            assert np.array_equal(a, b)
        assert np.abs(_fields(e)[1]).max() > 0


@pytest.mark.parametrize("n", [40, 200])
@pytest.mark.parametrize("shapes", [((50, 1),), ((20, 4), (50, 1))])
def test_replayed_steps_in_flight_read_the_samples_of_before(n, shapes, monkeypatch):
    """A capture of 500 steps replayed three times reads 1,500 samples, of which the host has counted
    500: an update past those does not overtake the replays."""
    monkeypatch.setenv("DG_BATCH_BY_MESH", "1")
    meshes = [_mesh(*s) for s in shapes]
    table = np.random.default_rng(5).standard_normal((len(meshes), STEPS)) * 1e-3
    with eng.Engine(meshes, "fp32") as a, eng.Engine(meshes, "fp32") as b:
        for e in (a, b):
            e.set_wavelet(0, table, eng.ALL_MESHES)
        a.step(1500)
        with Captured(b) as g:
            b.step_async(500)
        g.launch()
        b.synchronize()
        b.reset()
        b.step(500)
        g.launch(2)
        b.set_wavelet(700, np.full((len(meshes), n), 0.5), eng.ALL_MESHES)
        got = _fields(b)
        g.close()
        for x, y in zip(_fields(a), got):
            assert np.array_equal(x, y)
        assert np.abs(got[1]).max() > 0
