"""Waits that run out, and what is left of them: the report comes with the call that waits for the
stalled steps, every time, and nothing of it is left after a reset.
"""
import numpy as np
import pytest

from conftest import pkg
from stream_capture import Captured

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
STEPS = 30


def _mesh(cells, shots):
    return eng.mesh_from_setup(pkg.host.build_setup(pkg.workloads.small_square(n_cells=cells, steps=STEPS, shots=shots), full=False),
                               with_ref_ops=False)


def _run(e):
    """Fields and traces of a whole run from a loaded state."""
    rng = np.random.default_rng(2)
    for f in FIELDS:
        e.load(f, rng.standard_normal(e.info[0]["K"] * 6) * (1e-3 if f[0] == "V" else 1e3))
    e.step(STEPS)
    return [e.fetch(f, 0, eng.ALL_SHOTS) for f in FIELDS] + list(e.fetch_traces(0, STEPS))


def _timeout(call, *args):
    with pytest.raises(eng.DGError) as ei:
        call(*args)
    assert ei.value.code == -10


def test_reset_forgets_an_unreported_timeout(monkeypatch):
    """Enqueued steps of the resident form whose wait runs out, and a reset before anyone asked."""
    monkeypatch.setenv("DG_RESIDENT_STALL", "1")
    with eng.Engine(_mesh(20, 1), "fp64") as e:
        e.step_async(3)
        e.reset()
        e.synchronize()
        _timeout(e.step, 3)  # the hook still holds one message back


def test_the_wavefront_hook_on_a_context_that_steps_resident():
    """16 shots on a small mesh have a wavefront form beside the resident one: with a unit of it
    stalled, every step call reports the timeout, and with the hook taken back and a reset the
    context steps as a fresh one."""
    m = _mesh(10, 16)
    with eng.Engine(m, "fp32") as e:
        want = _run(e)
    with eng.Engine(m, "fp32") as e:
        e.step(2)
        e.debug_stall_wave(3)
        _timeout(e.step, 3)
        _timeout(e.step_timed, 1)
        e.debug_stall_wave(-1)
        e.reset()
        got = _run(e)
        assert e.stats()["launches"] == 1
    for a, b in zip(want, got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_resident_context_recovers(precision, monkeypatch):
    """After a timeout of the resident step, the hook taken back and a reset, the context steps as a
    fresh one."""
    m = _mesh(20, 1)
    with eng.Engine(m, precision) as e:
        want = _run(e)
    monkeypatch.setenv("DG_RESIDENT_STALL", "1")
    with eng.Engine(m, precision) as e:
        _timeout(e.step, 3)
        e.debug_stall_wave(-1)
        e.reset()
        got = _run(e)
        assert e.stats()["launches"] == 1
    for a, b in zip(want, got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("resident", ["0", "1"])
def test_a_timeout_in_a_replayed_capture_is_reported(resident, monkeypatch):
    """A captured wavefront step that stalls when it is replayed, after the captured call's own
    report was asked for."""
    monkeypatch.setenv("DG_RESIDENT", resident)
    monkeypatch.setenv("DG_WAVE_MIN", "0")
    with eng.Engine(_mesh(10, 16), "fp32") as e:
        with Captured(e) as g:
            e.step_async(2)
        g.launch()
        e.synchronize()
        e.debug_stall_wave(3)
        for _ in range(2):
            g.launch()
            _timeout(e.synchronize)
        e.debug_stall_wave(-1)
        g.launch()
        e.synchronize()
        g.close()
