"""Waits that run out, and what is left of them: the report comes with the call that waits for the
stalled steps, every time, and nothing of it is left after a reset.
"""
import numpy as np
import pytest

from conftest import pkg

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
