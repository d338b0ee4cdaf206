"""Several contexts alive in one process, of unlike sizes: making one changes nothing for another
(a kernel's shared-memory limit belongs to the kernel, not to the context that set it).
"""
import numpy as np
import pytest

from conftest import pkg

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
STEPS = 12


def _mesh(cells, shots, precision):
    ref = precision == "fp64_ref"
    w = pkg.workloads.small_square(n_cells=cells, steps=STEPS, shots=shots)
    return eng.mesh_from_setup(pkg.host.build_setup(w, full=ref), with_ref_ops=ref)


def _load(e):
    rng = np.random.default_rng(1)
    for f in FIELDS:
        e.load(f, rng.standard_normal(e.info[0]["K"] * 6) * (1e-3 if f[0] == "V" else 1e3))


def _fields(e):
    return [e.fetch(f, 0, eng.ALL_SHOTS) for f in FIELDS] + list(e.fetch_traces(0, e.steps_done))


# cells per side of the context made first and of those made after it: about the most elements
# that stay on the SMs, and little ones; every instance of the resident step's kernel
@pytest.mark.parametrize("precision,shots,first,later", [
    ("fp32", 1, 190, (16, 3)), ("fp32_kahan", 1, 160, (16,)), ("fp32", 2, 160, (122, 16)), ("fp32_kahan", 4, 90, (9,)),
    ("fp64", 1, 150, (122, 16)), ("fp64", 1, 122, (16,)), ("fp64_ref", 1, 122, (16,))])
def test_a_later_context_leaves_an_earlier_one_stepping(precision, shots, first, later):
    big = _mesh(first, shots, precision)
    with eng.Engine(big, precision) as e:
        _load(e)
        for _ in range(2):
            e.step(STEPS // 2)
        assert e.stats()["launches"] == 1
        want = _fields(e)
    with eng.Engine(big, precision) as a:
        _load(a)
        a.step(STEPS // 2)
        others = [eng.Engine(_mesh(n, shots, precision), precision) for n in later]
        for o in others:
            o.step(2)
        a.step(STEPS // 2)
        got = _fields(a)
        for o in others:
            o.step(2)
            o.close()
    for x, y in zip(want, got):
        assert np.array_equal(x, y)
    assert np.abs(want[5]).max() > 0
