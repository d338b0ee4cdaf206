"""FP32 shot counts without packed instances of their own (17 to 127 between the powers of two, and
above 128): the resident step, the wavefront step padded to the next count it has, and two launches
with two shots per thread give the same bits; half steps work on an automatic context of such a
count as they did; one (element, shot) per thread with the parsed operators agrees to rounding.
`DG_WAVE_MIN` sets the size from which on the automatic form is the wavefront step, `DG_RESIDENT=0`
keeps the wave field off the SMs.
"""
import numpy as np
import pytest

from conftest import pkg, rel_l2

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
STEPS = 40


def _mesh(cells, shots):
    w = pkg.workloads.small_square(n_cells=cells, steps=STEPS, shots=shots)
    return eng.mesh_from_setup(pkg.host.build_setup(w, full=False), with_ref_ops=False)


def _run(m, precision, halves=False, **kw):
    with eng.Engine(m, precision, **kw) as e:
        rng = np.random.default_rng(5)
        S, K = e.info[0]["S"], e.info[0]["K"]
        for q in {0, 1, S // 2, S - 1}:
            for f in FIELDS:
                e.load(f, rng.standard_normal(K * 6) * (1e-3 if f[0] == "V" else 1e3), 0, q)
        if halves:
            for _ in range(4):
                e.half_step(0)
                e.half_step(1)
            e.step_timed(2)
            e.step(STEPS - 6)
        else:
            e.step(STEPS)
        return e.stats()["kernel_family"], [e.fetch(f, 0, eng.ALL_SHOTS) for f in FIELDS] + list(e.fetch_traces(0, STEPS))


# 17 and 20 share 20 stored shots, 24 a lane count no warp holds whole, 41 pads to 48, 121 to 128;
# 130 has no wavefront form
@pytest.mark.parametrize("cells,shots", [(9, 17), (7, 20), (13, 24), (9, 41), (6, 121), (5, 130)])
@pytest.mark.parametrize("precision", ["fp32", "fp32_kahan"])
def test_every_form_gives_the_same_bits(precision, cells, shots, monkeypatch):
    m = _mesh(cells, shots)
    fam, resident = _run(m, precision)
    assert fam == 1
    monkeypatch.setenv("DG_RESIDENT", "0")
    _, two = _run(m, precision, wavefront=-1)
    monkeypatch.setenv("DG_WAVE_MIN", "0")
    fam, wave = _run(m, precision)
    assert fam == (6 if shots <= 128 else 1)
    _, halves = _run(m, precision, halves=True)
    for a, b, c, d in zip(two, resident, wave, halves):
        assert np.array_equal(a, b) and np.array_equal(a, c) and np.array_equal(a, d)
    _, one = _run(m, precision, variant=1)
    for a, b in zip(two, one):
        assert rel_l2(a, b) <= 2e-5


def test_explicit_requests_are_refused_as_before():
    m = _mesh(8, 24)
    for kw in ({"wavefront": 1}, {"variant": 2}):
        with pytest.raises(eng.DGError) as ei:
            eng.Engine(m, "fp32", **kw)
        assert ei.value.code == -7


def test_small_states_take_two_launches(monkeypatch):
    """16 shots below the wavefront step's size: two launches, the same bits as the wavefront."""
    m = _mesh(10, 16)
    monkeypatch.setenv("DG_RESIDENT", "0")
    fam, two = _run(m, "fp32")
    assert fam == 2
    monkeypatch.setenv("DG_WAVE_MIN", "0")
    fam, wave = _run(m, "fp32")
    assert fam == 6
    for a, b in zip(two, wave):
        assert np.array_equal(a, b)
