"""Which form a context takes, asserted where another form would give the same bits: the resident
step up to the lanes its kernels hold, and the autotuner's schedules of the forms that are tuned.
"""
import numpy as np
import pytest

from conftest import pkg

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
STEPS = 30
# lanes a block of the resident step holds, by precision and whether a lane is one shot
LANES = {("fp64", True): 384, ("fp64", False): 384, ("fp64_ref", True): 256, ("fp64_ref", False): 256,
         ("fp32", True): 512, ("fp32", False): 384, ("fp32_kahan", True): 384, ("fp32_kahan", False): 256}


def _mesh(cells, shots, precision):
    ref = precision == "fp64_ref"
    w = pkg.workloads.small_square(n_cells=cells, steps=STEPS, shots=shots)
    return eng.mesh_from_setup(pkg.host.build_setup(w, full=ref), with_ref_ops=ref)


def _run(m, precision, **kw):
    with eng.Engine(m, precision, **kw) as e:
        rng = np.random.default_rng(3)
        for s in {0, e.info[0]["S"] - 1}:
            for f in FIELDS:
                e.load(f, rng.standard_normal(e.info[0]["K"] * 6) * (1e-3 if f[0] == "V" else 1e3), 0, s)
        e.step(STEPS)
        stats = e.stats()
        return stats, [e.fetch(f, 0, eng.ALL_SHOTS) for f in FIELDS] + list(e.fetch_traces(0, STEPS))


@pytest.mark.parametrize("precision,cells,shots", [
    ("fp64", 168, 1), ("fp64", 169, 1), ("fp64", 118, 2), ("fp64", 119, 2), ("fp32", 194, 1), ("fp32", 195, 1), ("fp32", 168, 2),
    ("fp32", 169, 2), ("fp32_kahan", 168, 1), ("fp32_kahan", 169, 1), ("fp32_kahan", 136, 2), ("fp32_kahan", 138, 2),
    ("fp64_ref", 136, 1), ("fp64_ref", 138, 1)])
def test_the_resident_step_up_to_its_last_lane(precision, cells, shots, monkeypatch):
    """Just below and just above the most lanes: one launch for all steps there, two launches a
    step here, the same bits as with the resident step off."""
    m = _mesh(cells, shots, precision)
    stats, got = _run(m, precision)
    lanes = shots if precision.startswith("fp64") or shots == 1 else (shots + 1) // 2
    per_sm = -(-2 * cells * cells // 148) * lanes  # the most a block holds
    assert (stats["launches"] == 1) == bool(stats["resident"]) == (per_sm <= LANES[precision, shots == 1])
    assert stats["launches"] in (1, 2 * STEPS)
    monkeypatch.setenv("DG_RESIDENT", "0")
    stats, want = _run(m, precision)
    assert not stats["resident"] and stats["launches"] == 2 * STEPS
    for a, b in zip(want, got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision,shots,family", [("fp32", 16, (5, 6)), ("fp32_kahan", 16, (5, 6)), ("fp32", 24, (6,)),
                                                    ("fp64", 3, (1,)), ("fp32", 4, (7,)), ("fp32", 1, (3,))])
def test_tuned_schedules_give_the_same_bits(precision, shots, family, tmp_path, monkeypatch):
    """The autotuner's choice, and each schedule it can choose, read from its cache, in the forms that are
    tuned: the resident step is off, so the step calls run what was chosen."""
    monkeypatch.setenv("DG_RESIDENT", "0")
    monkeypatch.setenv("DG_WAVE_MIN", "0")
    m = _mesh(10, shots, precision)
    stats, want = _run(m, precision)
    assert stats["kernel_family"] in family
    cache = tmp_path / "tune.txt"
    stats, got = _run(m, precision, autotune=True, tune_cache=str(cache))
    assert stats["kernel_family"] in family
    (line,) = cache.read_text().splitlines()
    runs = [got]
    for block in (64, 128, 256):
        for persistent in ((0, 1) if 5 in family else (1,)):
            for margin in (10, 14):
                cache.write_text("%s %d %d %d\n" % (line.split()[0], block, persistent, margin))
                stats, got = _run(m, precision, autotune=True, tune_cache=str(cache))
                assert stats["block_threads"] == block and stats["kernel_family"] in family
                assert len(family) == 1 or stats["kernel_family"] == (6 if persistent else 5)
                runs.append(got)
    for got in runs:
        for a, b in zip(want, got):
            assert np.array_equal(a, b)
    assert np.abs(want[5]).max() > 0
