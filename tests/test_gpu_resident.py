"""The resident step (k_step_resident: the wave field of a small mesh stays on the SMs for a whole
step call) against the two-launch step, which `DG_RESIDENT=0` keeps.

Both feed the same arithmetic in the same order, so fields and traces are equal bit for bit: for
meshes of one block and of many, block edges inside and at the end of the mesh, one shot, odd
counts (padded) and several shots, calls of one step and of many, and after a checkpoint.
"""
import numpy as np
import pytest

from conftest import pkg

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
STEPS = 60


def _mesh(cells, shots, precision):
    w = pkg.workloads.small_square(n_cells=cells, steps=STEPS, shots=shots)
    s = pkg.host.build_setup(w, full=precision == "fp64_ref")
    return eng.mesh_from_setup(s, with_ref_ops=precision == "fp64_ref")


def _run(m, shots, precision, chunks, **kw):
    with eng.Engine(m, precision, **kw) as e:
        rng = np.random.default_rng(3)
        for q in range(shots):
            for f in FIELDS:
                e.load(f, rng.standard_normal(e.info[0]["K"] * 6) * (1e-3 if f[0] == "V" else 1e3), 0, q)
        launches = 0
        for c in chunks:
            e.step(c)
            launches += e.stats()["launches"]
        return launches, [e.fetch(f, 0, eng.ALL_SHOTS) for f in FIELDS] + list(e.fetch_traces(0, STEPS))


# 2 cells: 8 elements, one block; 8: 128, one full block; 9: 162, two; 50: 5,000, forty;
# 101: 20,402, more than 128 elements on every SM; 150: 45,000, FP64 and FP32 blocks of 305
@pytest.mark.parametrize("cells,shots", [(2, 1), (8, 1), (9, 1), (50, 1), (101, 1), (150, 1), (9, 2), (17, 3), (40, 14),
                                         (61, 5)])
@pytest.mark.parametrize("precision", ["fp64", "fp64_ref", "fp32", "fp32_kahan"])
def test_resident_equals_two_launches(precision, cells, shots, monkeypatch):
    m = _mesh(cells, shots, precision)
    monkeypatch.setenv("DG_RESIDENT", "0")
    two, want = _run(m, shots, precision, (STEPS,))
    monkeypatch.setenv("DG_RESIDENT", "1")
    one, got = _run(m, shots, precision, (1, 2, STEPS - 3))
    assert two == 2 * STEPS
    lanes = 2 * cells * cells * (shots if precision.startswith("fp64") else (shots + 1) // 2)
    if lanes <= 148 * 256:
        assert one == 3
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
    assert all(np.isfinite(a).all() for a in got) and np.abs(got[5]).max() > 0


def test_resident_without_reordering_and_without_receivers(monkeypatch):
    """The caller's own numbering (blocks with many outside faces), and a mesh without receivers."""
    m = _mesh(30, 1, "fp64")
    monkeypatch.setenv("DG_RESIDENT", "0")
    _, want = _run(m, 1, "fp64", (STEPS,), reorder=False)
    monkeypatch.setenv("DG_RESIDENT", "1")
    _, got = _run(m, 1, "fp64", (STEPS,), reorder=False)
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
    m["receiver"] = np.zeros((0, 2), dtype=np.int64)
    _, none = _run(m, 1, "fp64", (STEPS,))
    for a, b in zip(want[:5], none[:5]):
        assert np.array_equal(a, b)


def test_a_wait_that_runs_out_reports_timeout_and_the_context_recovers(monkeypatch):
    """Messages of one face that nobody sends to their reader: the reader's wait reaches its
    limit, the launch ends and the call reports DG_ERR_TIMEOUT, again on the next call; reset
    works on."""
    m = _mesh(20, 1, "fp64")
    monkeypatch.setenv("DG_RESIDENT_STALL", "1")
    with eng.Engine(m, "fp64") as e:
        for _ in range(2):
            with pytest.raises(eng.DGError) as ei:
                e.step(3)
            assert ei.value.code == -10
        e.reset()
        assert e.steps_done == 0 and not np.any(e.fetch("Vz"))


@pytest.mark.parametrize("n", [1, 3, 64, 65])
def test_wavelet_samples_sent_step_by_step(n):
    """Small wavelet updates go through a staging buffer without a wait: samples sent ahead of their
    steps, many times around the buffer and reusing the caller's array at once, give the steps of
    the whole table."""
    m = _mesh(8, 1, "fp64")
    total = 650
    w = np.random.default_rng(8).standard_normal(total) * 1e-2
    m["wavelet"] = np.zeros(total)
    with eng.Engine(m, "fp64") as a, eng.Engine(m, "fp64") as b:
        a.set_wavelet(0, w)
        a.step(total)
        buf = np.empty(n)
        for t in range(0, total, n):
            k = min(n, total - t)
            buf[:k] = w[t:t + k]
            b.set_wavelet(t, buf[:k])
            buf[:] = np.nan
            b.step_async(k)
        b.synchronize()
        for f in FIELDS:
            assert np.array_equal(a.fetch(f), b.fetch(f))
        assert np.abs(a.fetch("Vz")).max() > 0
