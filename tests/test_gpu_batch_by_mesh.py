"""A batch stepped mesh by mesh (a context per mesh, several meshes side by side) against the batch
whose launches take all meshes: the same bits out of every call, over meshes of different sizes,
shot counts and step counts, one of them past its last step.  `DG_BATCH_BY_MESH` picks the form.
"""
import numpy as np
import pytest

from conftest import pkg

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
# cells per side, shots, steps
MESHES = ((9, 1, 60), (14, 5, 60), (6, 16, 30), (11, 2, 60), (3, 1, 47))


def _batch(ref):
    out = []
    for cells, shots, steps in MESHES:
        w = pkg.workloads.small_square(n_cells=cells, steps=steps, shots=shots)
        out.append(eng.mesh_from_setup(pkg.host.build_setup(w, full=ref), with_ref_ops=ref))
    return out


def _run(meshes, precision, **kw):
    """Every call of a batch, its results in order."""
    got, energy = [], []
    with eng.Engine(meshes, precision, **kw) as e:
        fam = e.stats()["kernel_family"]
        for repeat in range(2):
            rng = np.random.default_rng(3)
            for k, (info, mesh) in enumerate(zip(e.info, MESHES)):
                for f in FIELDS:
                    e.load(f, rng.standard_normal(info["K"] * 6) * (1e-3 if f[0] == "V" else 1e3), k, mesh[1] - 1)
            e.step(3)
            e.set_wavelet(3, rng.standard_normal(2), 1)
            e.step_async(4)
            e.set_wavelet(7, rng.standard_normal((len(MESHES), 20)), eng.ALL_MESHES)
            e.half_step(0)
            e.half_step(1)
            e.step_timed(2)
            e.step_snapshots(20, 10, lambda t, vx, vz: got.extend([np.array(t), vx.copy(), vz.copy()]), 1, 4)
            energy.append([float(e.fetch("energy", k, 0)) for k in range(len(MESHES))])
            for part in e.fetch_traces(0, 30, mesh=eng.ALL_MESHES):
                got += list(part)
            e.step(25)  # past the ends of the third and the last mesh
            for k in range(len(MESHES)):
                got += [e.fetch(f, k, eng.ALL_SHOTS) for f in FIELDS] + list(e.fetch_traces(0, min(55, MESHES[k][2]), mesh=k))
            assert e.steps_done == 55
            e.reset()
    return fam, got, np.array(energy)


@pytest.mark.parametrize("precision", ["fp32", "fp32_kahan", "fp64", "fp64_ref"])
def test_same_bits_as_launches_over_all_meshes(precision, monkeypatch):
    meshes = _batch(precision == "fp64_ref")
    monkeypatch.setenv("DG_BATCH_BY_MESH", "0")
    fam, want, en0 = _run(meshes, precision)
    assert fam != 9
    monkeypatch.setenv("DG_BATCH_BY_MESH", "1")
    fam, got, en1 = _run(meshes, precision)
    assert fam == 9 and len(got) == len(want)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    # the energy is a sum over a state whose layout may differ: the same terms in another order
    assert np.abs(en1 - en0).max() <= 1e-12 * en0.max()
    assert all(np.isfinite(a).all() for a in want) and any(np.abs(a).max() > 0 for a in want)


def test_requested_forms_keep_the_batch(monkeypatch):
    monkeypatch.setenv("DG_BATCH_BY_MESH", "1")
    meshes = _batch(False)
    for kw in ({"variant": 1}, {"block_threads": 128}, {"watchdog_every": 5}):
        with eng.Engine(meshes, "fp32", **kw) as e:
            assert e.stats()["kernel_family"] != 9
