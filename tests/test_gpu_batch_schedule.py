"""How a batch is stepped: which batches go mesh by mesh, and that the order of the meshes in a call,
short or long, changes no value.
"""
import numpy as np
import pytest

from conftest import pkg

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
STEPS = 40


def _mesh(cells, shots):
    return eng.mesh_from_setup(pkg.host.build_setup(pkg.workloads.small_square(n_cells=cells, steps=STEPS, shots=shots), full=False),
                               with_ref_ops=False)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_calls_of_any_length(precision, monkeypatch):
    """Two meshes of more than 50,000 lanes and eighteen small ones (more than there are chains for
    those), in calls of 1, 5, 15, 16 and 3 steps, against launches over all meshes."""
    large = (115, 4) if precision == "fp32" else (115, 2)
    meshes = [_mesh(*s) for s in [(4 + k, 1 + k % 3) for k in range(9)] + [large, (115, 5)] + [(5 + k, 2) for k in range(9)]]
    out = []
    for by_mesh in ("0", "1"):
        monkeypatch.setenv("DG_BATCH_BY_MESH", by_mesh)
        with eng.Engine(meshes, precision) as e:
            assert (e.stats()["kernel_family"] == 9) == (by_mesh == "1")
            rng = np.random.default_rng(9)
            for k, info in enumerate(e.info):
                for f in FIELDS:
                    e.load(f, rng.standard_normal(info["K"] * 6) * (1e-3 if f[0] == "V" else 1e3), k, info["S"] - 1)
            for n in (1, 5, 15, 16, 3):
                e.step(n)
            out.append([e.fetch(f, k, eng.ALL_SHOTS) for k in range(len(meshes)) for f in FIELDS] +
                       list(e.fetch_traces(0, STEPS, eng.ALL_MESHES)))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert np.abs(out[0][0]).max() > 0


# (cells per side, shots) of the meshes: like sizes on both sides of 55,000 lanes a mesh, a large mesh
# among small ones (the mean above it, the others far below), and few small ones among larger ones
@pytest.mark.parametrize("shapes,precision,by_mesh", [
    ([(52, 22)] * 2, "fp32", True), ([(52, 20)] * 2, "fp32", False), ([(48, 12)] * 2, "fp64", True), ([(48, 11)] * 2, "fp64", False),
    ([(48, 128)] + [(5, 2)] * 4, "fp32", False), ([(50, 16)] * 4 + [(5, 2)] * 4, "fp64", False),
    ([(50, 36)] * 7 + [(5, 2)], "fp32_kahan", True), ([(48, 128)] * 2 + [(5, 2)], "fp32", True)])
def test_which_batches_go_mesh_by_mesh(shapes, precision, by_mesh):
    kinds = {s: _mesh(*s) for s in set(shapes)}
    with eng.Engine([kinds[s] for s in shapes], precision) as e:
        assert (e.stats()["kernel_family"] == 9) == by_mesh
        e.step(2)
        assert e.steps_done == 2
