"""States that do not fit L2 are swept in alternating directions: the stress half backwards, the
wavefront step's odd steps backwards (`DG_BACK=1` asks for it at any size).  The order of blocks
changes no value: fields and traces equal the one-direction sweeps bit for bit, in every
precision, on one mesh (last blocks and units partly filled), in a batch, and in the parts of a
split mesh.
"""
import numpy as np
import pytest

from conftest import pkg

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
STEPS = 41


def _mesh(cells, shots, ref):
    w = pkg.workloads.small_square(n_cells=cells, steps=STEPS, shots=shots)
    return eng.mesh_from_setup(pkg.host.build_setup(w, full=ref), with_ref_ops=ref)


def _fill(load, S, K):
    rng = np.random.default_rng(2)
    for q in range(min(S, 4)):
        for f in FIELDS:
            load(f, rng.standard_normal(K * 6) * (1e-3 if f[0] == "V" else 1e3), q)


@pytest.mark.parametrize("precision,cells,shots,kw", [
    ("fp64", 13, 1, {}), ("fp64_ref", 13, 2, {}), ("fp32", 13, 1, {}), ("fp32_kahan", 13, 3, {}), ("fp32", 11, 24, {}),
    ("fp32", 9, 16, {"wavefront": 1}), ("fp32_kahan", 10, 64, {"wavefront": 1}), ("fp32", 15, 1, {"wavefront": 1}),
    ("fp32", 9, 16, {"wavefront": 1, "block_threads": 256})])
def test_one_mesh(precision, cells, shots, kw, monkeypatch):
    monkeypatch.setenv("DG_RESIDENT", "0")
    monkeypatch.setenv("DG_WAVE_MIN", "0")
    m = _mesh(cells, shots, precision == "fp64_ref")
    out = []
    for back in ("0", "1"):
        monkeypatch.setenv("DG_BACK", back)
        with eng.Engine(m, precision, **kw) as e:
            _fill(lambda f, v, q: e.load(f, v, 0, q), shots, e.info[0]["K"])
            e.step(STEPS - 2)
            e.step_timed(2)
            out.append([e.fetch(f, 0, eng.ALL_SHOTS) for f in FIELDS] + list(e.fetch_traces(0, STEPS)))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert np.abs(out[0][5]).max() > 0


@pytest.mark.parametrize("precision,persistent", [("fp32", "0"), ("fp32", "1"), ("fp64", "0")])
def test_batch(precision, persistent, monkeypatch):
    monkeypatch.setenv("DG_MX_PERSISTENT", persistent)
    meshes = [_mesh(c, s, False) for c, s in ((9, 1), (13, 3), (7, 16))]
    out = []
    for back in ("0", "1"):
        monkeypatch.setenv("DG_BACK", back)
        with eng.Engine(meshes, precision) as e:
            for k in range(3):
                _fill(lambda f, v, q: e.load(f, v, k, q), e.info[k]["S"], e.info[k]["K"])
            e.step(STEPS)
            out.append([e.fetch(f, k, 0) for k in range(3) for f in FIELDS] + list(e.fetch_traces(0, STEPS, mesh=eng.ALL_MESHES)))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision,shots", [("fp64", 1), ("fp32", 1), ("fp32", 3)])
def test_split_parts(precision, shots, monkeypatch):
    m = _mesh(16, shots, False)
    with eng.Engine(m, precision, wavefront=-1) as whole:
        whole.step(STEPS)
        want = [whole.fetch(f, 0, shots - 1).reshape(-1, 6) for f in FIELDS]
    monkeypatch.setenv("DG_BACK", "1")
    for overlap in (False, True):
        with pkg.decompose.SplitRun(m, 3, precision, overlap=overlap, block_threads=64) as run:
            run.step(STEPS)
            for f, v in zip(FIELDS, want):
                assert np.array_equal(run.fetch(f, shots - 1), v)
