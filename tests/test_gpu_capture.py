"""Steps enqueued while the caller captures the context's stream: the capture holds plain launches
that take their step from the device's counters, so replaying it twice gives the fields of twice
the steps, for a mesh whose own calls run resident and for a batch that steps mesh by mesh.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import pkg

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")


def _load(e):
    rng = np.random.default_rng(1)
    for k, info in enumerate(e.info):
        for f in FIELDS:
            e.load(f, rng.standard_normal(info["K"] * 6) * (1e-3 if f[0] == "V" else 1e3), k, 0)


def _fields(e):
    return [e.fetch(f, k, eng.ALL_SHOTS) for k in range(len(e.info)) for f in FIELDS]


@pytest.mark.parametrize("shapes,steps", [([(10, 1)], 3), ([(10, 1)], 30), ([(9, 1), (12, 4), (5, 2)], 3),
                                          ([(9, 1), (12, 4), (5, 2)], 30)])
def test_replayed_capture(shapes, steps, monkeypatch):
    monkeypatch.setenv("DG_BATCH_BY_MESH", "1")
    meshes = [eng.mesh_from_setup(pkg.host.build_setup(pkg.workloads.small_square(n_cells=n, steps=80, shots=s), full=False),
                                  with_ref_ops=False) for n, s in shapes]
    with eng.Engine(meshes, "fp32") as e:
        _load(e)
        e.step(2 * steps)
        want = _fields(e)
    cu = C.CDLL("libcuda.so.1")
    with eng.Engine(meshes, "fp32") as e:
        _load(e)
        st, graph, run = C.c_void_p(e.stream().cuda_stream), C.c_void_p(), C.c_void_p()
        assert cu.cuStreamBeginCapture_v2(st, 1) == 0  # thread local
        e.step_async(steps)
        assert cu.cuStreamEndCapture(st, C.byref(graph)) == 0
        assert cu.cuGraphInstantiateWithFlags(C.byref(run), graph, C.c_ulonglong(0)) == 0
        for _ in range(2):
            assert cu.cuGraphLaunch(run, st) == 0
        assert cu.cuStreamSynchronize(st) == 0
        got = _fields(e)
        cu.cuGraphExecDestroy(run)
        cu.cuGraphDestroy(graph)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
