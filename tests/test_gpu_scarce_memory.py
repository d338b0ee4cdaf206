"""Contexts made where device memory is nearly full: a form that needs more of it than another gives
way, so what fits in the leaner form is still made and stepped.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import pkg

eng = pkg.engine
pytestmark = pytest.mark.gpu
FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")
MB = 1 << 20


class Filled:
    """Device memory with about `leave` bytes of it left, given back at the end."""

    def __init__(self, leave):
        import torch

        torch.cuda.synchronize()
        self.cu, self.held = C.CDLL("libcuda.so.1"), []
        for size in (1 << 30, 64 * MB, 2 * MB):
            while torch.cuda.mem_get_info()[0] - leave >= size and self._take(size):
                pass

    def _take(self, size):
        p = C.c_uint64()
        if self.cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(size)) != 0:
            return False
        self.held.append(p)
        return True

    def __enter__(self):
        return self

    def __exit__(self, *a):
        for p in self.held:
            self.cu.cuMemFree_v2(p)


def _mesh(cells, shots, steps):
    return eng.mesh_from_setup(pkg.host.build_setup(pkg.workloads.small_square(n_cells=cells, steps=steps, shots=shots), full=False),
                               with_ref_ops=False)


def test_a_failed_context_leaves_nothing_for_the_next(monkeypatch):
    """Contexts that do not fit are refused with DG_ERR_NOMEM, and the contexts made after them are made
    and stepped as if those had not been tried, a batch mesh by mesh as asked for."""
    monkeypatch.setenv("DG_BATCH_BY_MESH", "1")
    meshes = [_mesh(n, s, 8) for n, s in ((9, 1), (12, 3))]
    large = _mesh(250, 8, 8)
    for m, family in ((meshes[:1], 3), (meshes, 9)):
        with Filled(24 * MB):
            with pytest.raises(eng.DGError) as ei:
                eng.Engine([large] + m, "fp32")
            assert ei.value.code == -3
        with eng.Engine(m, "fp32") as e:
            assert e.stats()["kernel_family"] == family
            e.step(8)
            assert all(np.isfinite(e.fetch(f)).all() for f in FIELDS)


@pytest.mark.parametrize("env", [{}, {"DG_RESIDENT": "0"}, {"DG_RESIDENT": "0", "DG_WAVE_MIN": "0"}])
def test_padded_shots_count_the_trace_table(env, monkeypatch):
    """17 shots whose traces fill what is left but for half a shot's: there is no room for a padding
    shot, so the counts' own kernels run unpadded."""
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    steps, receivers = 4000, 40000
    m = _mesh(6, 17, steps)
    m["receiver"] = np.tile(m["receiver"], (receivers // len(m["receiver"]) + 1, 1))[:receivers]
    shot = steps * 2 * receivers * 4  # bytes of one shot's traces
    with eng.Engine(_mesh(6, 17, 8), "fp32") as e:
        e.step(8)
    with Filled(17 * shot + steps * receivers * 8 + shot // 2):
        with eng.Engine(m, "fp32") as e:
            e.step(8)
            assert e.steps_done == 8 and np.isfinite(e.fetch("Vz", 0, 16)).all()


def test_no_room_for_the_resident_steps_messages(monkeypatch):
    """The least memory in which a mesh steps in two launches, and a little more of it: the same mesh
    is made and steps there too where the engine would keep it on the SMs."""
    m = _mesh(150, 1, 12)

    def run():
        with eng.Engine(m, "fp64", reorder=False, graph_steps=-1) as e:
            e.step(12)
            return e.stats()["launches"], [e.fetch(f) for f in FIELDS]

    launches, want = run()  # loads the kernels, too
    assert launches == 1
    monkeypatch.setenv("DG_RESIDENT", "0")
    assert run()[0] == 24

    def fits(leave):
        with Filled(leave):
            try:
                run()
                return True
            except eng.DGError as err:
                assert err.code == -3
                return False

    low, high = 0, 256  # in 2 MB
    assert fits(high * 2 * MB)
    while high - low > 1:
        mid = (low + high) // 2
        low, high = (low, mid) if fits(mid * 2 * MB) else (mid, high)
    monkeypatch.setenv("DG_RESIDENT", "1")
    for more in range(0, 9):
        with Filled((high + more) * 2 * MB):
            launches, got = run()
        for a, b in zip(want, got):
            assert np.array_equal(a, b)
