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


@pytest.mark.parametrize("kinds", [
    # each wants every SM for its resident step
    [("fp64", 1, 150), ("fp64", 1, 150)], [("fp32", 1, 190), ("fp64_ref", 1, 122), ("fp32_kahan", 2, 120)],
    # beside a wavefront on resident blocks, a batch in one cooperative launch, and two-launch steps
    [("fp64", 1, 100), ("fp32", 64, 90), ("fp32", 5, 150)], [("fp32", 3, 40), ("batch", 0, 0), ("fp64", 1, 16)]])
def test_contexts_step_side_by_side_in_threads(kinds, monkeypatch):
    """Contexts stepped from a thread each, at the same time, give the values they give alone."""
    import threading

    monkeypatch.setenv("DG_MX_PERSISTENT", "1")  # batches only

    def make(kind):
        if kind[0] == "batch":
            return eng.Engine([_long(60, 4, "fp32"), _long(30, 1, "fp32")], "fp32")
        return eng.Engine(_long(kind[2], kind[1], kind[0]), kind[0])

    def steps(e):
        for _ in range(40):
            e.step(7)
            e.step_async(3)
        e.synchronize()
        for f in FIELDS:
            out.setdefault(id(e), []).append(e.fetch(f, 0, e.info[0]["S"] - 1))

    def work(e):
        try:
            steps(e)
        except Exception as err:  # noqa: BLE001
            errors.append(err)

    out, errors = {}, []
    alone, together = [make(k) for k in kinds], [make(k) for k in kinds]
    for e in alone + together:
        _load(e)
    for e in alone:
        work(e)
    threads = [threading.Thread(target=work, args=(e,)) for e in together]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(alone, together):
        for x, y in zip(out[id(a)], out[id(b)]):
            assert np.array_equal(x, y)
    for e in alone + together:
        e.close()


def _long(cells, shots, precision):
    ref = precision == "fp64_ref"
    w = pkg.workloads.small_square(n_cells=cells, steps=400, shots=shots)
    return eng.mesh_from_setup(pkg.host.build_setup(w, full=ref), with_ref_ops=ref)
