"""A capture of a context's stream, by the caller: what was enqueued inside it, to be replayed."""
import ctypes as C

_cu = None


def _call(name, *args):
    global _cu
    _cu = _cu or C.CDLL("libcuda.so.1")
    rc = getattr(_cu, name)(*args)
    assert rc == 0, (name, rc)


class Captured:
    """`with Captured(engine) as g: engine.step_async(n)`, then `g.launch()` as often as wanted."""

    def __init__(self, engine):
        self.stream = C.c_void_p(engine.stream().cuda_stream)
        self.graph, self.run = C.c_void_p(), C.c_void_p()

    def __enter__(self):
        _call("cuStreamBeginCapture_v2", self.stream, 1)  # thread local
        return self

    def __exit__(self, kind, value, trace):
        if kind is not None:  # the capture may be invalid by now: only end it
            _cu.cuStreamEndCapture(self.stream, C.byref(self.graph))
            return False
        _call("cuStreamEndCapture", self.stream, C.byref(self.graph))
        _call("cuGraphInstantiateWithFlags", C.byref(self.run), self.graph, C.c_ulonglong(0))
        return False

    def launch(self, times=1):
        """Enqueues the captured work on the context's stream, without a wait."""
        for _ in range(times):
            _call("cuGraphLaunch", self.run, self.stream)

    def close(self):
        if self.run:
            _call("cuGraphExecDestroy", self.run)
        if self.graph:
            _call("cuGraphDestroy", self.graph)
