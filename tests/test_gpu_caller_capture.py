"""Calls made while the caller captures the context's stream in a CUDA graph of its own."""
import ctypes as C

import numpy as np
import pytest

from clotho_gb300.tape import neutral_tape

pytestmark = pytest.mark.gpu

GLOBAL, THREAD, RELAXED = 0, 1, 2


class Capture:
    """A stream of the caller's, and the graph that is captured on it."""

    def __init__(self):
        for name in ("libcudart.so.13", "libcudart.so"):
            try:
                self.rt = C.CDLL(name)
                break
            except OSError:
                continue
        else:
            pytest.skip("no CUDA runtime library to capture with")
        self.rt.cudaStreamBeginCapture.argtypes = [C.c_void_p, C.c_int]
        self.rt.cudaStreamEndCapture.argtypes = [C.c_void_p, C.POINTER(C.c_void_p)]
        self.rt.cudaGraphInstantiate.argtypes = [C.POINTER(C.c_void_p), C.c_void_p, C.c_ulonglong]
        self.rt.cudaGraphLaunch.argtypes = [C.c_void_p, C.c_void_p]
        self.rt.cudaStreamSynchronize.argtypes = [C.c_void_p]
        s = C.c_void_p()
        assert self.rt.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
        self.stream = s.value

    def begin(self, mode):
        assert self.rt.cudaStreamBeginCapture(self.stream, mode) == 0

    def end(self):
        g, x = C.c_void_p(), C.c_void_p()
        assert self.rt.cudaStreamEndCapture(self.stream, C.byref(g)) == 0
        assert self.rt.cudaGraphInstantiate(C.byref(x), g, 0) == 0
        return x.value

    def replay(self, x, times):
        for _ in range(times):
            assert self.rt.cudaGraphLaunch(x, self.stream) == 0
        assert self.rt.cudaStreamSynchronize(self.stream) == 0


@pytest.mark.parametrize("mode", [GLOBAL, THREAD, RELAXED])
@pytest.mark.parametrize("N", [300, 40_000])   # a tape below and one above the pinned block
def test_tapes_are_refused_and_leave_the_context_whole(N, mode):
    import clotho_gb300 as cg
    rng = np.random.default_rng(N)
    tapes = [neutral_tape(rng, N, 5e-4, 2.0) for _ in range(5)]
    got = []
    for capture in (True, False):
        with cg.Population(N, 4_000, 1, max_events=200_000, max_mutations=1_000) as pop:
            pop.init(N)
            if capture:
                c = Capture()
                pop.set_stream(c.stream)
            for t in tapes:
                if capture:
                    c.begin(mode)
                    try:
                        with pytest.raises(cg.ClothoError, match="captured"):
                            pop.simulate(t)
                    finally:
                        c.end()
                pop.simulate(t)
            pop.check()
            got.append((pop.info(), pop.rows().tobytes(), pop.pairs().tobytes()))
    assert got[0] == got[1]
