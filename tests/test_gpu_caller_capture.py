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


def _descs(cg):
    return [cg.make_desc(n, 2_000, 1, mu=0.01, rho=0.3, fitness=f, p_neutral=0.2, seed=n)
            for n, f in ((400, "constant"), (37, "gaussian"), (900, "constant"), (1_500, "gaussian"))]


def _states(b):
    return [(b.info(i), b.rows(i).tobytes()) for i in range(len(b))]


@pytest.mark.parametrize("mode,before", [(RELAXED, 0), (RELAXED, 1), (GLOBAL, 1), (THREAD, 1)])
@pytest.mark.parametrize("change", ["add", "tune", "remove"])
def test_first_batch_step_after_a_change_is_captured(mode, before, change):
    # (in the stricter modes a context's first step of all is refused: it takes pinned memory)
    import clotho_gb300 as cg
    got = []
    for capture in (True, False):
        d = _descs(cg)
        b = cg.Batch(d[:3])
        b.init()
        c = Capture()
        b.set_stream(c.stream)
        for _ in range(before):
            b.step()
        for tune in (3, 24):      # twice: the second change is one under a graph that exists
            if change == "add" and len(b) < 4:
                b.add(d[3], 1_500)
            elif change == "remove" and len(b) > 2:
                b.remove(0)
            elif tune == 3 or not capture:
                b.set_tuning(row_blocks_per_sm=tune)
            if capture:
                c.begin(mode)
                try:
                    if change == "tune" and tune != 3:
                        b.set_tuning(row_blocks_per_sm=tune)
                    b.step()
                finally:
                    x = c.end()
                c.replay(x, 3)
                if tune == 3:
                    first = x
            else:
                for _ in range(3):
                    b.step()
        if change == "tune":      # the first graph's launch shapes still hold
            if capture:
                c.replay(first, 2)
            else:
                b.run(2)
        b.run(2)
        got.append(_states(b))
        b.close()
    assert got[0] == got[1]


def test_reads_between_replays_of_the_callers_graph():
    import clotho_gb300 as cg
    with cg.Population(200, 2_000, 1, mu=0.02, rho=0.4, p_neutral=0.0, fitness="gaussian", seed=5) as pop:
        pop.init(120)
        pop.run_philox(120, 3)
        c = Capture()
        pop.set_stream(c.stream)

        def reads(N):
            assert pop.info()["N"] == N
            for read in (pop.L.clotho_get_fitness, pop.L.clotho_get_phenotypes):
                buf = np.full(200, -7.0)
                assert read(pop.h, buf.ctypes.data_as(C.c_void_p)) == 0
                assert (buf[:N] != -7.0).all() and (buf[N:] == -7.0).all()

        c.begin(RELAXED)
        try:
            pop.simulate_philox(80)
        finally:
            x = c.end()
        reads(120)
        c.replay(x, 1)
        reads(80)
        pop.run_philox(150, 2)
        reads(150)
        c.replay(x, 2)
        reads(80)
        pop.check()
