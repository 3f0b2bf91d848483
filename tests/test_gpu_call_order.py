"""Calls return with work still queued; whatever order they come in, the results are those of the same calls with a
clotho_sync after each.  Tapes up to 1 MB are uploaded on the compute stream, larger ones on the copy stream, into
buffers that device-drawn steps use as well."""
import numpy as np
import pytest

from clotho_gb300.tape import neutral_tape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [["draw", "large"], ["large", "draw", "large", "draw", "large"],
                                   ["small", "draw", "large", "large", "draw", "large", "large"],
                                   ["large", "small", "large", "small", "small", "large", "large", "large", "small"],
                                   ["draw", "small", "small", "draw", "small", "large", "schedule", "large", "large"]])
def test_queued_calls_do_not_disturb_each_other(order):
    import clotho_gb300 as cg
    N, n = 30_000, 400
    rng = np.random.default_rng(len(order))
    tapes, at = [], N
    for kind in order:
        size = {"large": N, "small": n}.get(kind)
        if size:
            tapes.append(neutral_tape(rng, size, 2e-4, 2.0, T=2, p_neutral=0.0, parents=at))
        at = size or N
    assert {t.nbytes > (1 << 20) for t in tapes} == {k == "large" for k in order if k in ("large", "small")}
    got = []
    for sync in (False, True):
        with cg.Population(N, 4_000, 2, mu=2e-4, rho=2.0, p_neutral=0.0, max_events=130_000, seed=7) as pop:
            pop.init(N)
            left = list(tapes)
            for kind in order:
                if kind == "draw":
                    pop.run_philox(N, 40)
                elif kind == "schedule":
                    pop.run_philox_schedule(np.full(40, N))
                else:
                    pop.simulate(left.pop(0))
                if sync:
                    pop.sync()
            pop.check()
            got.append([pop.rows(), pop.genome_traits(), pop.pairs()])
    for a, b in zip(*got):
        assert a.shape == b.shape and a.tobytes() == b.tobytes()


@pytest.mark.parametrize("before", [0, 1, 3])
def test_calls_on_a_context_without_populations_are_refused(before):
    import ctypes as C

    import clotho_gb300 as cg
    desc = [cg.make_desc(500, 2_000, 2, mu=0.01, rho=0.4, p_neutral=0.3, seed=i + 1) for i in range(3)]
    b, fresh = cg.Batch(desc[:before]), cg.Batch(desc[:2])
    b.init()
    b.run(5)
    while len(b):
        b.remove(0)
    L, h, launches = b.L, b.h, b.launches
    buf = np.zeros(10_000, np.float64)
    p, n0 = buf.ctypes.data_as(C.c_void_p), C.c_uint32(0)
    for rc in (L.clotho_generation_philox(h, 500), L.clotho_run_philox(h, 500, 3), L.clotho_begin_generation(h, 500, 0),
               L.clotho_phenotype(h), L.clotho_fitness(h), L.clotho_get_phenotypes(h, p), L.clotho_get_fitness(h, p),
               L.clotho_get_genome_traits(h, p), L.clotho_get_pairs(h, p), L.clotho_get_free(h, p),
               L.clotho_get_alleles(h, p, None, None), L.clotho_get_fixed(h, p, None, None),
               L.clotho_seed_population(h, 10, 0, None, None, None, 1)):
        assert rc != 0
    assert L.clotho_batch_run_philox(h, C.byref(n0), 3) == 0 and L.clotho_run_philox(h, 500, 0) == 0
    assert b.launches == launches and not buf.any()
    for d in desc[:2]:
        b.add(d, 500)
    fresh.init()
    for x in (b, fresh):
        x.run(4)
    for i in range(2):
        assert b.rows(i).tobytes() == fresh.rows(i).tobytes() and b.info(i) == fresh.info(i)
    b.close()
    fresh.close()


def test_a_refused_call_is_reported_once():
    # the graph calls cannot capture on the legacy default stream
    import clotho_gb300 as cg
    with cg.Population(200, 2_000, 1, mu=0.02, rho=0.4, p_neutral=0.0, fitness="gaussian", seed=5) as pop:
        pop.init(120)
        for after in (pop.phenotypes, pop.margins, lambda: pop.simulate_philox(100)):
            pop.set_stream(1)
            with pytest.raises(cg.ClothoError, match="rc="):
                pop.run_philox(110, 3)
            pop.set_stream(None)
            after()
        pop.check()


@pytest.mark.parametrize("N", [90, 150])
def test_reads_after_a_call_that_failed_halfway(N):
    # the graph calls cannot capture on the legacy default stream; they fail there behind their first generation
    import ctypes as C

    import clotho_gb300 as cg
    with cg.Population(200, 2_000, 1, mu=0.02, rho=0.4, p_neutral=0.0, fitness="gaussian", seed=5) as pop:
        pop.init(120)
        pop.run_philox(120, 3)
        for n, call in ((N, lambda: pop.run_philox_schedule([N] * 3)), (N + 7, lambda: pop.run_philox(N + 7, 3))):
            pop.set_stream(1)
            with pytest.raises(cg.ClothoError, match="rc="):
                call()
            pop.set_stream(None)
            assert pop.info()["N"] == n
            for read in (pop.L.clotho_get_fitness, pop.L.clotho_get_phenotypes):
                buf = np.full(200, -7.0)
                assert read(pop.h, buf.ctypes.data_as(C.c_void_p)) == 0
                assert (buf[:n] != -7.0).all() and (buf[n:] == -7.0).all()
            call()
            assert pop.fitness().size == n
        pop.check()
