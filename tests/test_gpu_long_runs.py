"""Device-drawn runs replay graphs of one generation and, once a run is long, of several: any split of a run into
calls gives the rows and sizes of generation-by-generation calls, with a fixed size and with a schedule of sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(p):
    i = p.info()
    return [p.rows(), p.genome_traits(), p.fitness(), np.array([i["generation"], i["N"], i["A"], i["fixed_total"]])]


@pytest.mark.parametrize("fitness", ["constant", "gaussian"])
@pytest.mark.parametrize("splits", [[131], [1, 63, 1, 66], [9] * 14 + [5]])
def test_any_split_of_a_run(fitness, splits):
    import clotho_gb300 as cg
    N, sizes = 60, np.array([(7 * g * g + 5) % 61 + 1 for g in range(sum(splits))], np.uint32)
    for schedule in (False, True):
        got = []
        for calls in (splits, None):
            with cg.Population(64, 2_000, 2, mu=0.02, rho=0.5, p_neutral=0.2, fitness=fitness, seed=12) as pop:
                pop.init(N)
                at = 0
                for G in calls or [1] * int(sum(splits)):
                    if not calls:
                        pop.simulate_philox(int(sizes[at]) if schedule else N)
                    elif schedule:
                        pop.run_philox_schedule(sizes[at:at + G])
                    else:
                        pop.run_philox(N, G)
                    at += G
                pop.check()
                got.append(_state(pop))
        for a, b in zip(*got):
            assert a.shape == b.shape and a.tobytes() == b.tobytes()


def test_long_schedule_of_a_batch():
    import clotho_gb300 as cg
    descs = [cg.make_desc(64, 2_000, 1, mu=0.02, rho=0.5, fitness="constant", seed=3),
             cg.make_desc(300, 3_000, 2, mu=0.01, rho=1.5, p_neutral=0.1, fitness="gaussian", seed=4)]
    sizes = np.array([[(g * 11) % 64 + 1, (g * 37) % 300 + 1] for g in range(90)], np.uint32)
    got = []
    for split in ([90], [1] * 90, [40, 50]):
        b = cg.Batch(descs)
        b.init()
        at = 0
        for G in split:
            b.run_schedule(sizes[at:at + G])
            at += G
        got.append([(b.rows(i), b.info(i)) for i in range(2)])
        b.close()
    for other in got[1:]:
        for x, y in zip(got[0], other):
            assert np.array_equal(x[0], y[0]) and x[1] == y[1]
