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
