"""Populations of at most 8,192 slots rank them in one block's shared memory; wider capacities by global buckets.
The same population in both gives the same rows and phenotypes: few slots and as many as fit, positions that are all
equal, all in one bucket, or spread, zeros of both signs, breakpoints on positions."""
import numpy as np
import pytest

from clotho_gb300.tape import GenTape, neutral_tape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("A,where", [(1, "spread"), (700, "equal"), (1_024, "one bucket"), (1_025, "spread"),
                                     (4_097, "ties"), (7_900, "spread"), (7_680, "one bucket")])
def test_both_rank_paths_agree(A, where):
    import clotho_gb300 as cg
    N, T = 150, 2
    rng = np.random.default_rng(A)
    W = (A + 511) // 512 * 8
    rows = rng.integers(0, 2 ** 64, size=(2 * N, W), dtype=np.uint64) & rng.integers(0, 2 ** 64, size=(2 * N, W),
                                                                                   dtype=np.uint64)
    pos = rng.random(A)
    if where == "equal":
        pos[:] = 0.25
    elif where == "one bucket":
        pos = 0.5 + pos * 1e-9
    elif where == "ties":
        pos = np.round(pos, 2)
        pos[::50] = 0.0
        pos[1::50] = -0.0
    eff = rng.standard_normal(A * T).astype(np.float32)
    tapes = []
    for _ in range(3):
        t = neutral_tape(rng, N, 0.1, 3.0, T=T, p_neutral=0.0)
        ev = t.ev_pos.copy()
        ev[::3] = rng.choice(pos, ev[::3].size) + 0.0
        tapes.append(GenTape(N, t.M, t.pairs, t.swap, t.ev_off, ev, t.mut_seq, t.mut_pos, t.mut_eff))
    got = []
    for cap in (8_192, 9_000):
        with cg.Population(N, cap, T, max_events=4_000, max_mutations=200) as pop:
            pop.load_population(N, rows, pos, eff)
            out = []
            for t in tapes:
                pop.simulate(t)
                out += [pop.rows(), pop.genome_traits(), pop.free_list()]
            pop.check()
            got.append(out)
    for a, b in zip(*got):
        assert a.shape == b.shape and a.tobytes() == b.tobytes()
