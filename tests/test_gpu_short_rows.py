"""Rows of at most 64 words share a warp (4, 8, 16 or 32 lanes a row).  The form with one row a warp (narrow_build = 0)
gives the same rows, phenotypes and fitness to the bit: rows that fill their lanes and rows that do not, parents
narrower than their children, dense rows (more gathered alleles than a queue holds), breakpoint lists longer than
the device draws, more new alleles a row than a warp has lanes."""
import numpy as np
import pytest

from clotho_gb300.tape import GenTape, neutral_tape

pytestmark = pytest.mark.gpu


def _tape(rng, N, mu, rho, T):
    t = neutral_tape(rng, N, mu, rho, T=T, p_neutral=0.2)
    # one row with 150 breakpoints, one with 33 new alleles
    E = np.diff(t.ev_off).astype(np.int64)
    E[2] = 150
    off = np.concatenate([[0], np.cumsum(E)]).astype(np.uint32)
    pos = rng.random(int(off[-1]))
    pos[::5] = np.round(pos[::5], 2)   # ties
    M = t.M + 33
    eff = np.concatenate([t.mut_eff, rng.standard_normal(33 * T).astype(np.float32)])
    return GenTape(N, M, t.pairs, t.swap, off, pos, np.concatenate([t.mut_seq, np.full(33, 5, np.uint32)]),
                   np.concatenate([t.mut_pos, rng.random(33)]), eff)


@pytest.mark.parametrize("A0,T,dense,q1", [(60, 1, True, True), (500, 4, False, False), (512, 2, True, False),
                                           (1_000, 3, False, True), (1_024, 1, True, False), (1_500, 4, False, False),
                                           (2_040, 2, True, False)])
def test_short_rows_share_a_warp_and_change_nothing(A0, T, dense, q1):
    import clotho_gb300 as cg
    N, cap, G = 301, 4_000, 4
    rng = np.random.default_rng(A0)
    W = (A0 + 511) // 512 * 8
    rows = rng.integers(0, 2 ** 64, size=(2 * N, W), dtype=np.uint64)
    if not dense:
        for _ in range(3):
            rows &= rng.integers(0, 2 ** 64, size=(2 * N, W), dtype=np.uint64)
    pos = rng.random(A0)
    pos[1::9] = np.round(pos[1::9], 2)
    eff = rng.standard_normal(A0 * T).astype(np.float32)
    tapes = [_tape(rng, N, 0.1, 2.5, T) for _ in range(G)]
    got = []
    for narrow in (1, 0):
        with cg.Population(N, cap, T, mu=0.1, rho=2.5, p_neutral=0.2, fitness="gaussian_vs", fit_param=1e4, q1=q1,
                           max_events=8_000, max_mutations=400, seed=9) as pop:
            pop.set_tuning(narrow_build=narrow)
            pop.load_population(N, rows, pos, eff)
            out = []
            for t in tapes:
                pop.simulate(t)
                out += [pop.rows(), pop.genome_traits(), pop.fitness(), pop.free_list()]
            pop.run_philox(N, 3)
            pop.run_philox(77, 2)
            out += [pop.rows(), pop.genome_traits(), pop.fitness(), pop.free_list(), *pop.margins()]
            pop.check()
            got.append(out)
    for a, b in zip(*got):
        assert a.shape == b.shape and a.tobytes() == b.tobytes()


def test_short_rows_of_a_batch():
    import clotho_gb300 as cg
    sizes = np.array([[40, 333, 5], [2, 200, 90], [50, 1, 90], [64, 7, 1], [64, 300, 128]], np.uint32)
    got = []
    for narrow in (1, 0):
        b = cg.Batch([cg.make_desc(64, 500, 2, mu=0.3, rho=3.0, p_neutral=0.1, fitness="gaussian", seed=4),
                      cg.make_desc(333, 1_900, 4, mu=0.2, rho=1.0, p_neutral=0.1, fitness="constant", seed=5),
                      cg.make_desc(128, 900, 1, mu=0.5, rho=6.0, p_neutral=0.1, fitness="quadratic", fit_param=9.0,
                                   seed=6)])
        b.set_tuning(rows_per_item=96, narrow_build=narrow)
        b.init()
        b.run_schedule(sizes)
        got.append([(b.rows(i), *b.margins(i), b.info(i)) for i in range(3)])
        b.close()
    for x, y in zip(*got):
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1]) and np.array_equal(x[2], y[2]) and x[3] == y[3]


# 32 lanes a row: rows of 40 and 48 words and rows that grow from 56 words to 64
@pytest.mark.parametrize("A0,T,dense,q1", [(2_049, 4, False, True), (3_000, 1, True, False), (3_300, 2, False, False)])
def test_rows_of_33_to_64_words_change_nothing(A0, T, dense, q1):
    test_short_rows_share_a_warp_and_change_nothing(A0, T, dense, q1)
