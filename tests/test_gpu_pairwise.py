"""Pairwise differences against numpy at the edges of the 128 x 256 tiles, of the 16-column steps of a narrower
last tile and of the slot ranges that CTAs share, with full rows (the largest counts) and empty ones among random
ones.  Whole numbers: every distance is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,A", [(2, 1), (3, 512), (16, 513), (17, 4_097), (127, 2_000), (128, 1_024), (129, 5_000),
                                 (256, 600), (257, 9_000), (300, 70_000), (385, 20_480), (513, 3_000), (64, 600_001)])
def test_distances_match_numpy(n, A):
    import clotho_gb300 as cg
    rng = np.random.default_rng(n * 1_000_003 + A)
    N, W = max(n // 2 + 1, 4), (A + 511) // 512 * 8
    rows = rng.integers(0, 2 ** 64, size=(2 * N, W), dtype=np.uint64)
    rows[::5] &= rng.integers(0, 2 ** 64, size=rows[::5].shape, dtype=np.uint64)
    rows[1] = rows[-1] = np.uint64(0xffffffffffffffff)
    rows[2] = 0
    sample = rng.permutation(2 * N)[:n].astype(np.uint32)
    sample[-1] = 1
    with cg.Population(N, A, 1) as pop:
        pop.load_population(N, rows, rng.random(A), np.zeros(A, np.float32))
        got = pop.pairwise_difference(sample, distances=True)
        plain = pop.pairwise_difference(sample)
    bits = np.unpackbits(rows[sample].view(np.uint8), axis=1, bitorder="little")[:, :A].astype(np.float32)
    ones = bits.sum(1, dtype=np.float64)
    common = sum((bits[:, k:k + 65_536] @ bits[:, k:k + 65_536].T).astype(np.float64) for k in range(0, A, 65_536))
    d = (ones[:, None] + ones[None, :] - 2 * common)[np.triu_indices(n, 1)]
    assert np.array_equal(got["distances"], d.astype(np.uint32))
    for r in (got, plain):
        assert (r["min"], r["max"], r["count"], r["total"]) == (d.min(), d.max(), d.size, d.sum())
        assert r["mean"] == pytest.approx(d.mean(), rel=1e-12)
        assert r["variance"] == pytest.approx(max(0.0, (d * d).mean() - d.mean() ** 2), rel=1e-9, abs=1e-6)


def test_counts_far_above_a_tile_of_slots_stay_whole():
    # enough tiles that one CTA sums up all slots of a pair: rows that share almost all of 120,000 alleles
    import clotho_gb300 as cg
    n, A, free = 4_400, 120_000, 2_048
    rng = np.random.default_rng(3)
    rows = np.full((n, (A + 511) // 512 * 8), 0xffffffffffffffff, np.uint64)
    rows[:, :free // 64] = rng.integers(0, 2 ** 64, size=(n, free // 64), dtype=np.uint64)
    rows[:, free // 64::97] = 0
    with cg.Population(n // 2, A, 1) as pop:
        pop.load_population(n // 2, rows, rng.random(A), np.zeros(A, np.float32))
        got = pop.pairwise_difference(distances=True)
    bits = np.unpackbits(rows[:, :free // 64].view(np.uint8), axis=1, bitorder="little").astype(np.float32)
    ones = bits.sum(1)
    d = (ones[:, None] + ones[None, :] - 2 * (bits @ bits.T))[np.triu_indices(n, 1)]
    assert np.array_equal(got["distances"], d.astype(np.uint32))
    assert got["total"] == int(d.sum(dtype=np.float64))
