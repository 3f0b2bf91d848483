"""Pairwise differences of rows at and above the slots that one CTA sums up, with more tiles than share scratch at a
time.  Every row is one of 40 dense patterns, so the exact distances, their total and their squares follow from the
patterns' own; a pair of full rows has as many common alleles as there are slots, the largest sum there is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("A,n", [(524_288, 8_192), (524_289, 16_384)])
def test_many_tiles_of_wide_rows(A, n):
    import clotho_gb300 as cg
    rng = np.random.default_rng(A)
    K, W = 40, (A + 511) // 512 * 8
    bits = rng.random((K, A)) < np.linspace(0.9, 1.0, K)[:, None]
    bits[0] = False
    bits[-1] = True
    packed = np.zeros((K, W * 8), np.uint8)
    packed[:, :(A + 7) // 8] = np.packbits(bits, axis=1, bitorder="little")
    which = rng.integers(0, K, n)
    which[:2] = 0, K - 1
    rows = packed.view(np.uint64)[which]
    d = np.array([[np.count_nonzero(a != b) for b in bits] for a in bits], np.int64)
    with cg.Population(n // 2, A, 1) as pop:
        pop.load_population(n // 2, rows, rng.random(A), np.zeros(A, np.float32))
        del rows
        pop.pairwise_difference(n=16)
        free = cg.device_memory()[0]
        got = pop.pairwise_difference()
        used = free - cg.device_memory()[0]
        full = pop.pairwise_difference(distances=True)
    assert used <= 256 << 20, f"{used >> 20} MB of scratch"
    c = np.bincount(which, minlength=K).astype(object)
    total = sum(int(d[i, j]) * c[i] * c[j] for i in range(K) for j in range(K)) // 2
    squares = sum(int(d[i, j]) ** 2 * c[i] * c[j] for i in range(K) for j in range(K)) // 2
    pairs = n * (n - 1) // 2
    for r in (got, full):
        assert (r["count"], r["total"], r["min"], r["max"]) == (pairs, total, 0, A)
        assert r["mean"] == pytest.approx(total / pairs, rel=1e-12)
        assert r["variance"] == pytest.approx(squares / pairs - (total / pairs) ** 2, rel=1e-9)
    at = 0
    for i in range(n - 1):
        assert np.array_equal(full["distances"][at:at + n - 1 - i], d[which[i], which[i + 1:]]), i
        at += n - 1 - i
