"""Column and row margins against numpy over the shapes where the one-pass kernel splits: rows narrower and wider
than a warp's 64 words, a last partial word group, fewer rows than a block takes together, and more rows than a
lane's eight binary digits count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,A", [(1, 1), (3, 512), (31, 513), (32, 1024), (33, 1537), (250, 4096), (257, 4097),
                                 (129, 12_801), (4_001, 40), (40_000, 300), (9_000, 5_000)])
def test_margins_match_numpy(N, A):
    import clotho_gb300 as cg
    rng = np.random.default_rng(N * 100_003 + A)
    W = (A + 511) // 512 * 8
    rows = rng.integers(0, 2 ** 64, size=(2 * N, W), dtype=np.uint64)
    rows[::7] = np.uint64(0xffffffffffffffff)   # dense rows: every column's count is large
    rows[3::11] = 0
    bits = np.unpackbits(rows.view(np.uint8), axis=1, bitorder="little")[:, :A]
    with cg.Population(N, A, 1) as pop:
        pop.load_population(N, rows, rng.random(A), np.zeros(A, np.float32))
        col, row = pop.margins()
        st = pop.stats(8)
    assert np.array_equal(col, bits.sum(0, dtype=np.uint32))
    assert np.array_equal(row, bits.sum(1, dtype=np.uint32))
    c = bits.sum(0)
    assert st["segregating"] == int(((c > 0) & (c < 2 * N)).sum())
    assert np.array_equal(st["sfs"], np.bincount(np.minimum(c, 7), minlength=8))
