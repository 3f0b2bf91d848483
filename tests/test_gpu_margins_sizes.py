"""Margins at the largest populations: more strips of rows than a grid's second dimension takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_more_than_130_million_rows():
    # 40-word rows, the narrowest with a warp to each: 1,984 of them a block
    import clotho_gb300 as cg
    N, A = 65_100_000, 2_049
    desc = cg.make_desc(N, A, 1, mu=0.0, rho=0.0, max_fixed=1)
    if cg.footprint_of(desc) > 0.75 * cg.device_memory()[0]:
        pytest.skip("needs a device with 250 GB")
    thr = np.zeros(A, np.uint32)
    thr[[0, 63, 64, 700, 2_047, 2_048]] = 0xffffffff, 1 << 31, 1 << 31, 1 << 10, 1 << 31, 0xffffffff
    with cg.Population(N, A, 1, mu=0.0, rho=0.0, max_fixed=1) as pop:
        pop.seed_population(N, np.linspace(0, 1, A, endpoint=False), np.zeros(A, np.float32), thr, 5)
        col, row = pop.margins()
        st = pop.stats(4)
    p = thr / 2.0 ** 32
    assert np.abs(col - 2.0 * N * p).max() < 8 * np.sqrt(2.0 * N * 0.25)
    assert np.array_equal(np.flatnonzero(col), np.flatnonzero(thr))
    assert int(col.sum(dtype=np.uint64)) == int(row.sum(dtype=np.uint64))
    assert row.min() >= 0 and row.max() <= 6 and abs(float(row[-1_000_000:].mean()) - p.sum()) < 0.02
    assert st["segregating"] == int(((col > 0) & (col < 2 * N)).sum())
