"""Margins at the largest populations (more strips of rows than a grid's second dimension takes), and around the size up
to which both come in one copy."""
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


@pytest.mark.parametrize("N,A", [(1, 1), (7_935, 400), (7_936, 400), (7_937, 400), (20, 16_383), (20, 15_872)])
def test_margins_in_one_copy_or_two(N, A):
    # 16,384 counts in all at N = 7,936 and A = 400 (512 columns and 15,872 rows)
    import ctypes as C

    import clotho_gb300 as cg
    rng = np.random.default_rng(N + A)
    W = (A + 511) // 512 * 8
    rows = rng.integers(0, 2 ** 64, size=(2 * N, W), dtype=np.uint64)
    bits = np.unpackbits(rows.view(np.uint8), axis=1, bitorder="little")[:, :A]
    with cg.Population(N, A, 1) as pop:
        pop.load_population(N, rows, rng.random(A), np.zeros(A, np.float32))
        for want_col, want_row in ((True, True), (True, False), (False, True)):
            col, row = np.full(A + 8, 77, np.uint32), np.full(2 * N + 8, 77, np.uint32)
            p = [x.ctypes.data_as(C.c_void_p) if on else None for x, on in ((col, want_col), (row, want_row))]
            assert pop.L.clotho_margins(pop.h, *p) == 0
            assert np.array_equal(col[:A], bits.sum(0, dtype=np.uint32) if want_col else np.full(A, 77))
            assert np.array_equal(row[:2 * N], bits.sum(1, dtype=np.uint32) if want_row else np.full(2 * N, 77))
            assert (col[A:] == 77).all() and (row[2 * N:] == 77).all()
