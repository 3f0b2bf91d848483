"""A batch's blocks are dealt out in proportion to its populations' capacities: populations from one individual to
many times a block's, in one batch, give the rows, margins and sizes they give alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("row_blocks", [0, 1, 16])
def test_blocks_in_proportion_change_no_result(row_blocks):
    import clotho_gb300 as cg
    kw = [dict(N=1, acap=200, T=1, rho=0.5, fitness="constant"), dict(N=12_000, acap=9_000, T=2, rho=4.0,
          fitness="gaussian"), dict(N=3, acap=70_000, T=4, rho=2.0, fitness="quadratic"),
          dict(N=513, acap=2_000, T=1, rho=0.0, fitness="constant")]
    descs = [cg.make_desc(k["N"], k["acap"], k["T"], mu=0.05, rho=k["rho"], p_neutral=0.3, fitness=k["fitness"],
                          fit_param=9.0, seed=11 + i) for i, k in enumerate(kw)]
    b = cg.Batch(descs)
    if row_blocks:
        b.set_tuning(row_blocks_per_sm=row_blocks)
    b.init()
    b.run(5)
    for i, d in enumerate(descs):
        one = cg.Batch([d])
        one.init()
        one.run(5)
        assert np.array_equal(b.rows(i), one.rows(0))
        for x, y in zip(b.margins(i), one.margins(0)):
            assert np.array_equal(x, y)
        assert b.info(i) == one.info(0)
        one.close()
    b.close()
