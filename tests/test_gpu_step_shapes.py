"""The step's kernels at the sizes where their tiling can go wrong: rows of
faces just below, at and above the 64 faces of a flux block, the smallest grids,
odd sizes, and each limiter, bit for bit against the oracle (the FP64 path keeps
the reference's arithmetic, so the bound is equality)."""
import numpy as np
import pytest

from helpers import active, make_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hc(harm_lib):
    import harm_cool_b200
    return harm_cool_b200


@pytest.mark.parametrize("shape,lim", [((6, 8, 1), 0), ((21, 61, 1), 1), ((33, 62, 1), 0), ((20, 63, 1), 2),
                                       ((64, 128, 1), 0), ((9, 10, 4), 0), ((13, 62, 4), 1), ((31, 30, 6), 0),
                                       ((18, 64, 4), 2)])
def test_steps_match_oracle_at_tile_edges(shape, lim, hc, oracle_built):
    pr = hc.torus_problem(*shape, lim=lim)
    ctx = hc.Context(pr)
    ctx.init_torus()
    o = make_oracle(pr)
    p, fl = ctx.get_prims(with_flags=True)
    o.p[...] = p
    o.pflag[...] = fl
    o.set_time(*ctx.time())
    for n in range(4):
        ctx.step_ch()
        ctx.sync()
        assert o.step() == 0
        p, fl = ctx.get_prims(with_flags=True)
        np.testing.assert_array_equal(active(pr, p), active(pr, o.p), err_msg="step %d" % n)
        np.testing.assert_array_equal(active(pr, fl), active(pr, o.pflag))
        assert ctx.time() == o.time()
    ctx.close()
