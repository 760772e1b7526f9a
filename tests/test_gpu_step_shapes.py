"""The step's kernels at the sizes where their tiling can go wrong: rows of
faces just below, at and above the 64 faces of a flux block, the smallest grids,
odd sizes, each limiter, and both sides of the zone counts where the update goes from
one launch to several (56,832) and the inversion from one phi plane a block to four
(606,208), with phi planes that do not fill a group of four, bit for bit against the
oracle (the FP64 path keeps the reference's arithmetic, so the bound is equality)."""
import numpy as np
import pytest

from helpers import active, l1_rel, make_oracle

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


def perturbed(hc, pr):
    """The torus with 4 % noise on its internal energy, on the device and the oracle."""
    ctx = hc.Context(pr)
    ctx.init_torus()
    p, fl = ctx.get_prims(with_flags=True)
    act = active(pr, p)[:, 2:-2, 2:-2, 1]
    act *= 1. + 4e-2 * (np.random.default_rng(5).random(act.shape) - 0.5)
    ctx.put_prims(p, fl)
    o = make_oracle(pr)
    p, fl = ctx.get_prims(with_flags=True)
    o.p[...] = p
    o.pflag[...] = fl
    o.set_time(*ctx.time())
    return ctx, o


@pytest.mark.parametrize("shape", [(237, 239, 1), (241, 240, 1), (64, 148, 6), (101, 97, 6), (260, 240, 10)])
def test_steps_match_oracle_across_the_launch_rules(shape, hc, oracle_built):
    pr = hc.torus_problem(*shape)
    ctx, o = perturbed(hc, pr)
    for n in range(2):
        ctx.step_ch()
        ctx.sync()
        assert o.step() == 0
        p, fl = ctx.get_prims(with_flags=True)
        np.testing.assert_array_equal(active(pr, p), active(pr, o.p), err_msg="step %d" % n)
        np.testing.assert_array_equal(active(pr, fl), active(pr, o.pflag))
        assert ctx.time() == o.time()
    ctx.close()


@pytest.mark.parametrize("shape", [(237, 239, 1), (241, 240, 1), (64, 148, 6), (101, 97, 6), (260, 240, 10)])
def test_mixed_step_tracks_oracle_across_the_launch_rules(shape, hc, oracle_built):
    """one mixed step at FP32 round-off of the faces: 1e-6 in density, as on small grids"""
    pr = hc.torus_problem(*shape)
    ctx, o = perturbed(hc, pr)
    ctx.set_precision(hc.Context.MIXED)
    ctx.run(1)
    assert o.step() == 0
    l1 = l1_rel(active(pr, ctx.get_prims()), active(pr, o.p))
    assert l1[0] <= 1e-6, l1
    ctx.close()


@pytest.mark.parametrize("shape", [(40, 36, 1), (241, 240, 1), (24, 20, 6)])
def test_single_steps_before_and_after_the_graph(shape, hc):
    """a context's first single steps are launched kernel by kernel, later ones from the
    graph, and after a change of precision kernel by kernel again: the same steps"""
    pr = hc.torus_problem(*shape)
    a, b = hc.Context(pr), hc.Context(pr)
    for c in (a, b):
        c.init_torus()
    for n, mode in ((11, a.FP64), (2, a.MIXED), (9, a.FP64)):
        for c in (a, b):
            c.set_precision(mode)
        a.run(n)
        for k in range(n):
            if k % 2:
                b.step_ch()
            else:
                p = b.get_prims()
                b.step_ch_host(p)
        np.testing.assert_array_equal(a.get_prims(), b.get_prims())
        assert a.time() == b.time()
    a.close()
    b.close()
