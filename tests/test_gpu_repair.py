"""fixup_utoprim's repair paths at their edges, bit for bit against the oracle: one
failure, the longest list, one more (the plane repair), every zone; rows that
fill the ordered pass's block and one row too many for it; several phi planes, one
of them without failures; and gamma failures, which change the flags that later
zones' stencils read."""
import ctypes

import numpy as np
import pytest

from helpers import active, make_oracle

pytestmark = pytest.mark.gpu
LIST = 12  # FIX_LIST_MAX


@pytest.fixture(scope="module")
def hc(harm_lib):
    import harm_cool_b200
    return harm_cool_b200


def repair_both(hc, pr, fail, expect_marks=False):
    """fixup_utoprim on the same state and flags by the device and by the oracle."""
    from oracle.pyoracle import oracle_lib
    dp = ctypes.POINTER(ctypes.c_double)
    ctx = hc.Context(pr)
    rng = np.random.default_rng(3)
    p = np.zeros(pr.shape + (8,))
    p[..., 0] = 10. ** rng.uniform(-6, 0, pr.shape)
    p[..., 1] = p[..., 0] * 10. ** rng.uniform(-4, -1, pr.shape)
    p[..., 2:5] = rng.uniform(-.05, .05, pr.shape + (3,))
    p[..., 5:8] = 1e-3 * rng.standard_normal(pr.shape + (3,))
    fl = np.zeros(pr.shape, dtype=np.int8)
    active(pr, fl)[:, 2:-2, 2:-2] = fail
    ctx.put_prims(p, fl)
    a, b = p.copy(), p.copy()
    o = make_oracle(pr)
    o.pflag[...] = fl
    ctx.lib.harm_fixup_utoprim(ctx.h, a.ctypes.data_as(dp))
    oracle_lib().ora_fixup_utoprim(o.h, b.ctypes.data_as(dp))
    np.testing.assert_array_equal(active(pr, a)[:, 2:-2, 2:-2], active(pr, b)[:, 2:-2, 2:-2])
    _, fg = ctx.get_prims(with_flags=True)
    np.testing.assert_array_equal(active(pr, fg)[:, 2:-2, 2:-2], active(pr, o.pflag)[:, 2:-2, 2:-2])
    assert (active(pr, fg) == -33).any() == expect_marks
    ctx.close()


def flags(shape, count, seed=1):
    n1, n2, n3 = shape
    f = np.zeros(n1 * n2 * n3, dtype=np.int8)
    f[np.random.default_rng(seed).permutation(f.size)[:count]] = 101
    return f.reshape(n3, n1, n2)


@pytest.mark.parametrize("shape,count", [((20, 24, 1), 1), ((20, 24, 1), LIST), ((20, 24, 1), LIST + 1),
                                         ((20, 24, 1), 250), ((20, 24, 1), 480), ((7, 9, 1), 63), ((5, 300, 1), 1200),
                                         ((511, 8, 1), 3000), ((512, 8, 1), 3000), ((12, 10, 4), LIST),
                                         ((12, 10, 4), LIST + 1), ((12, 10, 4), 480)])
def test_repairs_match_oracle(shape, count, hc, oracle_built):
    repair_both(hc, hc.torus_problem(*shape), flags(shape, count))


def test_planes_without_failures_stay(hc, oracle_built):
    f = flags((16, 12, 6), 0)
    f[1, 3:9, 2:11] = 1
    f[4] = 2
    repair_both(hc, hc.torus_problem(16, 12, 6), f)


@pytest.mark.parametrize("shape", [(20, 24, 1), (12, 10, 4)])
def test_gamma_failures_repair_in_loop_order(shape, hc, oracle_built):
    """A metric whose theta entry is negative in some zones makes their floors
    fail in gamma, wherever the repair leaves a theta velocity (stencil averages)."""
    pr = hc.torus_problem(*shape)
    rng = np.random.default_rng(8)
    sick = rng.random((shape[0] + 4, shape[1] + 4)) < 0.3
    g = pr.geometry["gcov"]
    g[sick, 3, 2, 2] *= -1e4
    f = flags(shape, shape[0] * shape[1] * shape[2] // 4, seed=5)
    repair_both(hc, pr, f, expect_marks=True)


def clump(shape, count, at=(0, 0)):
    """count failures side by side in every phi plane but the second, in a near square
    whose first zone is at"""
    n1, n2, n3 = shape
    f = np.zeros((n3, n1, n2), dtype=np.int8)
    w = min(max(int(np.ceil(np.sqrt(count))), -(-count // (n2 - at[1]))), n1 - at[0])
    q = np.zeros((w, -(-count // w)), dtype=np.int8)
    q.reshape(-1)[:count] = 1
    f[:, at[0]:at[0] + w, at[1]:at[1] + q.shape[1]] = q
    if n3 > 1:
        f[1] = 0
    return f


# few lines with last resorts (swept alone), most of them (the ordered pass over all),
# more failures than the list holds (8,192) of either kind and more than a quarter of the
# zones, more rows than the ordered pass has threads (511), and more lines than bits (8,192)
@pytest.mark.parametrize("shape,f", [
    ((60, 80, 1), [(40, (0, 0))]), ((60, 80, 1), [(100, (50, 70)), (60, (3, 2))]), ((60, 80, 1), [(900, (20, 30))]),
    ((60, 80, 1), [(4300, (0, 0))]), ((200, 100, 1), [(8192, (5, 5))]), ((200, 100, 1), [(8193, (5, 5))]),
    ((150, 330, 1), [(8200, (0, 100))]), ((520, 40, 1), [(35, (500, 3))]), ((530, 40, 1), [(20000, (0, 0))]),
    ((8, 8300, 1), [(64, (0, 8000)), (50, (1, 4))]), ((8, 8300, 1), [(9000, (0, 100))]),
    ((24, 20, 6), [(30, (3, 4))]), ((24, 20, 6), [(400, (0, 0))]), ((70, 50, 10), [(1200, (10, 0))]),
    ((70, 50, 10), [(60, (60, 30)), (80, (0, 0))]), ((96, 80, 8), [(1300, (20, 30))])])
def test_clumps_match_oracle(shape, f, hc, oracle_built):
    fail = np.zeros((shape[2],) + shape[:2], dtype=np.int8)
    for count, at in f:
        fail |= clump(shape, count, at)
    repair_both(hc, hc.torus_problem(*shape), fail)


@pytest.mark.parametrize("shape,count", [((20, 24, 1), 32), ((20, 24, 1), 33), ((12, 10, 4), 32), ((12, 10, 4), 33),
                                         ((200, 100, 1), 9000), ((40, 36, 8), 9000), ((256, 192, 1), 700),
                                         ((96, 80, 8), 8192), ((96, 80, 8), 9000), ((96, 80, 8), 15360)])
def test_scattered_failures_match_oracle(shape, count, hc, oracle_built):
    repair_both(hc, hc.torus_problem(*shape), flags(shape, count))


@pytest.mark.parametrize("shape,count", [((60, 80, 1), 50), ((200, 100, 1), 9000), ((150, 330, 1), 8200),
                                         ((24, 20, 6), 60), ((96, 80, 8), 1200)])
def test_gamma_failures_in_clumps(shape, count, hc, oracle_built):
    """as test_gamma_failures_repair_in_loop_order, on few lines and beyond the list"""
    pr = hc.torus_problem(*shape)
    rng = np.random.default_rng(8)
    sick = rng.random((shape[0] + 4, shape[1] + 4)) < 0.3
    pr.geometry["gcov"][sick, 3, 2, 2] *= -1e4
    f = clump(shape, count, (10, 3)) | flags(shape, count // 2, seed=5)
    repair_both(hc, pr, f, expect_marks=True)
