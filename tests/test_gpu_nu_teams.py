"""The generator's two ways to share a node among warps (nine for up to 10,000
nodes, three above) give the same bits: a table of 10,100 nodes against single
nodes of it, and both sides of the line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LINE = 10000


@pytest.fixture(scope="module")
def hc(harm_lib):
    import harm_cool_b200
    return harm_cool_b200


@pytest.mark.parametrize("nx,ny", [(101, 100), (100, 100), (1, 3)])
def test_tables_match_single_nodes(nx, ny, hc):
    from harm_cool_b200 import eos_tables as et
    x, y = et.log_axis(nx, 1e6, 1e12) if nx > 1 else np.array([1e9]), et.log_axis(ny, 4e9, 8e10)
    hd = np.array([et.hdfac(7.0)])
    v, _ = hc.nu_tables(x, y, hd)
    rng = np.random.default_rng(4)
    i, j = rng.integers(0, nx, 40), rng.integers(0, ny, 40)
    a = hc.nu_abundance(x[i], y[j], np.full(40, hd[0]), device=0)
    got = v[0, i, j]
    for k, name in enumerate(("e", "p", "qnu", "tau")):
        np.testing.assert_array_equal(got[:, k], a[name], err_msg=name)


def test_node_list_over_the_line(hc):
    """the same 21 nodes, repeated past the line and alone"""
    from harm_cool_b200 import eos_tables as et
    rho, T = np.meshgrid(et.log_axis(7, 1e6, 1e12), et.log_axis(3, 6e9, 6e10))
    rho, T = rho.ravel(), T.ravel()
    hd = et.hdfac(5.0)
    one = hc.nu_abundance(rho, T, hd, device=0)
    n = LINE // 21 + 1
    many = hc.nu_abundance(np.tile(rho, n), np.tile(T, n), hd, device=0)
    for name in one:
        np.testing.assert_array_equal(many[name], np.tile(one[name], n), err_msg=name)
