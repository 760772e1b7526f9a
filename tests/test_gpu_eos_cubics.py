"""Tabulated T-direction cubics against the general way (tables whose missing nodes
are tracked take it): pressures, their differences and the guesses they leave, bit for
bit, over the table, its edges, points on nodes and points outside, for axes of 3 nodes
and more, in FP64 and with FP32 interpolation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(72, 72), (3, 4), (4, 3), (4, 4), (5, 40)])
@pytest.mark.parametrize("mixed", [False, True])
def test_tabulated_cubics_match_the_general_way(nx, ny, mixed, harm_lib):
    import harm_cool_b200 as hc
    from harm_cool_b200 import eos_tables as et
    gam = 4. / 3.
    xa, ya, val, consts = et.build_tables([3., 7., 40.], nx=nx, ny=ny, gam=gam)
    a, b = hc.Eos(xa, ya, val, consts), hc.Eos(xa, ya, val, consts)
    b.track_missing()
    rng = np.random.default_rng(nx * ny)
    n = 20000
    tab = rng.integers(0, 3, n).astype(np.int32)
    rho = 10. ** rng.uniform(1.5, 15.5, n)
    rho[:2000] = xa[rng.integers(0, nx, 2000)]               # on nodes
    rho0 = rho / consts["rho_unit"]
    T = 10. ** rng.uniform(4.2, 17.8, n)
    T[1000:3000] = ya[rng.integers(0, ny, 2000)]
    e = et.ideal_gas_radiation(np.clip(rho, xa[0], xa[-1]), T, 1.)[0]
    u = e * rng.uniform(0.5, 2., n) / consts["u_unit"]
    u[5000:7000] = e[5000:7000] / consts["u_unit"]
    guess = np.where(rng.random(n) < 0.3, 0., T * rng.uniform(0.3, 3., n))
    guess[1000:3000] = T[1000:3000]
    for what in ("pressure", "dpdu", "dpdrho"):
        p, g = a.batch(what, tab, rho0, u, guess, mixed=mixed)
        q, h = b.batch(what, tab, rho0, u, guess, mixed=mixed)
        assert np.array_equal(p, q, equal_nan=True) and np.array_equal(g, h, equal_nan=True), what
    assert not b.missing().any()
    a.close()
    b.close()
