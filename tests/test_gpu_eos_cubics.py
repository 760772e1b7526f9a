"""Tabulated T-direction cubics against the general way (batch calls on tables whose
missing nodes are tracked take it): pressures, their differences and the guesses they leave, bit for
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


def cool_run(pr, eos, mixed):
    import harm_cool_b200 as hc
    ctx = hc.Context(pr)
    ctx.init_torus()
    if mixed:
        ctx.set_precision(ctx.MIXED)
    ctx.set_eos(eos)
    ctx.run(1)
    ctx.run(4)
    out = ctx.get_prims(with_flags=True) + (ctx.eos_guess(),)
    ctx.close()
    return out


@pytest.mark.parametrize("mixed", [False, True])
def test_steps_on_tracked_tables(mixed, harm_lib):
    """A COOL_EOS step takes the tabulated cubics of tracked tables where they are
    finite: on complete tables it marks nothing, and filling only the nodes it marks,
    none around them, ends in the same state bit for bit (a NaN node that a run read
    without marking it would stay in its state).  The nodes with the smallest and the
    largest e and p are there from the start: they set the tables' scale in float."""
    import harm_cool_b200 as hc
    from harm_cool_b200 import eos_tables as et
    pr = hc.torus_problem(24, 20, 1, a=0.6, rin=4.0, rmax=11.8, beta=50.0)
    xa, ya, val, consts = et.build_tables(et.zone_radii(pr), nx=30, ny=30, rho=(1.e4, 1.e14), T=(1.e8, 1.e12),
                                          gam=pr.params.gam)
    consts["rho_unit"] = 1.e11
    consts["u_unit"] = consts["p_unit"] = 1.e11 * et.CL * et.CL
    eos = hc.Eos(xa, ya, val, consts)
    full = cool_run(pr, eos, mixed)
    eos.track_missing()
    same = cool_run(pr, eos, mixed)
    assert not eos.missing().any()
    eos.close()

    def fill(v, xa, ya, hd, mask, device):
        v[mask] = val[mask]
        return int(mask.sum()), 0.
    ends = [np.unravel_index(f(val[..., k]), val.shape[:3]) for k in (0, 1) for f in (np.argmin, np.argmax)]

    def make_eos(xa, ya, v, consts):
        for at in ends:
            v[at] = val[at]
        return hc.Eos(xa, ya, v, consts)
    lazy, how, have = et.on_demand(lambda e: cool_run(pr, e, mixed), xa, ya, consts, margin=0, max_passes=400,
                                   make_eos=make_eos, fill=fill)
    assert 0 < how["nodes"] < how["nodes_total"]
    for a, b, c in zip(full, same, lazy):
        assert np.array_equal(a, b) and np.array_equal(a, c)
