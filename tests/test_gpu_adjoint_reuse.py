"""The adjoint keeps its buffers and graphs in the context between calls: a call
after others with the same or other step counts, another state, another tile or
steps in between gives what a fresh context gives (the gradient's sums are atomic,
so to their rounding: 1e-12 of its norm)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hc(harm_lib):
    import harm_cool_b200
    return harm_cool_b200


def start(hc, pr):
    ctx = hc.Context(pr)
    ctx.init_torus()
    ctx.run(20)
    return ctx


def test_repeated_calls_match_a_fresh_context(hc):
    pr = hc.torus_problem(40, 36, 1)
    a = start(hc, pr)
    p, t = a.get_prims(), a.time()
    calls = [(6, 2, 1.0, None), (6, 2, 1.0, None), (6, 2, 1.01, None), (5, 3, 1.0, None), (1, 1, 1.0, None),
             (6, 2, 1.0, (64, 2)), (3, 10, 0.99, None)]
    for nsteps, every, scale, tile in calls:
        q = p.copy()
        q[..., 0] *= scale
        if tile:
            a.set_tile(*tile)
        got = []
        for ctx in (a, start(hc, pr)):
            ctx.put_prims(q)
            ctx.set_time(*t)
            J, g, _ = ctx.adjoint_mass_in(nsteps, every)
            got.append((J, g, ctx.get_prims(), ctx.time()))
        (J, g, e, s), (J1, g1, e1, s1) = got
        assert abs(J - J1) <= 1e-14 * abs(J1) and s == s1
        assert np.array_equal(e, e1)
        assert np.linalg.norm(g - g1) <= 1e-12 * np.linalg.norm(g1), (nsteps, every, scale)
        a.run(2)
    a.close()


def test_a_failed_call_leaves_the_next_one_whole(hc):
    pr = hc.torus_problem(24, 24, 1)
    a, b = start(hc, pr), start(hc, pr)
    p, t = a.get_prims(), a.time()
    a.adjoint_mass_in(3, 2)
    a.put_prims(p)
    a.set_time(pr.params.tf - 1e-3, 1e-3)  # the steps reach tf: refused
    with pytest.raises(hc.HarmError):
        a.adjoint_mass_in(3, 2)
    out = []
    for ctx in (a, b):
        ctx.put_prims(p)
        ctx.set_time(*t)
        out.append(ctx.adjoint_mass_in(3, 2)[:2])
    assert abs(out[0][0] - out[1][0]) <= 1e-13 * abs(out[1][0])
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 1e-12 * np.linalg.norm(out[1][1])


@pytest.mark.parametrize("nsteps", [1, 4])
def test_checkpoints_farther_apart_than_the_steps(nsteps, hc):
    """One segment, however far apart the checkpoints are asked for: what
    checkpoint_every = nsteps gives."""
    pr = hc.torus_problem(24, 24, 1)
    ctx = start(hc, pr)
    p, t = ctx.get_prims(), ctx.time()
    out = []
    for every in (nsteps, nsteps + 1, 1000, 2 ** 31 - 1):
        ctx.put_prims(p)
        ctx.set_time(*t)
        out.append(ctx.adjoint_mass_in(nsteps, every)[:2])
    for J, g in out[1:]:
        assert abs(J - out[0][0]) <= 1e-14 * abs(out[0][0])
        assert np.linalg.norm(g - out[0][1]) <= 1e-12 * np.linalg.norm(out[0][1])
    ctx.close()


@pytest.mark.parametrize("nsteps,every", [(5, 5), (7, 4), (8, 4), (13, 4)])
def test_one_two_and_more_segments_agree(nsteps, every, hc):
    """Full and short last segments in either set of records, against checkpoints at
    every step (the gradient's sums are atomic: 1e-12 of its norm)."""
    pr = hc.torus_problem(24, 24, 1)
    ctx = start(hc, pr)
    p, t = ctx.get_prims(), ctx.time()
    out = []
    for e in (1, every, every):
        ctx.put_prims(p)
        ctx.set_time(*t)
        out.append(ctx.adjoint_mass_in(nsteps, e)[:2])
    for J, g in out[1:]:
        assert abs(J - out[0][0]) <= 1e-14 * abs(out[0][0])
        assert np.linalg.norm(g - out[0][1]) <= 1e-12 * np.linalg.norm(out[0][1])
    ctx.close()


def test_another_tile_where_the_tile_is_used(hc):
    """above 56,832 zones the kept graphs are captured again for another tile"""
    pr = hc.torus_problem(241, 240, 1)
    ctx = start(hc, pr)
    p, t = ctx.get_prims(), ctx.time()
    out = []
    for tile in ((32, 4), (64, 2), (64, 2), (8, 16)):
        ctx.put_prims(p)
        ctx.set_time(*t)
        ctx.set_mass(0., 0.)  # J is a difference of the counter
        ctx.set_tile(*tile)
        out.append(ctx.adjoint_mass_in(3, 2)[:2])
    for J, g in out[1:]:
        assert J == out[0][0]
        assert np.linalg.norm(g - out[0][1]) <= 1e-12 * np.linalg.norm(out[0][1])
    ctx.close()


def test_kept_memory_is_given_back(hc):
    """by harm_adjoint_release, by another precision and by COOL_EOS; the next call makes
    it again"""
    import torch
    from harm_cool_b200 import eos_tables as et
    pr = hc.torus_problem(64, 64, 1)
    ctx = start(hc, pr)
    p, t = ctx.get_prims(), ctx.time()
    eos = hc.Eos(*et.build_tables(et.zone_radii(pr), gam=pr.params.gam))
    ctx.set_precision(ctx.MIXED)  # the buffers of both, made once
    ctx.set_eos(eos)
    ctx.set_eos(None)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]
    out = []
    for release in (ctx.adjoint_release, lambda: ctx.set_precision(ctx.MIXED), lambda: ctx.set_eos(eos),
                    ctx.adjoint_release):
        ctx.set_precision(ctx.FP64)
        ctx.set_eos(None)
        ctx.put_prims(p)
        ctx.set_time(*t)
        ctx.set_mass(0., 0.)
        out.append(ctx.adjoint_mass_in(20, 20)[:2])
        before = free()
        release()
        assert free() - before > 50e6  # 20 records twice of some 2 MB each
        ctx.adjoint_release()          # nothing kept: no error
    for J, g in out[1:]:
        assert J == out[0][0]
        assert np.linalg.norm(g - out[0][1]) <= 1e-12 * np.linalg.norm(out[0][1])
    ctx.close()
    eos.close()
