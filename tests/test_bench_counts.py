"""bench.py's count of kernel launches per step against the step's launch sequence, read
from the sources: which launches a half step makes for 2D, 3D, small, large and COOL_EOS
grids."""
import os
import re

import pytest

import bench
from harm_cool_b200 import build as hb


def source(name):
    return open(os.path.join(hb.CSRC, name)).read()


def test_fused_size_is_the_sources():
    text = source("harm_common.cuh")
    minb = int(re.search(r"UPD_MINB = (\d+);", text).group(1))
    sms, threads = re.search(r"FUSED_ZONES = (\d+)L \* UPD_MINB \* (\d+);", text).groups()
    assert bench.FUSED_ZONES == int(sms) * minb * int(threads)


# 2D: flux, update, repair, or flux, emf, cons, invert, bound, repair; 3D: flux, emf, update (or
# cons, invert), bound, repair, bound; and the sums once a step
@pytest.mark.parametrize("grid,count", [((128, 128, 1), 2 * 3 + 1), ((444, 128, 1), 2 * 3 + 1),
                                        ((445, 128, 1), 2 * 6 + 1), ((256, 256, 1), 2 * 6 + 1),
                                        ((24, 20, 6), 2 * 6 + 1), ((70, 50, 22), 2 * 7 + 1),
                                        ((288, 256, 256), 2 * 7 + 1)])
def test_gamma_law_launches(grid, count):
    assert bench.kernels_per_step(*grid) == count


def test_cool_launches():
    assert bench.kernels_per_step(256, 256, 1, cool=True) == 2 * 5 + 1
    assert bench.kernels_per_step(256, 256, 1, cool=True, tracers=True) == 2 * 5 + 2
    assert bench.kernels_per_step(16, 16, 4, cool=True) == 2 * 8 + 1


@pytest.mark.gpu
@pytest.mark.parametrize("grid,mixed,cool,tracers", [((64, 60, 1), False, False, False), ((241, 240, 1), True, False, False),
                                                     ((24, 20, 6), True, False, False), ((70, 50, 22), False, False, True),
                                                     ((32, 32, 1), False, True, False), ((32, 32, 1), True, True, True)])
def test_count_is_what_a_step_launches(grid, mixed, cool, tracers, harm_lib):
    torch = pytest.importorskip("torch")
    import harm_cool_b200 as hc
    from harm_cool_b200 import eos_tables as et
    from torch.profiler import ProfilerActivity, profile
    pr = hc.torus_problem(*grid, **(dict(a=0.6, rin=4.0, rmax=11.8, beta=50.0) if cool else {}))
    ctx = hc.Context(pr)
    ctx.init_torus()
    if mixed:
        ctx.set_precision(ctx.MIXED)
    if cool:
        ctx.set_eos(hc.Eos(*et.build_tables(et.zone_radii(pr), gam=pr.params.gam)))
    if tracers:
        ctx.tracers_put([(5, 5, 1 if grid[2] > 1 else 0)], [[1., 0.5, 0.1]])
    ctx.run(2)
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        ctx.run(3)
        torch.cuda.synchronize()
    n = sum(e.count for e in prof.key_averages() if "harm::" in e.key)
    if n == 0:
        pytest.skip("kernels are not traced here")
    assert n == 3 * bench.kernels_per_step(*grid, cool=cool, tracers=tracers)
    ctx.close()
