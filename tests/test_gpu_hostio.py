"""Copies of host arrays through the threaded lanes: sizes around the line where
they begin and around their chunks, arrays that do not fill them, calls from several
threads at once, and the batched inversion at its chunk edges."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hc(harm_lib):
    import harm_cool_b200
    return harm_cool_b200


# the lanes begin at 10 MB to the device (163,840 cells of 64 B) and at 20 MB to the host:
# just below and above each, whole and broken chunks between, and a 3D array with phi ghost
# planes
@pytest.mark.parametrize("shape", [(315, 406, 1), (316, 406, 1), (400, 400, 1), (400, 402, 1), (400, 500, 1),
                                   (568, 568, 1), (568, 570, 1), (700, 700, 1), (60, 70, 40), (60, 70, 100)])
def test_state_round_trip(shape, hc):
    pr = hc.torus_problem(*shape)
    ctx = hc.Context(pr)
    rng = np.random.default_rng(1)
    p = rng.standard_normal(pr.shape + (8,))
    fl = rng.integers(-100, 100, pr.shape).astype(np.int8)
    if shape[2] > 1:  # the phi ghosts come back as periodic copies
        for a in (p, fl):
            a[0], a[-1] = a[-2], a[1]
    ctx.put_prims(p, fl)
    q, gl = ctx.get_prims(with_flags=True)
    assert np.array_equal(p, q) and np.array_equal(fl, gl)
    ctx.close()


@pytest.mark.parametrize("shape", [(120, 128, 1), (600, 600, 1), (60, 70, 100)])
def test_pinned_arrays(shape, hc):
    """arrays the caller has pinned take one copy straight over the link"""
    import ctypes
    import torch
    pr = hc.torus_problem(*shape)
    ctx = hc.Context(pr)
    pinned = torch.empty(pr.shape + (8,), dtype=torch.float64, pin_memory=True).numpy()
    pinned[...] = np.random.default_rng(1).standard_normal(pinned.shape)
    if shape[2] > 1:
        pinned[0], pinned[-1] = pinned[-2], pinned[1]
    p = pinned.copy()
    ctx.put_prims(pinned)
    assert np.array_equal(ctx.get_prims(), p)
    pinned[...] = 0.
    ctx.lib.harm_get_prims(ctx.h, pinned.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None)
    assert np.array_equal(pinned, p)
    ctx.init_torus()
    q = ctx.get_prims()
    ctx.step_ch_host(q)
    ctx.init_torus()
    pinned[...] = ctx.get_prims()
    ctx.step_ch_host(pinned)
    assert np.array_equal(pinned, q)
    ctx.close()


def test_contexts_in_threads(hc):
    """one thread holds the lanes, the others copy plainly"""
    pr = hc.torus_problem(600, 600, 1)
    bad = []

    def work(seed):
        ctx = hc.Context(pr)
        for k in range(4):
            p = np.random.default_rng([seed, k]).standard_normal(pr.shape + (8,))
            ctx.put_prims(p)
            if not np.array_equal(ctx.get_prims(), p):
                bad.append((seed, k))
        ctx.close()
    ts = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


@pytest.mark.parametrize("n", [1, 127, 2048, 2049, 16 * 2048 + 1, 170001])
def test_batch_inversion_at_chunk_edges(n, hc):
    """every zone as it comes out alone or in any other split of the batch"""
    pr = hc.torus_problem(32, 32, 1)
    g = pr.geometry
    rng = np.random.default_rng(n)
    m = 500
    i, j = rng.integers(2, 34, m), rng.integers(2, 34, m)
    gcov, gcon = g["gcov"][i, j, 3].reshape(m, 16), g["gcon"][i, j, 3].reshape(m, 16)
    gdet = g["gdet"][i, j, 3]
    prim = np.zeros((m, 8))
    prim[:, 0], prim[:, 1] = 10. ** rng.uniform(-4, 0, m), 10. ** rng.uniform(-6, -2, m)
    U = np.zeros((m, 8))
    U[:, 0] = prim[:, 0] * gdet
    U[:, 1] = -prim[:, 1] * gdet
    U[:, 5:8] = 1e-3 * rng.standard_normal((m, 3))
    ref = prim.copy()
    ret = np.concatenate([hc.utoprim_2d_batch(U[k:k + 100], gcov[k:k + 100], gcon[k:k + 100], gdet[k:k + 100],
                                              ref[k:k + 100], 4. / 3.) for k in range(0, m, 100)])
    t = np.arange(n) % m
    out = prim[t].copy()
    got = hc.utoprim_2d_batch(U[t], gcov[t], gcon[t], gdet[t], out, 4. / 3.)
    assert np.array_equal(got, ret[t])
    assert np.array_equal(out, ref[t], equal_nan=True)


def test_batch_inversions_in_threads(hc):
    """one thread holds the lanes, the others take the plain path: the same results"""
    pr = hc.torus_problem(32, 32, 1)
    g = pr.geometry
    n = 60000
    rng = np.random.default_rng(2)
    i, j = rng.integers(2, 34, n), rng.integers(2, 34, n)
    gcov, gcon = g["gcov"][i, j, 3].reshape(n, 16), g["gcon"][i, j, 3].reshape(n, 16)
    gdet = g["gdet"][i, j, 3]
    prim = np.zeros((n, 8))
    prim[:, 0], prim[:, 1] = 10. ** rng.uniform(-4, 0, n), 10. ** rng.uniform(-6, -2, n)
    U = np.zeros((n, 8))
    U[:, 0] = prim[:, 0] * gdet
    U[:, 1] = -prim[:, 1] * gdet
    U[:, 5:8] = 1e-3 * rng.standard_normal((n, 3))
    ref = prim.copy()
    ret = hc.utoprim_2d_batch(U, gcov, gcon, gdet, ref, 4. / 3.)
    bad = []
    start = threading.Barrier(6)

    def work(k):
        start.wait()
        for _ in range(8):
            out = prim.copy()
            got = hc.utoprim_2d_batch(U, gcov, gcon, gdet, out, 4. / 3.)
            if not (np.array_equal(got, ret) and np.array_equal(out, ref, equal_nan=True)):
                bad.append(k)
    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
