"""The fixed-point sums of the FP32 spread against the same sums in integers."""
import numpy as np
import pytest

import oracle.lpr as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,nval", [(2, 1), (2, 3), (2, 12), (3, 1), (3, 2)])
def test_each_product_is_rounded_to_the_nearest_multiple_of_the_quantum(cuda_ok, d, nval):
    """One tap of weight 1, so a product is the value itself, and values halfway
    between two multiples of the quantum: every one rounds to the even multiple,
    whatever the order of the points, as numpy's rint does."""
    import torch
    from fastlpr_b200 import _lib, api
    n, G = 8192, [12] * d
    rng = np.random.default_rng(10 * d + nval)
    x = rng.random((n, d))
    vals = rng.integers(-2000, 2000, (n, nval)) + 0.5
    vals[0] = 1.5 * 2.0 ** 48      # the channel's absolute sum: quantum 1 on grids wider than the stencil
    ctx = api._Ctx(torch.device("cuda", 0))
    dx = ctx.upload(x)
    geom = api._make_geom(api._point_stats(ctx, dx, n, d), n, d, np.asarray(G), 0, True)
    cols = [ctx.upload(np.ascontiguousarray(c)) for c in vals.T]
    L, cells = _lib.ivec(geom.L), int(np.prod(geom.L))
    grid = ctx.empty((nval, cells), dtype=torch.float32)
    grid64 = ctx.empty((nval, cells))
    ws = ctx.ws(ctx.lib.flpr_spread_ws(d, n, L, 0, nval, 0))
    _lib.check(ctx.lib.flpr_spread(d, n, dx.data_ptr(), _lib.dvec(geom.kmap.ravel()), L, 0,
                                   _lib.dvec(geom.tau), nval, 0, _lib.pvec([c.data_ptr() for c in cols]),
                                   grid.data_ptr(), 0, ws.data_ptr(), ws.numel(), ctx.stream), "spread")
    _lib.check(ctx.lib.flpr_spread_grid64(d, n, L, 0, nval, ws.data_ptr(), ws.numel(),
                                          grid64.data_ptr(), ctx.stream), "grid64")
    got = grid64.cpu().numpy().reshape((nval,) + tuple(geom.L)) * n
    xs = (x - geom.mean) / geom.std - geom.center
    knots = oracle.knot_coordinates(xs, geom.L, np.asarray(G), geom.qin)
    want = oracle.spread_grid(knots, np.rint(vals), geom.L, 0, geom.tau)
    np.testing.assert_array_equal(got, want)


def _tap_weights(f, hx, ft, dtype):
    """exp(-(f - hx j)^2 / ft) of nine taps, every operation rounded to dtype."""
    j = np.arange(-4, 5)
    t = (np.asarray(f, np.longdouble)[:, None] - np.longdouble(hx) * j).astype(dtype)
    return np.exp(-(t * t) / dtype(ft))


@pytest.mark.parametrize("d", [2, 3])
def test_tap_weights_are_as_accurate_as_an_exponential_per_tap(cuda_ok, d):
    """Stencils that do not overlap, on an FP64 grid: a cell holds the product
    of d tap weights.  Its error against 80-bit arithmetic, over the error of
    the same formula in numpy: both round the argument alike, and the device's
    exponential (1 ulp at most) and the order of the products leave less than
    a sixth more.  Weights formed by recurrence have a third more."""
    import torch
    from fastlpr_b200 import _lib, api
    L, step = (512, 16) if d == 2 else (128, 16)
    rng = np.random.default_rng(d)
    cell = np.stack(np.meshgrid(*[np.arange(step // 2, L, step)] * d, indexing="ij"), -1).reshape(-1, d)
    two_pi, hx = 6.283185307179586, 2 * np.pi / L
    # knot map of mean 0 and spread 1 with a shift of 1/2: the knot of x is 2 pi (x + 1/2)
    x = (cell + rng.uniform(-0.49, 0.49, cell.shape)) / L - 0.5
    kmap = np.array([[0, 1, 0, 0, 1, 1, 0, 0.5, hx]] * d, dtype=float)
    n = x.shape[0]
    k = np.mod((np.mod(x + 0.5, 1.0) - 0.5 + 0.5) * two_pi, two_pi)
    m = np.rint(k / hx).astype(int)
    f = k - hx * m
    ft = 4 * np.pi * 4 / (L * L * 0.5)
    ctx = api._Ctx(torch.device("cuda", 0))
    dx = ctx.upload(x)
    Lv = _lib.ivec([L] * d)
    grid = ctx.empty((L,) * d)
    ws = ctx.ws(ctx.lib.flpr_spread_ws(d, n, Lv, 4, 1, 1))
    _lib.check(ctx.lib.flpr_spread(d, n, dx.data_ptr(), _lib.dvec(kmap.ravel()), Lv, 4,
                                   _lib.dvec([ft / 4] * d), 1, 1, _lib.pvec([]), grid.data_ptr(), 1,
                                   ws.data_ptr(), ws.numel(), ctx.stream), "spread")
    got = grid.cpu().numpy() * n
    num, den = 0.0, 0.0
    for i in range(n):
        w = [_tap_weights(f[i:i + 1, a], hx, ft, np.float64)[0] for a in range(d)]
        e = [_tap_weights(f[i:i + 1, a], hx, ft, np.longdouble)[0] for a in range(d)]
        w2, e2 = np.outer(w[0], w[1]), np.multiply.outer(e[0], e[1])
        if d == 3:
            w2, e2 = np.multiply.outer(w2, w[2]), np.multiply.outer(e2, e[2])
        ix = np.ix_(*[(m[i, a] + np.arange(-4, 5)) % L for a in range(d)])
        num += float(np.sum((got[ix] - e2) ** 2))
        den += float(np.sum((w2 - e2) ** 2))
    assert num ** 0.5 < 1.15 * den ** 0.5


@pytest.mark.parametrize("d,n,G,C,msp", [
    (1, 2, [2], 1, 4), (1, 255, [40], 32, 4), (1, 257, [300], 1, 4), (1, 3001, [1500], 31, 0),
    (2, 257, [40, 9], 11, 7), (2, 1500, [64, 48], 32, 12), (2, 400, [5, 20], 1, 9)])
def test_sorted_deposits_on_lines_and_under_wide_stencils(cuda_ok, d, n, G, C, msp):
    """The shared-memory deposits: one dimension, and the wider tiles of 2-D
    stencils beyond 13 taps, against one FP64 atomic per point, corner and
    channel (both round 2^-62 and 2^-53 of the channel's sum)."""
    import torch
    from conftest import rel_err
    from fastlpr_b200 import _lib, api
    rng = np.random.default_rng(n + C)
    x, cols = rng.random((n, d)), rng.standard_normal((n, C)) * 10.0 ** rng.integers(-3, 4, C)
    ctx = api._Ctx(torch.device("cuda", 0))
    dx = ctx.upload(x)
    geom = api._make_geom(api._point_stats(ctx, dx, n, d), n, d, np.asarray(G), 4, True)
    dc = [ctx.upload(np.ascontiguousarray(c)) for c in cols.T]
    ptrs = _lib.pvec([c.data_ptr() for c in dc])
    L, Gv = _lib.ivec(geom.L), _lib.ivec(G)
    grid = ctx.empty((1 + C, int(np.prod(geom.L))))
    ws = ctx.ws(ctx.lib.flpr_spread_ws(d, n, L, msp, 1 + C, 1))
    _lib.check(ctx.lib.flpr_spread(d, n, dx.data_ptr(), _lib.dvec(geom.kmap.ravel()), L, msp,
                                   _lib.dvec(geom.tau), 1 + C, 1, ptrs, grid.data_ptr(), 1,
                                   ws.data_ptr(), ws.numel(), ctx.stream), "spread")
    ax = _lib.dvec(api._axes_arg(api._raw_axes(geom, {})))
    M, NP = int(np.prod(G)), (2 ** d) * (2 ** d + 1) // 2
    a, b = ([ctx.empty((M, C)), ctx.empty((M, NP)), ctx.empty(C)] for _ in range(2))
    ws2 = ctx.ws(ctx.lib.flpr_deposit_sorted_ws(d, n, L, msp, 1 + C))
    _lib.check(ctx.lib.flpr_deposit_sorted(d, n, dx.data_ptr(), L, msp, 1 + C, 1, ptrs, ws.data_ptr(),
                                           ws.numel(), ax, Gv, _lib.ivec(api._node0_cells(geom)),
                                           *[t.data_ptr() for t in a], ws2.data_ptr(), ws2.numel(),
                                           ctx.stream), "deposit_sorted")
    _lib.check(ctx.lib.flpr_deposit(d, n, dx.data_ptr(), ax, Gv, C, ptrs,
                                    *[t.data_ptr() for t in b], ctx.stream), "deposit")
    for u, v in zip(a, b):
        u, v = u.cpu().numpy(), v.cpu().numpy()
        for k in range(u.shape[-1]):
            assert rel_err(u[..., k], v[..., k]) < 1e-12


@pytest.mark.parametrize("d,G,n", [(2, [96, 80], 40000), (3, [12, 10, 14], 60000), (1, [400], 500000)])
def test_the_item_size_setting_changes_the_work_items(cuda_ok, d, G, n):
    """Every candidate of the autotuner makes another number of work items of
    clustered points, and the same grid."""
    import torch
    from fastlpr_b200 import _lib, api, autotune
    rng = np.random.default_rng(n)
    x = 0.4 + 0.02 * rng.random((n, d))
    x[0], x[1] = 0.0, 1.0
    ctx = api._Ctx(torch.device("cuda", 0))
    dx, y = ctx.upload(x), ctx.upload(rng.standard_normal(n))
    geom = api._make_geom(api._point_stats(ctx, dx, n, d), n, d, np.asarray(G), 4, True)
    L = _lib.ivec(geom.L)
    ws = ctx.ws(ctx.lib.flpr_spread_ws(d, n, L, 4, 2, 0))
    tiles = [-(-int(v) // t) for v, t in zip(geom.L, {1: [256], 2: [8, 8], 3: [1, 8, 8]}[d])]
    # the workspace begins with the tiles' counts, their offsets and their first work items
    ntiles = int(np.prod(tiles))
    first = (-(-4 * ntiles // 256) - (-4 * (ntiles + 1) // 256)) * 64
    saved = autotune.get_params()
    items, grids = [], []
    try:
        for ip in autotune.ITEM_POINTS:
            autotune.set_params({"spread_item_points": ip})
            grid = ctx.empty((2, int(np.prod(geom.L))), dtype=torch.float32)
            _lib.check(ctx.lib.flpr_spread(d, n, dx.data_ptr(), _lib.dvec(geom.kmap.ravel()), L, 4,
                                           _lib.dvec(geom.tau), 2, 1, _lib.pvec([y.data_ptr()]),
                                           grid.data_ptr(), 0, ws.data_ptr(), ws.numel(), ctx.stream),
                       "spread")
            items.append(int(ws[:4 * (first + ntiles + 1)].view(torch.int32)[-1]))
            grids.append(grid)
    finally:
        autotune.set_params(saved)
    assert len(set(items)) == (len(items) if d > 1 else 1)
    assert all(torch.equal(g, grids[0]) for g in grids)


@pytest.mark.parametrize("m", [1023, 1024, 1025])
@pytest.mark.parametrize("d,prec", [(2, 0), (2, 1), (3, 0), (3, 1)])
def test_the_largest_work_items(cuda_ok, d, prec, m):
    """A tile that fills the largest work item but one point, all of it, and
    one point more, against the oracle; the rounding of the grid's type."""
    import torch
    from conftest import rel_err
    from fastlpr_b200 import _lib, api, autotune
    rng = np.random.default_rng(m + d)
    G, n = [40, 40, 40][:d], m + 2
    ctx = api._Ctx(torch.device("cuda", 0))
    x = 0.5 + 0.0001 * rng.random((n, d))
    x[0], x[1] = 0.0, 1.0
    dx, v = ctx.upload(x), rng.standard_normal((n, 3))
    geom = api._make_geom(api._point_stats(ctx, dx, n, d), n, d, np.asarray(G), 4, True)
    cols = [ctx.upload(np.ascontiguousarray(c)) for c in v.T]
    L = _lib.ivec(geom.L)
    grid = ctx.empty((3, int(np.prod(geom.L))), dtype=torch.float64 if prec else torch.float32)
    ws = ctx.ws(ctx.lib.flpr_spread_ws(d, n, L, 4, 3, prec))
    saved = autotune.get_params()
    try:
        autotune.set_params({"spread_item_points": 65536})
        _lib.check(ctx.lib.flpr_spread(d, n, dx.data_ptr(), _lib.dvec(geom.kmap.ravel()), L, 4,
                                       _lib.dvec(geom.tau), 3, 0, _lib.pvec([c.data_ptr() for c in cols]),
                                       grid.data_ptr(), prec, ws.data_ptr(), ws.numel(), ctx.stream), "spread")
    finally:
        autotune.set_params(saved)
    xs = (x - geom.mean) / geom.std - geom.center
    knots = oracle.knot_coordinates(xs, geom.L, np.asarray(G), geom.qin)
    want = oracle.spread_grid(knots, v, geom.L, 4, geom.tau)
    got = grid.double().cpu().numpy().reshape(want.shape) * n
    for c in range(3):
        assert rel_err(got[c], want[c]) < (1e-12 if prec else 2e-7)


@pytest.mark.parametrize("d,G,n,item", [(2, [100, 100], 20000, 64), (2, [40, 40], 20000, 64), (3, [12, 12, 12], 9000, 32),
                                        (2, [60, 80], 100000, 256)])
def test_few_points_make_small_work_items(cuda_ok, d, G, n, item):
    """Items of 32 or 64 points where items of 256 would leave most of the device idle."""
    import torch
    from fastlpr_b200 import _lib, api
    x = np.random.default_rng(n).random((n, d))
    ctx = api._Ctx(torch.device("cuda", 0))
    dx = ctx.upload(x)
    geom = api._make_geom(api._point_stats(ctx, dx, n, d), n, d, np.asarray(G), 4, True)
    L = _lib.ivec(geom.L)
    ws = ctx.ws(ctx.lib.flpr_spread_ws(d, n, L, 4, 1, 1))
    grid = ctx.empty(tuple(geom.L))
    _lib.check(ctx.lib.flpr_spread(d, n, dx.data_ptr(), _lib.dvec(geom.kmap.ravel()), L, 4,
                                   _lib.dvec(geom.tau), 1, 1, _lib.pvec([]), grid.data_ptr(), 1,
                                   ws.data_ptr(), ws.numel(), ctx.stream), "spread")
    ntiles = int(np.prod([-(-int(v) // t) for v, t in zip(geom.L, [8, 8] if d == 2 else [1, 8, 8])]))
    first = (-(-4 * ntiles // 256) - (-4 * (ntiles + 1) // 256)) * 64
    ints = ws[:4 * (first + ntiles + 1)].view(torch.int32).cpu().numpy()
    counts = ints[:ntiles]
    assert counts.sum() == n and counts.max() > item
    assert ints[-1] == np.sum(-(-counts // item))
