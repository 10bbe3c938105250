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
