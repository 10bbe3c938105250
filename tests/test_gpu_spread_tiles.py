"""The register-accumulating spread kernels at the sizes where their work
changes shape: batches of 32 points, items of at most 1024, channels per lane
and per warp, footprints from one tap up, grids of a single tile."""
import numpy as np
import pytest

import oracle.lpr as oracle
from conftest import elem_rel_err, rel_err

pytestmark = pytest.mark.gpu

# FP64: the sums of n products in another order; FP32: half an ulp of the
# float grid (6e-8) and the fixed-point quantum, both of the largest cell
TOL = {1: 1e-12, 0: 2e-7}


def _spread(x, vals, G, msp, prec, ones=1, geom=None):
    import torch
    from fastlpr_b200 import _lib, api
    n, d = x.shape
    ctx = api._Ctx(torch.device("cuda", 0))
    dx = ctx.upload(x)
    if geom is None:
        geom = api._make_geom(api._point_stats(ctx, dx, n, d), n, d, np.asarray(G), msp, True)
    cols = [ctx.upload(np.ascontiguousarray(c)) for c in vals.T]
    C = ones + len(cols)
    grid = ctx.empty((C, int(np.prod(geom.L))), dtype=torch.float64 if prec else torch.float32)
    ws = ctx.ws(ctx.lib.flpr_spread_ws(d, n, _lib.ivec(geom.L), msp, C, prec))
    _lib.check(ctx.lib.flpr_spread(d, n, dx.data_ptr(), _lib.dvec(geom.kmap.ravel()),
                                   _lib.ivec(geom.L), msp, _lib.dvec(geom.tau), C, ones,
                                   _lib.pvec([c.data_ptr() for c in cols]), grid.data_ptr(), prec,
                                   ws.data_ptr(), ws.numel(), ctx.stream), "spread")
    torch.cuda.synchronize()
    return grid.double().cpu().numpy().reshape((C,) + tuple(geom.L)) * n, geom


def _reference(x, vals, G, geom, msp):
    xs = (x - geom.mean) / geom.std - geom.center
    xmod = oracle.knot_coordinates(xs, geom.L, np.asarray(G), geom.qin)
    return oracle.spread_grid(xmod, vals, geom.L, msp, geom.tau)


def _points(n, d, seed, clustered):
    rng = np.random.default_rng(seed)
    x = rng.random((n, d))
    if clustered:
        x[2:] = 0.4 + 0.02 * x[2:]     # a few cells hold nearly all points
        x[0], x[1] = 0.0, 1.0
    return x, rng


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("d,n,G,msp,nval,clustered", [
    (2, 2, [4, 4], 4, 0, False), (2, 31, [9, 40], 4, 1, False), (2, 33, [16, 16], 4, 3, False),
    (2, 1025, [33, 20], 4, 5, True), (2, 9000, [40, 24], 4, 8, True), (2, 4000, [64, 48], 4, 11, False),
    (2, 4000, [64, 48], 4, 12, True), (2, 3000, [30, 31], 4, 18, False), (2, 700, [17, 30], 4, 40, False),
    (2, 900, [20, 20], 0, 4, False), (2, 900, [20, 21], 1, 11, False), (2, 900, [21, 20], 2, 12, False),
    (2, 900, [5, 20], 3, 7, False), (2, 900, [20, 20], 5, 9, False), (2, 900, [20, 6], 6, 11, True),
    (3, 2, [4, 4, 4], 4, 0, False), (3, 33, [5, 9, 7], 4, 1, False), (3, 5000, [12, 16, 10], 4, 2, True),
    (3, 1025, [3, 20, 8], 3, 3, False), (3, 800, [9, 6, 12], 2, 0, False), (3, 800, [9, 9, 9], 1, 4, False),
    (3, 800, [10, 8, 9], 0, 1, False), (3, 300, [2, 9, 2], 4, 1, False), (3, 300, [6, 6, 6], 5, 1, False)])
def test_tiles_match_oracle(cuda_ok, d, n, G, msp, nval, clustered, prec):
    x, rng = _points(n, d, 7 * n + nval, clustered)
    vals = rng.standard_normal((n, nval)) * 10.0 ** rng.integers(-3, 4, nval)
    g, geom = _spread(x, vals, G, msp, prec)
    ref = _reference(x, np.column_stack([np.ones(n), vals]), G, geom, msp)
    for c in range(1 + nval):
        assert rel_err(g[c], ref[c]) < TOL[prec], c


@pytest.mark.parametrize("d,G", [(2, [32, 32]), (3, [12, 12, 12])])
def test_fixed_point_sums_do_not_depend_on_the_order(cuda_ok, d, G):
    """Knots on the cells and values of few bits: products that would round by
    the parity of the sum if ties could occur."""
    rng = np.random.default_rng(5)
    x = rng.integers(0, G[0], (6000, d)) / (G[0] - 1.0)
    x[0], x[1] = 0.0, 1.0
    vals = np.column_stack([rng.integers(-4, 5, 6000) * 0.5, np.where(np.arange(6000) == 7, 2.0 ** 51, 1.0)])
    a, geom = _spread(x, vals, G, 4, 0)
    p = np.concatenate([[0, 1], 2 + rng.permutation(5998)])
    b, _ = _spread(x[p], vals[p], G, 4, 0, geom=geom)
    np.testing.assert_array_equal(a, b)


def test_constant_channel_may_be_left_out(cuda_ok):
    x, rng = _points(2000, 2, 3, False)
    vals = rng.standard_normal((2000, 3))
    g, geom = _spread(x, vals, [30, 30], 4, 1, ones=0)
    ref = _reference(x, vals, [30, 30], geom, 4)
    for c in range(3):
        assert rel_err(g[c], ref[c]) < TOL[1]


@pytest.mark.parametrize("d,n,G,C,narrow", [
    (2, 2, [4, 4], 1, False), (2, 255, [9, 40], 10, False), (2, 257, [40, 9], 11, False),
    (2, 3000, [30, 31], 12, True), (2, 1500, [64, 48], 23, False), (2, 700, [5, 20], 32, True),
    (2, 5000, [16, 16], 2, True), (1, 300, [40], 11, False)])
def test_sorted_deposits_at_the_edges(cuda_ok, d, n, G, C, narrow):
    """Sorted deposits against one FP64 atomic per point, corner and channel;
    `narrow`: a raw grid inside the data, so points lie beyond it."""
    import torch
    from fastlpr_b200 import _lib, api
    x, rng = _points(n, d, 11 * n + C, n == 5000)
    cols = rng.standard_normal((n, C)) * 10.0 ** rng.integers(-3, 4, C)
    ctx = api._Ctx(torch.device("cuda", 0))
    dx = ctx.upload(x)
    geom = api._make_geom(api._point_stats(ctx, dx, n, d), n, d, np.asarray(G), 4, True)
    dc = [ctx.upload(np.ascontiguousarray(c)) for c in cols.T]
    ptrs = _lib.pvec([c.data_ptr() for c in dc])
    L, Gv = _lib.ivec(geom.L), _lib.ivec(G)
    grid = ctx.empty((1 + C, int(np.prod(geom.L))), dtype=torch.float32)
    ws = ctx.ws(ctx.lib.flpr_spread_ws(d, n, L, 4, 1 + C, 0))
    _lib.check(ctx.lib.flpr_spread(d, n, dx.data_ptr(), _lib.dvec(geom.kmap.ravel()), L, 4,
                                   _lib.dvec(geom.tau), 1 + C, 1, ptrs, grid.data_ptr(), 0,
                                   ws.data_ptr(), ws.numel(), ctx.stream), "spread")
    ax = _lib.dvec(api._axes_arg(api._raw_axes(geom, {"xrange": [[0.2, 0.7]] * d} if narrow else {})))
    M, NP = int(np.prod(G)), (2 ** d) * (2 ** d + 1) // 2

    def outputs():
        return ctx.empty((M, C)), ctx.empty((M, NP)), ctx.empty(C)

    a, b = outputs(), outputs()
    ws2 = ctx.ws(ctx.lib.flpr_deposit_sorted_ws(d, n, L, 4, 1 + C))
    _lib.check(ctx.lib.flpr_deposit_sorted(d, n, dx.data_ptr(), L, 4, 1 + C, 1, ptrs, ws.data_ptr(),
                                           ws.numel(), ax, Gv, _lib.ivec(api._node0_cells(geom)),
                                           a[0].data_ptr(), a[1].data_ptr(), a[2].data_ptr(),
                                           ws2.data_ptr(), ws2.numel(), ctx.stream), "deposit_sorted")
    _lib.check(ctx.lib.flpr_deposit(d, n, dx.data_ptr(), ax, Gv, C, ptrs, b[0].data_ptr(),
                                    b[1].data_ptr(), b[2].data_ptr(), ctx.stream), "deposit")
    torch.cuda.synchronize()
    for c in range(C):
        assert rel_err(a[0][:, c].cpu().numpy(), b[0][:, c].cpu().numpy()) < 1e-12
    for u, v in zip(a[1:], b[1:]):
        assert rel_err(u.cpu().numpy(), v.cpu().numpy()) < 1e-12


@pytest.mark.parametrize("d,n,G,ny,mstride,f32", [(1, 2, [2], 1, 1, True), (1, 5000, [40], 2, 12, False),
                                                  (2, 257, [30, 7], 3, 3, True), (3, 900, [4, 5, 6], 1, 1, False),
                                                  (2, 50, [60, 50], 4, 5, False)])
def test_fit_outputs_match_their_parts(cuda_ok, d, n, G, ny, mstride, f32):
    import torch
    from fastlpr_b200 import _lib, api
    rng = np.random.default_rng(n)
    ctx = api._Ctx(torch.device("cuda", 0))
    M, H = int(np.prod(G)), 3
    x = ctx.upload(rng.random((n, d)) * 1.2 - 0.1)
    m, y = ctx.upload(rng.standard_normal((H, M, mstride))), ctx.upload(rng.standard_normal((ny, n)))
    S = ctx.upload(rng.random((H, M))).to(torch.float32 if f32 else torch.float64)
    ax, Gv = _lib.dvec([0.0, 1.0 / 40] * d), _lib.ivec(G)
    for pick in (0, 2, -1):
        sel = torch.tensor([pick], dtype=torch.int32, device=x.device)
        yh, res, surf, s0, so = (ctx.empty(s) for s in ((n, ny), (n, ny), (M, ny), (M,), (1,)))
        _lib.check(ctx.lib.flpr_fit_outputs(
            d, n, x.data_ptr(), ax, Gv, ny, mstride, H, m.data_ptr(), S.data_ptr(), 0 if f32 else 1,
            sel.data_ptr(), _lib.pvec([y[c].data_ptr() for c in range(ny)]), yh.data_ptr(),
            res.data_ptr(), surf.data_ptr(), s0.data_ptr(), so.data_ptr(), ctx.stream), "outputs")
        assert float(so[0]) == pick
        if pick < 0:
            assert all(bool(torch.isnan(t).all()) for t in (yh, res, surf, s0))
            continue
        vals, ref = m[pick][:, :ny].t().contiguous(), ctx.empty((ny, n))
        _lib.check(ctx.lib.flpr_interp_eval(d, n, x.data_ptr(), ax, Gv, ny, vals.data_ptr(),
                                            ref.data_ptr(), ctx.stream), "interp_eval")
        assert torch.equal(yh, ref.t()) and torch.equal(res, y.t() - ref.t())
        assert torch.equal(surf, vals.t()) and torch.equal(s0, S[pick].double())


@pytest.mark.parametrize("n", [1, 255, 257, 700000])
def test_input_stats_flags(cuda_ok, n):
    import torch
    from fastlpr_b200 import api
    rng = np.random.default_rng(n)
    ctx = api._Ctx(torch.device("cuda", 0))
    x, y = rng.random((n, 2)), rng.random((2, n))

    def flags(x, y):
        dx, dy = ctx.upload(x), ctx.upload(y)
        v = api._input_stats_dev(ctx, dx, n, 2, [dy[0], dy[1]]).cpu().numpy()
        return v[:8], list(v[8:])

    st, fl = flags(x, y)
    assert fl == [0, 0, 0, 0]
    np.testing.assert_array_equal(st, api._point_stats(ctx, ctx.upload(x), n, 2).ravel())
    for k, (bad, where) in enumerate([(np.nan, 0), (-np.inf, 0), (np.nan, 1), (np.inf, 1)]):
        xx, yy = x.copy(), y.copy()
        if where == 0:
            xx[n - 1, 1] = bad
        else:
            yy[1, n - 1] = bad
        assert flags(xx, yy)[1] == [float(j == k) for j in range(4)]


@pytest.mark.parametrize("d,n,G,H", [(1, 40, [30], 1), (1, 3000, [50], 17), (2, 33, [9, 12], 7), (2, 2000, [20, 31], 9),
                                     (3, 500, [6, 9, 7], 16), (3, 300, [5, 5, 6], 20), (1, 300, [16], 530)])
def test_density_scores_at_the_edges(cuda_ok, d, n, G, H):
    """Bandwidths that fill 8 or 16 lanes or not, a last batch of one point,
    more bandwidths than one launch takes; FP64, so to 1e-9 of the oracle."""
    import fastlpr_b200
    rng = np.random.default_rng(13 * n + H)
    x = rng.standard_normal((n, d))
    h = np.column_stack([np.linspace(0.3, 1.2, H)] * d)
    opts = {"N": G if d > 1 else G[0], "precision": "fp64"}
    k, o = fastlpr_b200.cv_fastkde(x, h, dict(opts)), oracle.cv_fastkde(x, h, {"N": opts["N"]})
    assert rel_err(k.metadata["fhat_all"], o["fhat_all"]) < 1e-9
    assert rel_err(k.lcv["lcv_m"], o["lcv_m"]) < 1e-9 and rel_err(k.lcv["lcv_sd"], o["lcv_sd"]) < 1e-9


@pytest.mark.parametrize("C", [1, 4, 5, 12, 13, 24, 25, 32])
@pytest.mark.parametrize("order,nt,f32", [(0, 1, True), (1, 3, True), (1, 4, False), (2, 6, True)])
def test_solve_reduce_channels(cuda_ok, C, order, nt, f32):
    """Every padded channel count, against the unfused solve and its sums."""
    import torch
    from fastlpr_b200 import _lib, api
    rng = np.random.default_rng(C * 10 + nt)
    ctx = api._Ctx(torch.device("cuda", 0))
    H, M, keep, prec = 3, 1237, min(C, 2), 0 if f32 else 1
    real = torch.float32 if f32 else torch.float64
    A = rng.standard_normal((H, M, nt, nt + 2))
    A = A @ A.transpose(0, 1, 3, 2)
    S = np.stack([A[:, :, i, j] for i in range(nt) for j in range(i, nt)])
    S, T = ctx.upload(S).to(real), ctx.upload(rng.standard_normal((nt, C, H, M))).to(real)
    Q = ctx.upload(rng.standard_normal((M, C)))
    m, kept, dots, sc = (ctx.empty(s) for s in ((H, M, C), (H, M, keep), (C, H), (1,)))
    a = (order, nt, H, H, M, C, S.data_ptr(), T.data_ptr(), 1e-6)
    _lib.check(ctx.lib.flpr_solve(*a, m.data_ptr(), sc.data_ptr(), prec, ctx.stream), "solve")
    _lib.check(ctx.lib.flpr_solve_reduce(*a, keep, kept.data_ptr(), Q.data_ptr(), dots.data_ptr(),
                                         sc.data_ptr(), prec, ctx.stream), "solve_reduce")
    m, kept, q = m.cpu().numpy(), kept.cpu().numpy(), Q.cpu().numpy()
    np.testing.assert_allclose(kept, m[:, :, :keep], rtol=1e-9, atol=1e-9)
    scale = np.einsum("hmc,mc->ch", np.abs(m), np.abs(q))
    assert np.all(np.abs(dots.cpu().numpy() - np.einsum("hmc,mc->ch", m, q)) <= 1e-11 * scale)


@pytest.mark.parametrize("prec,tol", [("fp32", 1e-5), ("fp64", 1e-11)])
@pytest.mark.parametrize("order,dof", [(0, False), (0, True), (1, False)])
@pytest.mark.parametrize("G", [[20, 24], [48, 40], [90, 120], [200, 250], [300, 400]])
def test_row_products_up_to_the_nyquist_term(cuda_ok, G, order, dof, prec, tol):
    """Kernels narrower than a grid step fill the whole band: every element of a
    row, the real DC and Nyquist ones too, single products and pairs, for each
    transform length."""
    import fastlpr_b200
    rng = np.random.default_rng(G[0] + order)
    n = 40 * G[0] * G[1]
    x = rng.random((n, 2))
    y = np.sin(2 * np.pi * x[:, 0]) * np.cos(2 * np.pi * x[:, 1]) + 0.1 * rng.standard_normal(n)
    step = np.sqrt(12.0) / np.array(G)
    h = np.outer([0.8, 1.5, 4.0], step)
    opts = {"order": order, "N": G, "precision": prec, "calc_dof": dof}
    a = fastlpr_b200.cv_fastlpr(x, y, h, opts)
    b = fastlpr_b200.cv_fastlpr(x, y, h, dict(opts, _no_fused=True))
    assert rel_err(a.yhat, b.yhat) < tol and rel_err(a.s0, b.s0) < tol
    assert elem_rel_err(a.gcv_yhat["gcv_m"], b.gcv_yhat["gcv_m"]) < tol
