"""Products and their inverse transforms: workspaces sized by the transforms
that run, lengths that are no powers of two, batches with a remainder."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("G,L,qout,nprod", [
    ([2, 2, 2], [4, 4, 4], [1, 1, 1], 1), ([5, 6, 7], [11, 13, 15], [6, 7, 8], 3),
    ([9, 4, 31], [18, 7, 63], [9, 3, 32], 7), ([21, 30, 17], [41, 59, 34], [0, 29, 17], 5),
    ([1, 3, 3], [3, 5, 6], [2, 2, 3], 520)])
def test_3d_products_fit_the_workspace_of_their_grid(cuda_ok, G, L, qout, nprod, prec):
    """flpr_conv with exactly the bytes of flpr_conv_grid_ws, and with those of
    flpr_conv_ws, against numpy's transform of the whole padded grid.  FP64:
    rounding of about 60 additions along three axes; FP32: of the values stored
    between the passes."""
    import torch
    from fastlpr_b200 import _lib, api
    ctx = api._Ctx(torch.device("cuda", 0))
    rng = np.random.default_rng(sum(L) + nprod)
    H, npow, C = 3, 2, 2
    half = L[0] * L[1] * (L[2] // 2 + 1)
    spec = np.fft.rfftn(rng.standard_normal((C, *L)), axes=(1, 2, 3))
    F = [np.fft.fft(rng.standard_normal((H, npow, n)), axis=-1) for n in L]
    prods = [(int(rng.integers(C)), int(rng.integers(H)), [int(v) for v in rng.integers(npow, size=3)])
             for _ in range(nprod)]
    sp = torch.from_numpy(spec.reshape(C, half).astype(np.complex64 if prec == 0 else np.complex128)).cuda()
    Fd = torch.from_numpy(np.concatenate([f.ravel() for f in F])).cuda()
    Gc, Lc, qc = _lib.ivec(G), _lib.ivec(L), _lib.ivec(qout)
    args = (_lib.ivec([p[0] for p in prods]), _lib.ivec([p[1] for p in prods]),
            _lib.ivec([v for p in prods for v in p[2]]))
    want = []
    for c, h, pw in prods:
        k = (F[0][h, pw[0]][:, None, None] * F[1][h, pw[1]][None, :, None]
             * F[2][h, pw[2]][None, None, :L[2] // 2 + 1])
        full = np.fft.irfftn(spec[c] * k, s=L, axes=(0, 1, 2)) * np.prod(L) * 0.37
        want.append(full[tuple(slice(q, q + g) for q, g in zip(qout, G))].ravel())
    for size in (ctx.lib.flpr_conv_grid_ws(ctx.handle, 3, Gc, Lc, nprod, prec),
                 ctx.lib.flpr_conv_ws(ctx.handle, 3, Lc, nprod, prec)):
        assert size > 0
        out = ctx.empty((nprod, int(np.prod(G))), dtype=torch.float64 if prec else torch.float32)
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        _lib.check(ctx.lib.flpr_conv(ctx.handle, 3, Gc, Lc, qc, H, npow, sp.data_ptr(), Fd.data_ptr(),
                                     nprod, *args, 0.37, 0, out.data_ptr(), prec, ws.data_ptr(), size,
                                     ctx.stream), "conv")
        assert rel_err(out.double().cpu().numpy(), np.array(want)) < (1e-13 if prec else 1e-5)
    few = torch.empty(256, dtype=torch.uint8, device="cuda")
    assert ctx.lib.flpr_conv(ctx.handle, 3, Gc, Lc, qc, H, npow, sp.data_ptr(), Fd.data_ptr(), nprod, *args,
                             0.37, 0, out.data_ptr(), prec, few.data_ptr(), 256, ctx.stream) != 0


def _conv1d(G, L, nprod, prec):
    """A 1-D product list ready to run, its output and what it should be."""
    import torch
    from fastlpr_b200 import _lib, api
    ctx = api._Ctx(torch.device("cuda", 0))
    rng = np.random.default_rng(L + nprod)
    spec = np.fft.rfft(rng.standard_normal(L))
    F = np.fft.fft(rng.standard_normal(L))
    sp = torch.from_numpy(spec.astype(np.complex64 if prec == 0 else np.complex128)).cuda()
    Fd = torch.from_numpy(F).cuda()
    Gc, Lc, qc, zero = _lib.ivec([G]), _lib.ivec([L]), _lib.ivec([L - G]), _lib.ivec([0] * nprod)
    out = ctx.empty((nprod, G), dtype=torch.float64 if prec else torch.float32)
    ws = ctx.ws(ctx.lib.flpr_conv_grid_ws(ctx.handle, 1, Gc, Lc, nprod, prec))

    def run():
        _lib.check(ctx.lib.flpr_conv(ctx.handle, 1, Gc, Lc, qc, 1, 1, sp.data_ptr(), Fd.data_ptr(), nprod,
                                     zero, zero, zero, 1.0 / L, 0, out.data_ptr(), prec, ws.data_ptr(),
                                     ws.numel(), ctx.stream), "conv")
    return run, out, np.fft.irfft(spec * F[:L // 2 + 1], L)[L - G:], (sp, Fd, ws)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("G,L", [(1, 2), (2047, 4093), (2048, 4094), (2049, 4096), (4097, 8191),
                                 (100001, 200003), (1, 65538), (65537, 65537)])
def test_long_rows_are_cut_into_pieces(cuda_ok, G, L, prec):
    """1-D products around the length of a piece (2048 elements of a spectrum
    or of the kept grid) against numpy; FP32: a transform's 1e-6 times the three
    of a prime length."""
    run, out, want, _keep = _conv1d(G, L, 3, prec)
    run()
    for row in out.double().cpu().numpy():
        assert rel_err(row, want) < (1e-12 if prec else 2e-5)


def test_one_long_row_takes_no_longer_than_many_short_ones(cuda_ok):
    """The same number of elements as one 1-D product and as 1024 of them: the
    device is filled by both (a block per product took 30 times as long)."""
    import torch

    def ms(G, L, nprod):
        run, _, _, _keep = _conv1d(G, L, nprod, 0)
        times = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            run()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return np.median(times[2:])

    assert ms(1 << 20, 1 << 21, 1) < 5.0 * ms(1 << 10, 1 << 11, 1 << 10)
