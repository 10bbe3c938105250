"""Density scores of few bandwidths: lanes are not left idle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,G", [(1, [30]), (2, [9, 12]), (3, [6, 7, 5])])
@pytest.mark.parametrize("H", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n", [33, 1000])
def test_scores_of_few_bandwidths_match_the_oracle(cuda_ok, d, G, H, n):
    import fastlpr_b200
    import oracle.lpr as oracle
    from conftest import rel_err
    x = np.random.default_rng(n + H).standard_normal((n, d))
    h = np.repeat(np.geomspace(0.3, 0.9, H)[:, None], d, 1)
    opts = {"N": G if d > 1 else G[0], "precision": "fp64"}
    got, want = fastlpr_b200.cv_fastkde(x, h, dict(opts)), oracle.cv_fastkde(x, h, {"N": opts["N"]})
    assert rel_err(got.lcv["lcv_m"], want["lcv_m"]) < 1e-9
    assert rel_err(got.lcv["lcv_sd"], want["lcv_sd"]) < 1e-9


def test_one_bandwidth_takes_less_than_eight(cuda_ok):
    """4e6 points on a line: a third of the time measured, with eight lanes
    for every point whatever the number of bandwidths the same."""
    import torch
    from fastlpr_b200 import _lib, api
    ctx = api._Ctx(torch.device("cuda", 0))
    n, G = 4000000, 1024
    x = ctx.upload(np.random.default_rng(1).random((n, 1)))
    Gv, ax = _lib.ivec([G]), _lib.dvec([0.0, 1.0 / (G - 1)])

    def ms(H):
        s = torch.rand((H, G), dtype=torch.float64, device=x.device) + 0.5
        f, lcv = ctx.empty((H, G)), ctx.empty((H, 2))
        ws = ctx.ws(ctx.lib.flpr_kde_ws(n, H, G))
        _lib.check(ctx.lib.flpr_kde_density(1, n, Gv, H, s.data_ptr(), 1, 1.0 / G, f.data_ptr(),
                                            ws.data_ptr(), ws.numel(), ctx.stream), "density")
        times = []
        for _ in range(9):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            _lib.check(ctx.lib.flpr_kde_scores(1, n, x.data_ptr(), None, ax, Gv, H, _lib.dvec([1.0] * H),
                                               lcv.data_ptr(), ws.data_ptr(), ws.numel(), ctx.stream),
                       "scores")
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return np.median(times[2:])

    assert ms(1) < 0.7 * ms(8)
