"""Fits of the same shape from several threads, each on its own stream."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,N", [(1, [300]), (2, [40, 48]), (3, [14, 12, 16])])
def test_threads_with_streams_of_their_own_give_the_same_fits(cuda_ok, d, N):
    """The threads share cuFFT plans; results as one after the other (FP32
    sums are exact, the FP64 reductions of a fit are not ordered: 1e-9)."""
    import torch
    import fastlpr_b200
    from conftest import rel_err
    rng = np.random.default_rng(d)
    h = np.repeat(np.geomspace(0.1, 0.5, 6)[:, None], d, 1)
    opts = {"order": 1, "N": N if d > 1 else N[0]}
    data = []
    for _ in range(4):
        x = rng.random((2000, d))
        data.append((x, np.sin(5 * x[:, 0]) + 0.1 * rng.standard_normal(2000)))
    want = [fastlpr_b200.cv_fastlpr(x, y, h, dict(opts)) for x, y in data]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            return [fastlpr_b200.cv_fastlpr(*data[i], h, dict(opts)) for _ in range(12)]

    with ThreadPoolExecutor(4) as pool:
        for i, runs in enumerate(pool.map(work, range(4))):
            for r in runs:
                assert rel_err(r.yhat, want[i].yhat) < 1e-9
                assert rel_err(r.gcv_yhat["gcv_m"], want[i].gcv_yhat["gcv_m"]) < 1e-9
