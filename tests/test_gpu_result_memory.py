"""What a kept result holds in memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _held(a):
    """Bytes that stay allocated while this array does."""
    import torch
    while isinstance(a, np.ndarray) and a.base is not None:
        a = a.base
    return a.untyped_storage().nbytes() if isinstance(a, torch.Tensor) else a.nbytes


@pytest.mark.parametrize("n,N,dy,cplx", [(300, [40], 1, False), (20000, [24, 20], 1, False),
                                         (60000, [64], 3, False), (400000, [30, 40], 1, True),
                                         (300000, [700, 500], 1, False), (2000, [90, 80], 2, False)])
def test_a_kept_result_holds_little_more_than_itself(cuda_ok, n, N, dy, cplx):
    """Every array of a fit, and of one through cv_fastlpr_many, keeps at most
    eight times its own bytes (and 512, the granule of small allocations)."""
    import fastlpr_b200
    rng = np.random.default_rng(n)
    d = len(N)
    x = rng.random((n, d))
    y = rng.standard_normal((n, dy)) + (1j * rng.standard_normal((n, dy)) if cplx else 0)
    y = y[:, 0] if dy == 1 else y
    h = np.repeat(np.geomspace(0.1, 0.5, 4)[:, None], d, 1)
    opts = {"order": 1, "N": N if d > 1 else N[0]}
    one = fastlpr_b200.cv_fastlpr(x, y, h, dict(opts))
    many = fastlpr_b200.cv_fastlpr_many([(x, y, h, dict(opts))] * 2)
    for r in [one] + many:
        for a in (r.yhat, r.metadata["residuals"], r.fpp_yhat.values, r.s0):
            assert _held(a) <= 8 * a.nbytes + 512
        for name in ("yhat", "s0"):
            np.testing.assert_array_equal(getattr(r, name), getattr(one, name))
