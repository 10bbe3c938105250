"""Coordinates that lie in no cell of the grid: NaN, and an axis without extent."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _usable():
    import torch
    torch.cuda.synchronize()
    assert float(torch.ones(3, device="cuda").sum()) == 3.0


@pytest.mark.parametrize("d,method,extrapolate", [(1, "linear", False), (2, "linear", False), (3, "linear", False),
                                                  (2, "linear", True), (2, "cubic", False)])
def test_nan_queries_give_nan_and_leave_the_others_alone(cuda_ok, d, method, extrapolate):
    import torch
    from fastlpr_b200.interpolant import GridInterpolant
    rng = np.random.default_rng(d)
    axes = [np.linspace(0, 1, 6 + a) for a in range(d)]
    f = GridInterpolant(axes, rng.random([len(a) for a in axes]), torch.device("cuda", 0), method=method,
                        extrapolate=extrapolate)
    pts = rng.random((70, d))
    want = f(pts)
    bad = pts.copy()
    bad[::7, d - 1] = np.nan
    got = f(bad)
    assert np.all(np.isnan(got[::7]))
    keep = np.arange(70) % 7 != 0
    np.testing.assert_array_equal(got[keep], want[keep])
    _usable()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("d,n", [(1, 300), (2, 300), (2, 20000), (3, 400)])
def test_a_constant_predictor_is_refused(cuda_ok, d, n, precision):
    """As the oracle does: every GCV score is NaN."""
    import fastlpr_b200
    import oracle.lpr as oracle
    rng = np.random.default_rng(n + d)
    x = rng.random((n, d))
    x[:, d - 1] = 0.7
    y = np.sin(3 * x[:, 0]) + 0.1 * rng.standard_normal(n)
    h = np.repeat([[0.2], [0.4]], d, 1)
    opts = {"order": 0, "N": [12] * d, "gcv_interp_method": "linear", "dof_interp_method": "linear"}
    with pytest.raises(ValueError, match="All GCV scores"):
        oracle.cv_fastlpr(x, y, h, dict(opts))
    with pytest.raises(ValueError, match="All GCV scores"):
        fastlpr_b200.cv_fastlpr(x, y, h, dict(opts, precision=precision))
    _usable()


@pytest.mark.parametrize("d", [1, 2, 3])
def test_nan_points_on_the_device_stay_in_range(cuda_ok, d):
    """cv_fastlpr_device does not scan its inputs: whatever a NaN point gives,
    no kernel leaves its arrays."""
    import torch
    import fastlpr_b200
    rng = np.random.default_rng(d)
    x = torch.from_numpy(rng.random((900, d))).cuda()
    x[17, d - 1] = float("nan")
    y = torch.from_numpy(rng.standard_normal(900)).cuda()
    for precision in ("fp32", "fp64"):
        try:
            fastlpr_b200.cv_fastlpr_device(x, y, np.repeat([[0.2], [0.4]], d, 1),
                                           {"order": 1, "N": [12] * d, "precision": precision})
        except ValueError:
            pass
        _usable()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("d", [1, 2, 3])
def test_a_density_of_a_constant_predictor_is_refused(cuda_ok, d, precision):
    """As the oracle does: its scores are NaN."""
    import fastlpr_b200
    import oracle.lpr as oracle
    x = np.random.default_rng(d).random((500, d))
    x[:, d - 1] = 0.3
    h, N = np.repeat([[0.2], [0.4]], d, 1), [16] * d if d > 1 else 16
    with pytest.raises(ValueError, match="NaN or Inf"):
        oracle.cv_fastkde(x, h, {"N": N})
    with pytest.raises(ValueError, match="NaN or Inf"):
        fastlpr_b200.cv_fastkde(x, h, {"N": N, "precision": precision})
    _usable()
