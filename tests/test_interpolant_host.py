"""GridInterpolant's attributes on the CPU."""
import numpy as np
import torch

from fastlpr_b200.interpolant import GridInterpolant


def test_bounds_are_formed_once_and_can_be_set():
    f = GridInterpolant([np.linspace(0, 2, 5), np.linspace(-1, 1, 4)], np.zeros((5, 4)), torch.device("cpu"))
    assert f.bounds == [(0.0, 2.0), (-1.0, 1.0)] and f.bounds is f.bounds
    f.bounds = [(0.5, 1.0), (0.0, 0.0)]
    assert f.bounds == [(0.5, 1.0), (0.0, 0.0)]
