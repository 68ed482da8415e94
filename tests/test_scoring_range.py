"""Distances whose squares leave the range of floats, or whose squares' rounding
errors do: the RMS comes from sums as good as FP64's all the same."""

import ctypes

import numpy as np
import pytest

from sky_cuda import _abi

pytestmark = pytest.mark.gpu


def _score(e):
    """One band of zeros: a sample's distance is its reference's lightness (to the square
    root's rounding, squares below 2^-126 as 0)."""
    import torch
    n = len(e)
    lab = torch.zeros((n, 3), dtype=torch.float32, device="cuda")
    lab[:, 0] = torch.as_tensor(e, device="cuda")
    bands = torch.zeros((1, n), dtype=torch.float32, device="cuda")
    res = (_abi.SkyComboScore * 1)()
    picks, weights = (ctypes.c_uint32 * 1)(0), (ctypes.c_float * 3)(1.0, 1.0, 1.0)
    lib = _abi.load_library()
    _abi.check(lib.sky_cuda_score_combos(ctypes.c_void_p(bands.data_ptr()), 1, n, ctypes.c_void_p(lab.data_ptr()), 1.0,
                                         picks, weights, 1, 1, res, None), lib)
    assert res[0].finite == n
    return res[0]


@pytest.mark.parametrize("size", [1.5e19, 1.3e18, 2.0**60, 2.0**60 * (1 - 2.0**-24), 0.731, 2.0**-40 * (1 + 2.0**-22),
                                  2.0**-40 * (1 - 2.0**-23), 1.7e-13, 3.1e-17, 1.1e-19, 1e-25, 1e-42, 0.0])
def test_equal_distances(gpu, size):
    """Mean and RMS are the distance: 32 terms of a thread off by 32 x 2^-47 of it, then some
    hundred FP64 additions."""
    r = _score(np.full(4 * 1024 + 37, size, dtype=np.float32))
    assert r.mean == pytest.approx(r.max, rel=1e-12, abs=0.0)
    assert r.rmse == pytest.approx(r.max, rel=1e-12, abs=0.0)
    assert r.max == pytest.approx(size if size > 2.0**-63 else 0.0, rel=1e-6, abs=0.0)


def test_distances_of_all_sizes(gpu):
    e = np.resize(np.array([1.5e19, 1.0, 1e-30, 0.0, 3.1e-17], dtype=np.float32), 9000)
    r = _score(e)
    assert r.rmse == pytest.approx(r.max * np.sqrt(0.2), rel=1e-12, abs=0.0)
    assert r.mean == pytest.approx((r.max + 1.0) * 0.2, rel=1e-6, abs=0.0)
