"""The scoring kernels at the edges of their tiles, chunks and histograms:
few and ragged samples, combinations off the block's group, equal distances,
non-finite samples, more combinations than one chunk of distances holds; and
the reference's scale and Oklab against the host's reference_scale and oklab."""

import ctypes

import numpy as np
import pytest

from sky_cuda._abi import check, load_library
from sky_cuda.scoring import oklab, reference_scale, score_combos

from test_scoring import _numpy_score

pytestmark = pytest.mark.gpu

NAMES = ("mean", "rmse", "p50", "p90", "p95", "p99", "max", "score")


def _case(samples, combos, channels, seed):
    rng = np.random.default_rng(seed)
    bands = rng.gamma(2.0, 1.0, (7, samples)).astype(np.float32)
    ref = bands.astype(np.float64).T @ rng.uniform(0.0, 1.0, (7, 3))
    picks = rng.integers(0, 7, (combos, channels))
    coeff = rng.uniform(0.5, 3.0, (combos, channels, 3)).astype(np.float32)
    return bands, ref, picks, coeff


def _close(got, want):
    # the tolerance of test_scoring: FP32 distances with cube roots on the special-function unit
    assert got["finite"] == want["finite"]
    for k in NAMES:
        assert got[k] == pytest.approx(want[k], rel=2e-4, abs=2e-6), k


@pytest.mark.parametrize("samples,combos,channels", [(1, 1, 1), (2, 5, 3), (31, 4, 2), (1023, 3, 4), (1024, 1, 5),
                                                     (1025, 9, 1), (30011, 6, 7)])
def test_sizes(gpu, samples, combos, channels):
    import torch
    bands, ref, picks, coeff = _case(samples, combos, channels, samples)
    got = score_combos(torch.as_tensor(bands, device="cuda"), ref, picks, coeff)
    scale = reference_scale(ref[:, 1])
    for c in range(combos):
        _close(got[c], _numpy_score(bands, ref, picks[c], coeff[c], scale))


def test_more_than_one_chunk(gpu):
    import torch
    bands, ref, picks, coeff = _case(200_003, 90, 2, 5)  # 2^24 / 200 003 = 83, in groups of 4: 80 a chunk
    got = score_combos(torch.as_tensor(bands, device="cuda"), ref, picks, coeff)
    scale = reference_scale(ref[:, 1])
    for c in (0, 79, 80, 82, 83, 89):
        _close(got[c], _numpy_score(bands, ref, picks[c], coeff[c], scale))


def test_equal_distances_and_samples_left_out(gpu):
    """All distances equal (every target in one bin to the last bit), some samples not finite, one
    combination with none that is."""
    import torch
    bands = np.ones((2, 500), dtype=np.float32)
    bands[0, 100:] = np.inf
    bands[1, :] = np.nan
    ref = np.full((500, 3), 0.5)
    coeff = np.full((2, 1, 3), 0.25, dtype=np.float32)
    a, b = score_combos(torch.as_tensor(bands, device="cuda"), ref, np.array([[0], [1]]), coeff, scale=1.0)
    assert a["finite"] == 100 and a["p50"] == a["p90"] == a["p95"] == a["p99"] == a["max"] > 0.0
    assert a["mean"] == pytest.approx(a["max"], rel=1e-12) and a["rmse"] == pytest.approx(a["max"], rel=1e-7)
    assert b["finite"] == 0 and all(np.isnan(b[k]) for k in NAMES)


@pytest.mark.parametrize("samples", [1, 2, 1000, 70_001])
@pytest.mark.parametrize("kind", ["positive", "mixed", "none"])
def test_reference_scale_and_lab(gpu, samples, kind):
    import torch
    rng = np.random.default_rng(samples)
    ref = rng.lognormal(0.0, 3.0, (samples, 3))
    if kind == "mixed":
        ref *= rng.choice([-1.0, 0.0, 1.0], (samples, 3))
        ref[rng.random(samples) < 0.3, 1] = np.nan
        ref[rng.random(samples) < 0.1, 1] = -np.inf
    if kind == "none":
        ref[:, 1] = np.nan
    lib = load_library()
    d = torch.as_tensor(ref, device="cuda")
    lab = torch.empty((samples, 3), dtype=torch.float32, device="cuda")
    scale = ctypes.c_double(0.0)
    check(lib.sky_cuda_score_reference(ctypes.c_void_p(d.data_ptr()), samples, None, ctypes.c_void_p(lab.data_ptr()),
                                       ctypes.byref(scale), None), lib)
    assert scale.value == reference_scale(ref[:, 1])  # an element of the data: exact
    want = oklab(ref / scale.value)
    ok = np.isfinite(want).all(axis=1)
    # FP64 on both sides, one rounding to float; the sums may cancel to the rounding of their largest term
    big = np.abs(np.cbrt(ref[ok] / scale.value)).max(axis=1, keepdims=True) if ok.any() else 1.0
    assert np.all(np.abs(lab.cpu().numpy()[ok] - want[ok]) <= 2.0**-23 * np.abs(want[ok]) + 2.0**-44 * big)
