"""Reference spectra as users hold them: read-only (a memory-mapped asset, a broadcast
view), strided, of other types."""

import warnings

import numpy as np
import pytest

from sky_cuda.scoring import score_combos

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["read-only", "strided", "list", "float32"])
def test_reference_arrays(gpu, form):
    import torch
    rng = np.random.default_rng(1)
    bands = torch.as_tensor(rng.gamma(2.0, 1.0, (5, 200)).astype(np.float32), device="cuda")
    ref = rng.uniform(0.1, 1.0, (200, 3)).astype(np.float32).astype(np.float64)
    args = np.array([[0, 3]]), np.ones((1, 2, 3), dtype=np.float32)
    want = score_combos(bands, ref, *args)
    other = {"read-only": ref.copy(), "strided": np.repeat(ref, 2, axis=0)[::2], "list": ref.tolist(),
             "float32": ref.astype(np.float32)}[form]
    if form == "read-only":
        other.flags.writeable = False
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        got = score_combos(bands, other, *args)
    assert got[0]["p50"] == want[0]["p50"] and got[0]["mean"] == pytest.approx(want[0]["mean"], rel=1e-13)
