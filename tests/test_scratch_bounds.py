"""Device memory that the calls take for themselves stays within what they say."""

import ctypes
import threading

import numpy as np
import pytest

from sky_cuda import _abi
from sky_cuda.mie import MieDistribution, bake_phase

import mie_oracle as mo

pytestmark = pytest.mark.gpu


def _most_used(call):
    """Device bytes in use during `call` over those before it, looked at all the time."""
    import torch
    torch.cuda.synchronize()
    start, _ = torch.cuda.mem_get_info()
    least, done = [start], threading.Event()

    def watch():
        while not done.is_set():
            least[0] = min(least[0], torch.cuda.mem_get_info()[0])

    t = threading.Thread(target=watch)
    t.start()
    try:
        call()
    finally:
        done.set()
        t.join()
    return start - least[0]


def test_mie_series_scratch(gpu):
    """A bake is refused where its derivatives' recurrences (max(terms, |m x|) + 17 entries of 16
    bytes an item) and coefficients (terms of 16 bytes) exceed 16 GB: it takes no more than those."""
    bands, radii = 40, 250
    r = np.geomspace(190.0, 210.0, radii)
    lam = np.linspace(500.0, 600.0, bands)
    terms = [[mo.mie_terms(2.0 * np.pi * v / (w * 1e-3)) for v in r] for w in lam]
    series = 16 * (2 * int(np.sum(terms)) + 17 * bands * radii)
    bake_phase(MieDistribution(1.0, 2.0, 0.9, 1.1, radii=4), [550.0], [1.0 + 1e-3j], bins=8)  # the first call's set-up

    def bake():
        for _ in range(5):
            bake_phase(MieDistribution(200.0, 2.0, 190.0, 210.0, radii=radii), lam, np.full(bands, 1.0 + 1e-3j), bins=8)

    used = _most_used(bake)
    # besides the series: items, efficiencies and whole pages (2 MB an allocation)
    assert 0.5 * series < used <= series + 120 * bands * radii + (24 << 20), (used, series)


def test_score_scratch(gpu):
    """The states of a fixed number of combinations are held at a time, however many there are;
    the scores do not depend on how they fall into passes."""
    import torch
    samples, combos, channels = 33, 500_000, 4
    rng = np.random.default_rng(3)
    bands = torch.as_tensor(rng.gamma(2.0, 1.0, (7, samples)).astype(np.float32), device="cuda")
    lab = torch.as_tensor(rng.uniform(0.0, 1.0, (samples, 3)).astype(np.float32), device="cuda")
    picks = rng.integers(0, 7, (combos, channels)).astype(np.uint32)
    xyz = rng.uniform(0.1, 1.0, (combos, channels, 3)).astype(np.float32)
    lib = _abi.load_library()

    def score(first, count):
        res = (_abi.SkyComboScore * count)()
        p, x = picks[first:first + count], xyz[first:first + count]
        _abi.check(lib.sky_cuda_score_combos(
            ctypes.c_void_p(bands.data_ptr()), 7, samples, ctypes.c_void_p(lab.data_ptr()), 1.0,
            p.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), x.ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
            count, channels, res, None), lib)
        return res

    score(0, 1)
    found = []
    used = _most_used(lambda: found.append(score(0, combos)))
    # 1024 combinations' histograms (5 of 2048 words), 8192 states (88 B), bands and weights (16 B a channel),
    # the distances of 1024 combinations, whole pages
    most = 1024 * 5 * 2048 * 4 + 8192 * (88 + 16 * channels) + 1024 * samples * 4 + (8 << 20)
    assert 40 << 20 < used <= most, (used, most)
    for first in (0, 8190, 16383, combos - 3):
        for i, one in enumerate(score(first, 3)):
            whole = found[0][first + i]
            assert one.finite == whole.finite == samples
            for f in ("p50", "p90", "p95", "p99", "max"):
                assert getattr(one, f) == getattr(whole, f)
            for f in ("mean", "rmse", "score"):  # FP64 sums in any order
                assert getattr(one, f) == pytest.approx(getattr(whole, f), rel=1e-13)
