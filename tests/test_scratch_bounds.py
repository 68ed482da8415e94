"""Device memory that the calls take for themselves stays within what they say."""

import threading

import numpy as np
import pytest

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
