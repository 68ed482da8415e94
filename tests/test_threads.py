"""Host threads with scenes of their own: every call succeeds and returns what it
returns alone, whatever size of tables another thread's launches of the same
kernels need.  A thread repeats its call for a second and a half."""

import threading
import time

import numpy as np
import pytest

from sky_cuda import GpuScene, RenderConfig, synthetic_scene, wavelengths
from sky_cuda import _abi
from sky_cuda.mie import MieDistribution, bake_phase
from sky_cuda.scene import SyntheticAtmosphere

pytestmark = pytest.mark.gpu


def _scene(data_dir, bands, layers=64):
    return synthetic_scene(wavelengths(400.0, 700.0, bands), data_dir, sun_elevation_deg=10.0,
                           atmosphere=SyntheticAtmosphere(layers=layers))


def _chains(per_lane):
    import torch
    return per_lane * 1024 * torch.cuda.get_device_properties(0).multi_processor_count


def _render(scene, chains, tracking):
    spp = -(-chains // (32 * 16 * scene.band_count))
    gs = GpuScene(scene)
    cfg = RenderConfig(width=32, height=16, spp=spp, phase_sampling=_abi.PHASE_TABULATED, tracking=tracking)
    return lambda: gs.render(cfg)[0].values


def _gradient(scene, chains):
    import torch
    from sky_cuda.adjoint import AdjointRenderer
    spp = -(-chains // (32 * 16 * scene.band_count))
    r = AdjointRenderer(GpuScene(scene), RenderConfig(width=32, height=16, spp=spp,
                                                      phase_sampling=_abi.PHASE_TABULATED))
    layer = torch.ones(r.param_count, device="cuda")
    layer[-2], layer[-1] = 0.9, 0.7
    dloss = torch.ones((16, 32, r.bands), device="cuda")
    return lambda: r.backward(layer, None, dloss)[0].cpu().numpy()


def _bake(radius_um):
    """One sphere of a series long enough for more than 48 KB of coefficients."""
    d = MieDistribution(radius_um, 1.5, radius_um, radius_um, radii=1)
    return lambda: bake_phase(d, [550.0], [1.5 + 0.5j], bins=64)[0]


CALLS = {
    "stage queues": lambda data: [_render(_scene(data, b), _chains(3), _abi.TRACKING_RESIDUAL_CARRY)
                                  for b in (81, 4, 40, 200)],
    "ray loop": lambda data: [_render(_scene(data, 81, n), 32 * 16 * 81 * 4, _abi.TRACKING_MERGED_LAYERS)
                              for n in (1000, 760, 900, 820)],
    "gradient": lambda data: [_gradient(_scene(data, 8, n), _chains(45)) for n in (64, 20, 90, 48)],
    "mie": lambda data: [_bake(r) for r in (300.0, 400.0, 500.0, 350.0)],
}


@pytest.mark.parametrize("kind", list(CALLS))
def test_scenes_of_different_sizes_in_threads(gpu, data_dir, kind):
    calls = CALLS[kind](data_dir)
    alone = [c() for c in calls]
    found, failed = [None] * len(calls), []

    def repeat(i):
        end = time.time() + 1.5
        while time.time() < end and not failed:
            try:
                found[i] = calls[i]()
            except Exception as e:  # what a user of the thread would see
                failed.append(f"call {i}: {e!r}")

    threads = [threading.Thread(target=repeat, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for a, b in zip(alone, found):
        np.testing.assert_allclose(b, a, rtol=0.0, atol=2e-4 * np.abs(a).max())
