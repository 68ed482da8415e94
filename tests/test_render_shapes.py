"""SkyTuning.variant acts on small renders too: the ray loop has a kernel per shape.
A scene of 1000 layers, whose tables leave an SM room for three blocks, shows it:
two blocks per SM (variant 1) against three (variant 0) take 1.22 times as long."""

import pytest

from sky_cuda import GpuScene, RenderConfig, synthetic_scene, wavelengths
from sky_cuda import _abi
from sky_cuda.autotune import _time_render
from sky_cuda.scene import SyntheticAtmosphere

pytestmark = pytest.mark.gpu


def test_small_renders_run_the_asked_shape(gpu, data_dir):
    scene = synthetic_scene(wavelengths(380.0, 780.0, 41), data_dir, sun_elevation_deg=20.0,
                            atmosphere=SyntheticAtmosphere(layers=1000))
    cfg = RenderConfig(width=64, height=32, spp=24, phase_sampling=_abi.PHASE_TABULATED,
                       tracking=_abi.TRACKING_MERGED_LAYERS, rr_start_depth=8)
    with GpuScene(scene) as gs:
        ms = {}
        for variant in (0, 1):
            gs.set_tuning(variant=variant)
            ms[variant] = _time_render(gs, cfg, 10)
    assert ms[1] > 1.08 * ms[0], ms


def _large(data_dir, bands=256):
    return synthetic_scene(wavelengths(380.0, 780.0, bands), data_dir, sun_elevation_deg=20.0,
                           atmosphere=SyntheticAtmosphere(layers=1000))


@pytest.mark.parametrize("species", [0, 1])
def test_one_block_per_sm_has_the_most_warps(gpu, data_dir, species):
    """Tables that leave the stage queues room for one block per SM: the smaller shapes, which
    then kept half of their warps (1.21 times variant 2's time), run as variant 2."""
    cfg = RenderConfig(width=64, height=32, spp=32, phase_sampling=_abi.PHASE_TABULATED,
                       tracking=_abi.TRACKING_MERGED_LAYERS, rr_start_depth=8)
    with GpuScene(_large(data_dir)) as gs:
        ms = {}
        for variant in (0, 2):
            gs.set_tuning(variant=variant, all_species=species)
            ms[variant] = _time_render(gs, cfg, 5)
    assert ms[0] < 1.08 * ms[2], ms
