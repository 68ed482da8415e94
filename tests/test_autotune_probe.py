"""The autotuner's probe runs the kernel that the render itself runs: the stage
queues where the render has the chains for them, the ray loop below."""

import pytest

from sky_cuda import GpuScene, RenderConfig, SkyCudaError
from sky_cuda import _abi
from sky_cuda import autotune as at

from test_autotune_host import FakeScene, fake_timing  # noqa: F401  (a fixture)


class TwoKernels(FakeScene):
    """A scene whose renders run the stage queues from `line` samples per pixel on."""

    def __init__(self, line):
        super().__init__()
        self.line = line

    def queue_spp(self, config):
        return self.line


@pytest.mark.parametrize("spp,line,probe", [
    (1024, 229, 229),   # the render takes the queues, an eighth of it would not
    (1024, 100, 128),   # an eighth does
    (1024, 1024, 1024),  # the smallest render that takes them is its own probe
    (1024, 1025, 128),  # the render takes the ray loop
    (80, 70, 70), (80, 90, 64), (16, 8, 16), (16, 17, 16),
])
def test_probe_stays_on_the_renders_side(fake_timing, spp, line, probe):  # noqa: F811
    at.autotune(TwoKernels(line), RenderConfig(width=32, height=16, spp=spp), space={"variant": (0, 1)})
    assert [p.spp for p in fake_timing] == [probe, probe]


@pytest.mark.gpu
def test_queue_spp_of_a_scene(gpu, dome_scene, ref_scene):
    import torch
    lanes = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    for scene, per_lane in ((dome_scene, 24), (ref_scene, 34)):
        with GpuScene(scene) as gs:
            cfg = RenderConfig(width=32, height=16, spp=1, tracking=_abi.TRACKING_MERGED_LAYERS)
            assert gs.queue_spp(cfg) == -(-per_lane * lanes // (32 * 16 * gs.band_count))
            gs.set_tuning(all_species=1)
            assert gs.queue_spp(cfg) == -(-34 * lanes // (32 * 16 * gs.band_count))
            cfg = RenderConfig(width=32, height=16, spp=1, tracking=_abi.TRACKING_SEGMENT_RESTART)
            assert gs.queue_spp(cfg) == -(-5 * lanes // (32 * 16 * gs.band_count))
            with pytest.raises(SkyCudaError, match="tracking"):
                gs.queue_spp(RenderConfig(width=32, height=16, spp=1, tracking=3))


@pytest.mark.gpu
def test_autotune_of_a_render_just_above_the_line(gpu, dome_scene):
    with GpuScene(dome_scene) as gs:
        cfg = RenderConfig(width=32, height=16, spp=1, phase_sampling=_abi.PHASE_TABULATED,
                           tracking=_abi.TRACKING_MERGED_LAYERS)
        line = gs.queue_spp(cfg)
        cfg = RenderConfig(**{**cfg.__dict__, "spp": 2 * line})
        assert 64 < line and 2 * line // 8 < line and at._probe_spp(gs, cfg) == line
        best, trials = at.autotune(gs, cfg, space={"variant": (0, 1, 2)})
        ms = {t["variant"]: v for t, v in trials}
        # 8 warps per block take 1.25 times as long as 16 in the queues; in the ray loop, with
        # these tables, the shapes are within a few percent of each other
        assert best["variant"] != 1 and ms[1] > 1.1 * min(ms.values())
