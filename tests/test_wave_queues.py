"""The wavefront kernel's path pool and stage queues at their edges: images of
few cells, samples per cell off the warp size, jobs of unequal size in one
launch, every tracking mode, shape and species count.  Renders of few chains
per lane take the ray loop instead, so these have just enough chains to take
the queues.  Both consume each chain's random stream in the plain kernel's
order, so its cell sums and theirs are sums of the same radiances: equal to
the FP64 rounding of summing n terms in any order, at most n 2^-52 relative
on either side for non-negative terms."""

import numpy as np
import pytest

from sky_cuda import FLAG_ACCUMULATE, GpuScene, RenderConfig, RenderWatchdog
from sky_cuda import _abi

pytestmark = pytest.mark.gpu

MERGED, CARRY, RESTART = _abi.TRACKING_MERGED_LAYERS, _abi.TRACKING_RESIDUAL_CARRY, _abi.TRACKING_SEGMENT_RESTART
# chains per lane from which a mode takes the queues
PER_LANE = {MERGED: 34, CARRY: 2, RESTART: 5}


def _samples(cells: int, tracking: int) -> int:
    """Samples per cell that take a render of `cells` to the queues, one more than a multiple of 32."""
    import torch
    lanes = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    return -(-PER_LANE[tracking] * lanes // cells // 32) * 32 + 33


def _buffers(cells):
    import torch
    return [torch.full((cells,), 7.0, dtype=torch.float64, device="cuda") for _ in range(2)]


def _sums(gs, cfg, buffers=None):
    import torch
    s, q = buffers or _buffers(cfg.pixels * gs.band_count)
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    gs.render_device(cfg, {"cell_sum": s.data_ptr(), "cell_sumsq": q.data_ptr(), "status": st.data_ptr()},
                     torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(st.item()) == 0
    return s.cpu().numpy(), q.cpu().numpy()


def _same(a, b, n):
    for x, y in zip(a, b):
        np.testing.assert_allclose(x, y, rtol=2 * n * 2.0**-52, atol=0)


@pytest.mark.parametrize("tracking", [RESTART, CARRY, MERGED])
@pytest.mark.parametrize("width,height,phase", [(1, 1, _abi.PHASE_TABULATED), (13, 5, _abi.PHASE_ISOTROPIC),
                                                (127, 63, _abi.PHASE_TABULATED)])
@pytest.mark.parametrize("tables", ["dome", "ref"])
def test_queues_trace_the_plain_kernels_chains(gpu, dome_scene, ref_scene, tables, width, height, phase, tracking):
    scene = dome_scene if tables == "dome" else ref_scene
    spp = _samples(width * height * scene.band_count, tracking)
    cfg = dict(width=width, height=height, spp=spp, phase_sampling=phase, tracking=tracking, sample_offset=2)
    with GpuScene(scene) as gs:
        want = _sums(gs, RenderConfig(**cfg, kernel=_abi.KERNEL_PLAIN))
        for _ in range(2):  # the order in which warps meet at the queues differs from run to run
            _same(_sums(gs, RenderConfig(**cfg, kernel=_abi.KERNEL_WAVEFRONT)), want, spp)


@pytest.mark.parametrize("variant,blocks", [(0, 0), (1, 0), (2, 1)])
def test_every_shape_and_a_capped_block_count(gpu, dome_scene, variant, blocks):
    spp = _samples(9 * 7 * dome_scene.band_count, MERGED)
    cfg = dict(width=9, height=7, spp=spp, phase_sampling=_abi.PHASE_TABULATED, tracking=MERGED)
    with GpuScene(dome_scene) as gs:
        gs.set_tuning(variant=variant, max_blocks_per_sm=blocks)
        _same(_sums(gs, RenderConfig(**cfg)), _sums(gs, RenderConfig(**cfg, kernel=_abi.KERNEL_PLAIN)), spp)


def test_jobs_of_unequal_size_share_the_queues(gpu, dome_scene):
    """Three jobs whose cells and samples differ, one adding to sums it holds: the chain-to-job lookup."""
    import torch
    stream = torch.cuda.current_stream().cuda_stream
    base = dict(phase_sampling=_abi.PHASE_TABULATED, tracking=MERGED)
    with GpuScene(dome_scene) as gs:
        n = _samples(24 * 12 * gs.band_count, MERGED)
        cfgs = [RenderConfig(width=24, height=12, spp=n, seed=11, **base),
                RenderConfig(width=7, height=3, spp=4 * n + 1, seed=12,
                             output_projection=_abi.PROJECTION_SKY_VIEW_LUT, **base),
                RenderConfig(width=16, height=16, spp=8, sample_offset=8, flags=FLAG_ACCUMULATE, seed=13, **base)]
        first = RenderConfig(width=16, height=16, spp=8, seed=13, **base)
        bufs = [_buffers(c.pixels * gs.band_count) for c in cfgs]
        _sums(gs, first, bufs[2])
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        gs.render_batch([(c, None, {"cell_sum": b[0].data_ptr(), "cell_sumsq": b[1].data_ptr(),
                                    "status": st.data_ptr()}) for c, b in zip(cfgs, bufs)], stream)
        torch.cuda.synchronize()
        assert int(st.item()) == 0
        for c, b in zip(cfgs, bufs):
            want = _buffers(c.pixels * gs.band_count)
            if c.flags:
                _sums(gs, RenderConfig(**{**first.__dict__, "kernel": _abi.KERNEL_PLAIN}), want)
            want = _sums(gs, RenderConfig(**{**c.__dict__, "kernel": _abi.KERNEL_PLAIN}), want)
            _same([x.cpu().numpy() for x in b], want, c.spp + 8)


@pytest.mark.parametrize("large", [0, 20, 39])
def test_many_jobs_smaller_than_a_batch(gpu, dome_scene, large):
    """One job of most chains among 39 of a few each, which a warp's 32 chains span: the lookup
    that starts from the job of the warp's last chains."""
    import torch
    stream = torch.cuda.current_stream().cuda_stream
    base = dict(phase_sampling=_abi.PHASE_TABULATED, tracking=MERGED)
    with GpuScene(dome_scene) as gs:
        cfgs = [RenderConfig(width=1, height=1, spp=1 + i % 3, seed=i, **base) for i in range(40)]
        cfgs[large] = RenderConfig(width=24, height=12, spp=_samples(24 * 12 * gs.band_count, MERGED), seed=5, **base)
        bufs = [_buffers(c.pixels * gs.band_count) for c in cfgs]
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        gs.render_batch([(c, None, {"cell_sum": b[0].data_ptr(), "cell_sumsq": b[1].data_ptr(),
                                    "status": st.data_ptr()}) for c, b in zip(cfgs, bufs)], stream)
        torch.cuda.synchronize()
        assert int(st.item()) == 0
        for c, b in zip(cfgs, bufs):
            _same([x.cpu().numpy() for x in b], _sums(gs, RenderConfig(**{**c.__dict__, "kernel": _abi.KERNEL_PLAIN})),
                  c.spp)


def test_iteration_limit_stops_the_queues(gpu, dome_scene):
    spp = _samples(16 * 8 * dome_scene.band_count, MERGED)
    cfg = RenderConfig(width=16, height=8, spp=spp, phase_sampling=_abi.PHASE_TABULATED, tracking=MERGED)
    with GpuScene(dome_scene) as gs:
        gs.set_tuning(iteration_limit=5)
        with pytest.raises(RenderWatchdog, match="iteration limit"):
            gs.render(cfg)
        gs.set_tuning(iteration_limit=0)
        film, stats = gs.render(cfg)
        assert stats.watchdog == 0 and np.all(np.isfinite(film.values)) and film.values.sum() > 0
