"""The stage queues' instantiations that renders of test size do not reach: event
counting in every tracking mode and over several jobs, the smaller shapes with
four species and layer-by-layer tracking, tables that leave an SM room for one
block, and a gradient whose forward takes the queues and whose backward the ray
loop.  Cell sums are sums of the plain kernel's radiances (FP64 rounding of n
terms in any order, twice n 2^-52); its event counts are theirs."""

import numpy as np
import pytest

from sky_cuda import GpuScene, RenderConfig, synthetic_scene, wavelengths
from sky_cuda import _abi
from sky_cuda.adjoint import AdjointRenderer
from sky_cuda.scene import SyntheticAtmosphere

from test_adjoint_queues import _backward, _chains, _forward

pytestmark = pytest.mark.gpu

MERGED, CARRY, RESTART = _abi.TRACKING_MERGED_LAYERS, _abi.TRACKING_RESIDUAL_CARRY, _abi.TRACKING_SEGMENT_RESTART


def _outputs(cells, counted):
    import torch
    out = {"cell_sum": torch.zeros(cells, dtype=torch.float64, device="cuda"),
           "status": torch.zeros(1, dtype=torch.int32, device="cuda")}
    if counted:
        out["counters"] = torch.zeros(8, dtype=torch.int64, device="cuda")
    return out


def _render(gs, cfg, counted=False):
    import torch
    out = _outputs(cfg.pixels * gs.band_count, counted)
    gs.render_device(cfg, {k: t.data_ptr() for k, t in out.items()}, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(out["status"].item()) == 0
    return out["cell_sum"].cpu().numpy(), out["counters"].cpu().numpy() if counted else None


def _config(gs, width, height, tracking, phase, **kw):
    cfg = dict(width=width, height=height, tracking=tracking, phase_sampling=phase, **kw)
    return dict(cfg, spp=gs.queue_spp(RenderConfig(spp=1, **cfg)) + 1)


@pytest.mark.parametrize("tracking", [RESTART, CARRY, MERGED])
@pytest.mark.parametrize("tables,lights", [("dome", 1), ("ref", 1)])
def test_event_counts(gpu, dome_scene, ref_scene, tables, lights, tracking):
    with GpuScene(dome_scene if tables == "dome" else ref_scene) as gs:
        cfg = _config(gs, 33, 17, tracking, _abi.PHASE_TABULATED, direct_light_samples=lights, rr_start_depth=3)
        want, events = _render(gs, RenderConfig(kernel=_abi.KERNEL_PLAIN, **cfg), counted=True)
        got, counted = _render(gs, RenderConfig(**cfg), counted=True)
        plain, _ = _render(gs, RenderConfig(**cfg))
        for x in (got, plain):
            np.testing.assert_allclose(x, want, rtol=2 * cfg["spp"] * 2.0**-52, atol=0)
        np.testing.assert_array_equal(counted, events)


def test_event_counts_of_two_jobs(gpu, dome_scene):
    """The counters of a launch are its first job's, over all its jobs."""
    import torch
    with GpuScene(dome_scene) as gs:
        a = RenderConfig(**_config(gs, 20, 10, MERGED, _abi.PHASE_TABULATED, seed=3))
        b = RenderConfig(**{**a.__dict__, "width": 5, "height": 7, "spp": 40, "seed": 4})
        out = [_outputs(c.pixels * gs.band_count, True) for c in (a, b)]
        gs.render_batch([(c, None, {k: t.data_ptr() for k, t in o.items()}) for c, o in zip((a, b), out)],
                        torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        want = [_render(gs, RenderConfig(**{**c.__dict__, "kernel": _abi.KERNEL_PLAIN}), counted=True) for c in (a, b)]
        for o, (sums, _), c in zip(out, want, (a, b)):
            assert int(o["status"].item()) == 0
            np.testing.assert_allclose(o["cell_sum"].cpu().numpy(), sums, rtol=2 * c.spp * 2.0**-52, atol=0)
        np.testing.assert_array_equal(out[0]["counters"].cpu().numpy(), want[0][1] + want[1][1])


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("tracking", [RESTART, CARRY, MERGED])
@pytest.mark.parametrize("phase", [_abi.PHASE_TABULATED, _abi.PHASE_ISOTROPIC])
def test_smaller_shapes_with_four_species(gpu, ref_scene, variant, tracking, phase):
    with GpuScene(ref_scene) as gs:
        gs.set_tuning(variant=variant)
        cfg = _config(gs, 16, 9, tracking, phase, seed=9)
        want, _ = _render(gs, RenderConfig(kernel=_abi.KERNEL_PLAIN, **cfg))
        got, _ = _render(gs, RenderConfig(**cfg))
        np.testing.assert_allclose(got, want, rtol=2 * cfg["spp"] * 2.0**-52, atol=0)


@pytest.fixture(scope="module")
def large_scene(data_dir):
    """256 bands and 1000 layers: 77 KB of staged tables."""
    return synthetic_scene(wavelengths(380.0, 780.0, 256), data_dir, sun_elevation_deg=20.0,
                           atmosphere=SyntheticAtmosphere(layers=1000))


@pytest.mark.parametrize("species", [0, 1])
@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("tracking", [CARRY, MERGED])
def test_tables_that_leave_room_for_one_block(gpu, large_scene, species, variant, tracking):
    with GpuScene(large_scene) as gs:
        gs.set_tuning(variant=variant, all_species=species)
        cfg = _config(gs, 16, 8, tracking, _abi.PHASE_TABULATED, seed=2)
        want, _ = _render(gs, RenderConfig(kernel=_abi.KERNEL_PLAIN, **cfg))
        got, _ = _render(gs, RenderConfig(**cfg))
        np.testing.assert_allclose(got, want, rtol=2 * cfg["spp"] * 2.0**-52, atol=0)


@pytest.mark.parametrize("per_lane", [11, 40])
def test_gradient_from_the_other_kernels_radiances(gpu, data_dir, per_lane):
    """Between 10 and 44 chains per lane the forward's chain radiances come from the queues and
    the replay runs in the ray loop: as the ray loop's own first trace, to the rounding that
    test_adjoint_queues derives."""
    import torch
    scene = synthetic_scene(wavelengths(420.0, 680.0, 6), data_dir, sun_elevation_deg=25.0)
    spp = -(-per_lane * _chains(False) // 10 // (64 * 32 * 6))
    cfg = RenderConfig(width=64, height=32, spp=spp, phase_sampling=_abi.PHASE_TABULATED, tracking=MERGED,
                       rr_start_depth=3, seed=5)
    rng = np.random.default_rng(6)
    with GpuScene(scene) as gs:
        r = AdjointRenderer(gs, cfg)
        assert _chains(False) <= r.chain_count < _chains(True)
        layer = torch.tensor(np.concatenate([rng.uniform(0.8, 1.2, r.param_count - 2), [0.9, 0.7]]).astype(np.float32),
                             device="cuda")
        band = torch.tensor(rng.uniform(0.9, 1.1, (6, 4)).astype(np.float32), device="cuda")
        dloss = torch.tensor(rng.uniform(0.5, 1.5, (32, 64, 6)).astype(np.float32), device="cuda")
        chains = r.new_chain_buffer()
        _forward(r, layer, band, chains, None)
        for x, y in zip(_backward(r, layer, band, dloss, chains, None), _backward(r, layer, band, dloss, None, None)):
            assert np.abs(x - y).max() <= 2e-4 * np.abs(y).max()
