"""The differentiable renderer's stage-queue kernels, which launches of many
chains per lane take, against its ray loop, which event counting forces: the
same chains, so the same sums and chain radiances (up to a last-bit rounding of
one chain in a thousand, 1e-6 of a chain's radiance), and gradients equal to the
order of their FP32 additions.

Tolerances: sums of n radiances whose terms differ by at most 1e-6 relative;
gradients 2e-4 of the largest, the FP32 rounding (6e-8) of sums whose terms
cancel to 1/3000 of their magnitudes.  (The ray loop traces a cell in one warp:
of a single cell's millions of chains it adds all terms into one FP32 sum per
parameter, which then says nothing about the last percent; gradients are
compared where cells keep the chip's blocks busy.)"""

import ctypes

import numpy as np
import pytest

from sky_cuda import GpuScene, RenderConfig, synthetic_scene, wavelengths
from sky_cuda import _abi
from sky_cuda._abi import SkyAdjointGrads, SkyDeviceOutputs, check
from sky_cuda.adjoint import AdjointRenderer

pytestmark = pytest.mark.gpu


def _chains(grad: bool) -> int:
    import torch
    return (44 if grad else 10) * 1024 * torch.cuda.get_device_properties(0).multi_processor_count


def _forward(r, layer, band, chains, counters):
    import torch
    cells = r.pixels * r.bands
    out = {"cell_sum": torch.empty(cells, dtype=torch.float64, device="cuda"),
           "cell_sumsq": torch.empty(cells, dtype=torch.float64, device="cuda")}
    o = SkyDeviceOutputs()
    for k, t in out.items():
        setattr(o, k, t.data_ptr())
    o.status = r._status.data_ptr()
    if counters is not None:
        o.counters = counters.data_ptr()
    p = r._params(layer, band, chains=chains)
    check(r.lib.sky_cuda_adjoint_forward(r.gs.handle, ctypes.byref(r._c_config), ctypes.byref(p), ctypes.byref(o),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), r.lib)
    r.check_status()
    return out


def _backward(r, layer, band, dloss, chains, counters):
    import torch
    lg = torch.zeros(r.param_count, dtype=torch.float64, device="cuda")
    bg = torch.zeros(r.bands * 4, dtype=torch.float64, device="cuda")
    g = SkyAdjointGrads()
    g.dloss_dfilm, g.layer_grad, g.band_grad = dloss.data_ptr(), lg.data_ptr(), bg.data_ptr()
    g.status = r._status.data_ptr()
    if counters is not None:
        g.counters = counters.data_ptr()
    p = r._params(layer, band, chains=chains)
    check(r.lib.sky_cuda_adjoint_backward(r.gs.handle, ctypes.byref(r._c_config), ctypes.byref(p), ctypes.byref(g),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), r.lib)
    r.check_status()
    return lg.cpu().numpy(), bg.cpu().numpy()


@pytest.mark.parametrize("width,height,bands,lights,phase", [(1, 1, 1, 1, _abi.PHASE_TABULATED),
                                                             (37, 19, 3, 2, _abi.PHASE_ISOTROPIC),
                                                             (64, 31, 32, 1, _abi.PHASE_TABULATED)])
def test_queues_match_the_ray_loop(gpu, data_dir, width, height, bands, lights, phase):
    import torch
    scene = synthetic_scene(wavelengths(420.0, 680.0, bands), data_dir, sun_elevation_deg=25.0)
    rng = np.random.default_rng(bands)
    spp = -(-_chains(True) // (width * height * bands)) + 1  # just enough chains for both passes
    cfg = RenderConfig(width=width, height=height, spp=spp, direct_light_samples=lights, phase_sampling=phase,
                       tracking=_abi.TRACKING_MERGED_LAYERS, rr_start_depth=3, seed=5)
    with GpuScene(scene) as gs:
        r = AdjointRenderer(gs, cfg)
        layer = torch.tensor(np.concatenate([rng.uniform(0.8, 1.2, r.param_count - 2), [0.9, 0.7]]).astype(np.float32),
                             device="cuda")
        band = torch.tensor(rng.uniform(0.9, 1.1, (bands, 4)).astype(np.float32), device="cuda")
        dloss = torch.tensor(rng.uniform(0.5, 1.5, (height, width, bands)).astype(np.float32), device="cuda")
        dloss[: height // 4] = 0.0  # rows without a loss
        count = torch.zeros(8, dtype=torch.int64, device="cuda")
        chains, loop_chains = r.new_chain_buffer(), r.new_chain_buffer()
        got, want = _forward(r, layer, band, chains, None), _forward(r, layer, band, loop_chains, count)
        assert int(count[6].item()) == r.chain_count
        a, b = chains.cpu().numpy(), loop_chains.cpu().numpy()
        assert np.mean(a != b) <= 1e-2 and np.all(np.abs(a - b) <= 1e-6 * np.abs(b))
        for k in got:
            np.testing.assert_allclose(got[k].cpu().numpy(), want[k].cpu().numpy(), rtol=4e-6, atol=0)
        if width * height * bands < 2000:
            return
        for buf in (chains, None):  # replay alone, and the gradient kernel's own first trace
            for x, y in zip(_backward(r, layer, band, dloss, buf, None),
                            _backward(r, layer, band, dloss, buf, count)):
                assert np.abs(x - y).max() <= 2e-4 * np.abs(y).max()


def test_a_batch_takes_the_queues(gpu, data_dir):
    """Two suns in one launch against a launch each: films and gradients add up."""
    import torch
    scene = synthetic_scene(wavelengths(420.0, 680.0, 4), data_dir, sun_elevation_deg=25.0)
    spp = -(-_chains(True) // (48 * 24 * 4)) + 1
    cfg = RenderConfig(width=48, height=24, spp=spp, phase_sampling=_abi.PHASE_TABULATED,
                       tracking=_abi.TRACKING_MERGED_LAYERS, seed=8)
    suns = [(0.0, 0.6, 0.8), (0.8, 0.6, 0.0)]
    with GpuScene(scene) as gs:
        r = AdjointRenderer(gs, cfg)
        layer = torch.ones(r.param_count, device="cuda")
        layer[-2], layer[-1] = 0.9, 0.76
        band = torch.ones((4, 4), device="cuda")
        dloss = torch.ones((24, 48, 4), device="cuda")
        films = r.forward_batch(layer, band, suns)
        lg, bg = r.backward_batch(layer, band, [dloss, dloss], suns)
        each = [r.forward(layer, band, sun=s) for s in suns]
        for x, y in zip(films, each):
            np.testing.assert_allclose(x["cell_sum"].cpu().numpy(), y["cell_sum"].cpu().numpy(), rtol=4e-6, atol=0)
        one = [r.backward(layer, band, dloss, sun=s) for s in suns]
        for x, y in ((lg, one[0][0] + one[1][0]), (bg, one[0][1] + one[1][1])):
            assert float((x - y).abs().max()) <= 2e-4 * float(y.abs().max())


@pytest.mark.parametrize("layers", [84, 85, 113, 114])
def test_layer_gradient_copies(gpu, data_dir, layers):
    """Two copies of the layer gradient per warp up to 84 layers, one up to 113, one per block above."""
    import torch
    scene = synthetic_scene(wavelengths(420.0, 680.0, 6), data_dir, sun_elevation_deg=25.0).bake_majorants(layers)
    spp = -(-_chains(True) // (32 * 16 * 6)) + 1
    cfg = RenderConfig(width=32, height=16, spp=spp, phase_sampling=_abi.PHASE_TABULATED,
                       tracking=_abi.TRACKING_MERGED_LAYERS, seed=8)
    with GpuScene(scene) as gs:
        r = AdjointRenderer(gs, cfg)
        assert r.param_count == 3 * layers + 2
        layer = torch.ones(r.param_count, device="cuda")
        layer[-2], layer[-1] = 0.9, 0.76
        band = torch.ones((6, 4), device="cuda")
        dloss = torch.ones((16, 32, 6), device="cuda")
        chains = r.new_chain_buffer()
        _forward(r, layer, band, chains, None)
        count = torch.zeros(8, dtype=torch.int64, device="cuda")
        for x, y in zip(_backward(r, layer, band, dloss, chains, None),
                        _backward(r, layer, band, dloss, chains, count)):
            assert np.abs(x - y).max() <= 2e-4 * np.abs(y).max()
