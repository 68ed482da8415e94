"""Rounding of the layer gradients where one launch holds many times the chains
that take it to the stage queues: their FP32 copies in shared memory are moved to
FP64 often enough that the sums are no further from the truth than the ray loop's
(which event counting forces) of the same launch.  The truth is the sum of 1/110
parts of the launch, other samples each, whose FP32 sums hold so many times fewer
terms."""

import numpy as np
import pytest

from sky_cuda import GpuScene, RenderConfig, synthetic_scene, wavelengths
from sky_cuda import _abi
from sky_cuda.adjoint import AdjointRenderer

from test_adjoint_queues import _backward, _chains, _forward

pytestmark = pytest.mark.gpu

WIDTH, HEIGHT, BANDS, PARTS = 64, 32, 6, 110


@pytest.mark.parametrize("layers", [100, 114, 200, 600])
def test_layer_gradients_lose_no_precision(gpu, data_dir, layers):
    import torch
    scene = synthetic_scene(wavelengths(420.0, 680.0, BANDS), data_dir, sun_elevation_deg=25.0).bake_majorants(layers)
    per_part = -(-8 * _chains(True) // (WIDTH * HEIGHT * BANDS * PARTS))
    cfg = dict(width=WIDTH, height=HEIGHT, phase_sampling=_abi.PHASE_TABULATED,
               tracking=_abi.TRACKING_MERGED_LAYERS, rr_start_depth=8, seed=5)
    rng = np.random.default_rng(layers)
    with GpuScene(scene) as gs:
        r = AdjointRenderer(gs, RenderConfig(spp=per_part * PARTS, **cfg))
        layer = torch.tensor(np.concatenate([rng.uniform(0.8, 1.2, r.param_count - 2), [0.9, 0.76]]).astype(np.float32),
                             device="cuda")
        band = torch.tensor(rng.uniform(0.9, 1.1, (BANDS, 4)).astype(np.float32), device="cuda")
        dloss = torch.tensor(rng.uniform(0.5, 1.5, (HEIGHT, WIDTH, BANDS)).astype(np.float32), device="cuda")
        chains = r.new_chain_buffer()
        _forward(r, layer, band, chains, None)
        queues, _ = _backward(r, layer, band, dloss, chains, None)
        loop, _ = _backward(r, layer, band, dloss, chains, torch.zeros(8, dtype=torch.int64, device="cuda"))
        truth = np.zeros(r.param_count)
        part_chains = None
        for i in range(PARTS):
            part = AdjointRenderer(gs, RenderConfig(spp=per_part, sample_offset=i * per_part, **cfg))
            part_chains = part.new_chain_buffer() if part_chains is None else part_chains
            part.forward(layer, band, chains=part_chains)
            truth += part.backward(layer, band, dloss, chains=part_chains)[0].cpu().numpy() / PARTS
    layers_only = slice(0, 3 * layers)
    error = [np.abs(x - truth)[layers_only].max() for x in (queues, loop)]
    print(f"{layers} layers: queues {error[0]:.2e}, ray loop {error[1]:.2e}, largest {np.abs(truth[layers_only]).max():.2e}")
    assert error[0] <= error[1]
