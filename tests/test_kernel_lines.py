"""Where the stage queues take over from the ray loop: residual carry with one
aerosol species from 2 chains per lane on, with four, whose renders of 2 to 5 chains
per lane the queues made up to 16 % slower, from 5."""

import numpy as np
import pytest

from sky_cuda import GpuScene, RenderConfig
from sky_cuda import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tables,per_lane", [("dome", 2), ("ref", 5)])
def test_residual_carry(gpu, dome_scene, ref_scene, tables, per_lane):
    import torch
    scene = dome_scene if tables == "dome" else ref_scene
    lanes = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    cfg = dict(width=64, height=32, phase_sampling=_abi.PHASE_TABULATED, tracking=_abi.TRACKING_RESIDUAL_CARRY, seed=3)
    with GpuScene(scene) as gs:
        spp = gs.queue_spp(RenderConfig(spp=1, **cfg))
        assert spp == -(-per_lane * lanes // (64 * 32 * gs.band_count))
        for n in (spp - 1, spp):  # either side: the plain kernel's sums
            sums = []
            for kernel in (_abi.KERNEL_PLAIN, _abi.KERNEL_WAVEFRONT):
                s = torch.zeros(64 * 32 * gs.band_count, dtype=torch.float64, device="cuda")
                st = torch.zeros(1, dtype=torch.int32, device="cuda")
                gs.render_device(RenderConfig(spp=n, kernel=kernel, **cfg),
                                 {"cell_sum": s.data_ptr(), "status": st.data_ptr()},
                                 torch.cuda.current_stream().cuda_stream)
                assert int(st.item()) == 0
                sums.append(s.cpu().numpy())
            # FP64 sums of the same n radiances in any order
            np.testing.assert_allclose(sums[1], sums[0], rtol=2 * n * 2.0**-52, atol=0)
