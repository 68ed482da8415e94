"""Images whose cells overflow 64 bits are refused like others that are too large.
(2^31 x 2^31 pixels of four bands are 2^64 cells, and two of its rows 2^32 pixels:
taken as 0, they would divide the host's set-up of the launch by zero.)"""

import subprocess
import sys

import pytest

from sky_cuda import _abi

from conftest import DATA_DIR, PKG

pytestmark = pytest.mark.gpu

CALL = """
import ctypes, sys
sys.path.insert(0, sys.argv[1])
from sky_cuda import GpuScene, RenderConfig, synthetic_scene, wavelengths
width, height, row_count = map(int, sys.argv[3:])
gs = GpuScene(synthetic_scene(wavelengths(400.0, 700.0, 4), sys.argv[2], sun_elevation_deg=10.0))
c = RenderConfig(width=width, height=height, spp=1).to_c()
c.row_count = row_count
print(gs.lib.sky_cuda_render(gs.handle, ctypes.byref(c), (ctypes.c_float * 4)(), 4, None))
"""


@pytest.mark.parametrize("width,height,row_count", [(2**31, 2**31, 0), (2**31, 2**31, 2), (2**32 - 1, 2**32 - 1, 0),
                                                    (2**16, 2**14, 0), (2**15 + 1, 2**15, 0)])
def test_too_large(gpu, width, height, row_count):
    res = subprocess.run([sys.executable, "-c", CALL, str(PKG), str(DATA_DIR), str(width), str(height), str(row_count)],
                         capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, (res.returncode, res.stderr)
    assert int(res.stdout) == _abi.SKY_ERR_INVALID_CONFIG
