"""The stage queues' backstop counts a warp's polls of empty queues in a row, not
over the whole launch: a launch of many minutes whose warps idle now and then
runs on.  Nor does a launch without a limit on its batches end at the 2^32-th."""

import subprocess
import sys

import pytest

from conftest import PKG, ROOT

sys.path.insert(0, str(PKG))
import build as skybuild  # noqa: E402


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    """queue_harness.cu, compiled as the library is."""
    exe = tmp_path_factory.mktemp("queues") / "queue_harness"
    cmd = [skybuild.nvcc(), *skybuild.ARCH, *skybuild.NVCC_FLAGS, "-I", str(skybuild.CSRC),
           str(ROOT / "tests" / "queue_harness.cu"), "-o", str(exe)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return exe


def _run(harness):
    res = subprocess.run([str(harness)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stderr
    return [tuple(map(int, line.split())) for line in res.stdout.splitlines()]


@pytest.mark.gpu
def test_no_limit_on_the_batches(gpu, harness):
    assert _run(harness)[1] == (1, 0, 0)  # the count starts again from 0


@pytest.mark.gpu
def test_a_batch_ends_the_count_of_empty_polls(gpu, harness):
    first, second, status = _run(harness)[0]
    # 200 takes end the one, 199 or 200 the other
    assert status == 0 and max(first, second) == 200 and min(first, second) >= 199
