"""A program that resets the device's primary context (its own context, as
cudaDeviceReset does) and starts again in the same process: nothing that belongs
to the old context may be remembered.  In a child process, so that the reset
does not reach the other tests.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import ctypes
from slosh_b200 import scenes
from slosh_b200.pipeline import MpmPipeline

def run(dim):
    sc = scenes.dam_break_2d(h=1 / 64) if dim == 2 else scenes.random_scene_3d(4000, "sand", 1 / 64, seed=1)
    data = scenes.build_mpm_data(sc)
    MpmPipeline().launch_step(data, 5)
    out, kernels = data.download_particles(), data.kernels_per_substep
    data.close()
    return out.tobytes(), kernels

before = [run(2), run(3)]
assert ctypes.CDLL("libcuda.so.1").cuDevicePrimaryCtxReset_v2(0) == 0
after = [run(2), run(3)]
assert before == after and [k for _, k in after] == [1, 1]
print("same bits")
"""


def test_small_scenes_step_after_a_context_reset(cuda_lib):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "same bits" in r.stdout
