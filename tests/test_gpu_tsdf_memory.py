"""GPU: a closed TSDF volume's memory is the device's again.

In a process of its own, which has no context: 54 M voxels, 650 MB of grid and
chain heads, less than the working-memory pool may keep between calls while
something uses it.
"""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import sys
sys.path[:0] = sys.argv[1:]
import numpy as np, torch
import recon_mvs as M, synthetic as S
torch.zeros(1, device="cuda")
free = lambda: torch.cuda.mem_get_info()[0]
def volume(side):
    cfg, frames = S.tsdf_capture(width=160, height=120, f=150.0, n_frames=1, voxel=0.4 / side, truncation=0.004)
    cfg["bbox_max_z"] = cfg["origin_z"] + 0.2
    vol = M.TsdfVolume(M.TsdfConfig(**cfg))
    vol.IntegrateDepthFrame(*frames[0])
    return vol
volume(20).close()  # the kernels' modules are loaded
before = free()
vol = volume(520)
during, n = free(), int(np.prod(vol.dims()))
vol.close()
print(before, during, free(), n)
"""


def test_a_closed_volume_gives_its_memory_back():
    out = subprocess.run([sys.executable, "-c", CODE] + [p for p in sys.path if p], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    before, during, after, n = map(int, out.stdout.split())
    margin = 64 << 20  # far below the volume's 12 bytes a voxel
    assert n > 50 << 20 and before - during >= 12 * n - margin
    assert abs(after - before) < margin
