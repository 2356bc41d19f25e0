"""GPU: the TSDF update chains against the oracle, bit for bit.

A voxel's updates of one frame are chained, sorted back into the reference's
order and folded: coarse voxels give chains longer than the buffer the fold
sorts in registers (24), ragged frames end in partial warps, axis-aligned rays
put steps exactly on voxel faces, and cameras inside or beside the grid put
projections on the frame's edges -- the cases in which a cheaper form of the
reference's arithmetic has to give way to it.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,voxel,trunc,yaw", [
    (33, 17, 0.004, 0.012, 0.0),     # a ragged frame, axis-aligned centre ray
    (64, 48, 0.05, 0.08, 0.03),      # long chains
    (160, 120, 0.02, 0.02, -0.4),    # a camera turned half out of the grid
    (1, 1, 0.01, 0.03, 0.0),
    (40, 30, 0.01, 0.0005, 0.1),     # truncation below the voxel size
])
def test_chains_match_the_oracle(w, h, voxel, trunc, yaw):
    import recon_mvs as M
    import synthetic as S

    rng = np.random.default_rng(w)
    f = 0.9 * w
    cfgd = dict(voxel_size_m=voxel, truncation_m=trunc, min_depth_m=0.05, max_depth_m=2.0, fx=f, fy=f, cx=w / 2.0,
                cy=h / 2.0, origin_x=-0.3, origin_y=-0.2, origin_z=0.1, bbox_max_x=0.3, bbox_max_y=0.2,
                bbox_max_z=0.8, min_confidence=30)
    frames = []
    for i in range(3):
        depth = np.clip(400 + 60 * rng.standard_normal((h, w)) * (i > 0), 0, 65535).astype(np.uint16)
        conf = rng.integers(20, 256, (h, w)).astype(np.uint8)
        frames.append((depth, conf, S.tsdf_pose(0.02 * i, -0.01 * i, 0.0, yaw * i), 0.003 + 0.001 * i))
    cfg = O.tsdf_config(**cfgd)
    want = O.tsdf_fuse(cfg, frames)
    vol = M.TsdfVolume(M.TsdfConfig(**cfgd))
    try:
        got = [vol.IntegrateDepthFrame(*fr) for fr in frames]
        t, wt = vol.grid()
        pc = vol.ExtractPoints()
    finally:
        vol.close()
    assert got == want["integrated"]
    np.testing.assert_array_equal(t, want["tsdf"])
    np.testing.assert_array_equal(wt, want["weight"])
    for k, v in (("positions", pc.positions), ("normals", pc.normals), ("confidences", pc.confidences),
                 ("voxel_index", pc.keys)):
        np.testing.assert_array_equal(v, want[k], err_msg=k)
