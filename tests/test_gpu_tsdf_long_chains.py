"""GPU: long TSDF chains and poses that are not exact rotations, bit for bit.

A voxel's chain of up to 6 records is folded by one thread in registers, a longer
one by a warp that marks its records and reads the box of pixels and steps that
holds them in order.  A grid of one voxel takes every pixel of a frame into one
chain: single rows of a few pixels give chains just below and above the line, a
whole frame the longest there is.  A truncation of fifty voxels over noisy
depths spreads a voxel's records over more steps than a warp has lanes.  A pose
whose rotation was stored in FP32, or is scaled, takes the walk's general
direction.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def compare(cfgd, frames):
    import recon_mvs as M

    want = O.tsdf_fuse(O.tsdf_config(**cfgd), frames)
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
    return want


def config(w, h, voxel, trunc, **kw):
    f = 0.9 * max(w, h)
    c = dict(voxel_size_m=voxel, truncation_m=trunc, min_depth_m=0.05, max_depth_m=2.0, fx=f, fy=f,
             cx=(w - 1) / 2.0, cy=(h - 1) / 2.0, origin_x=-0.3, origin_y=-0.2, origin_z=0.1, bbox_max_x=0.3,
             bbox_max_y=0.2, bbox_max_z=0.8, min_confidence=30)
    c.update(kw)
    return c


def frames_of(w, h, n, sigma, pose=None, seed=0):
    import synthetic as S

    rng = np.random.default_rng(seed)
    out = []
    for i in range(n):
        depth = np.clip(400 + sigma * rng.standard_normal((h, w)), 1, 65535).astype(np.uint16)
        conf = rng.integers(20, 256, (h, w)).astype(np.uint8) if i else None
        m = S.tsdf_pose(0.01 * i, -0.01 * i, 0.0, 0.03 * i)
        out.append((depth, conf, pose(m) if pose else m, 0.003 + 0.001 * i))
    return out


ONE = dict(origin_x=-2.0, origin_y=-2.0, origin_z=-1.6, bbox_max_x=1.0, bbox_max_y=1.0, bbox_max_z=1.0)


@pytest.mark.parametrize("w,h", [(1, 1), (2, 1), (3, 1), (4, 1), (5, 1), (6, 1), (7, 1), (8, 1), (1, 7), (33, 9),
                                 (97, 61), (160, 120)])
def test_a_grid_of_one_voxel(w, h):
    want = compare(config(w, h, 4.0, 0.5, **ONE), frames_of(w, h, 2, 40.0))
    assert want["tsdf"].size == 1 and want["weight"].ravel()[0] > 0


@pytest.mark.parametrize("w,h,voxel,trunc,sigma", [
    (64, 48, 0.01, 0.5, 60.0),     # 103 steps; records of a voxel over many of them
    (65, 33, 0.05, 0.08, 20.0),
    (160, 120, 0.02, 0.16, 5.0),
    (320, 240, 0.01, 0.03, 2.0),
])
def test_long_chains(w, h, voxel, trunc, sigma):
    compare(config(w, h, voxel, trunc), frames_of(w, h, 3, sigma))


@pytest.mark.parametrize("pose", [lambda m: m.astype(np.float32).astype(np.float64),
                                  lambda m: np.vstack([m[:3] * [[1.002] * 3 + [1.0]], m[3:]])])
def test_poses_that_are_not_exact_rotations(pose):
    frames = frames_of(64, 48, 3, 5.0, pose)
    R = frames[2][2][:3, :3]
    assert np.abs(R.T @ R - np.eye(3)).max() > 4e-16
    compare(config(64, 48, 0.01, 0.04), frames)
