"""GPU: the fusion's point arithmetic against the oracle, bit for bit.

Divisions that share a divisor share its correctly rounded reciprocal and pinhole
slopes are tabled; results and keys have to be those of the reference's own
divisions -- for voxel sizes whose quotients are huge, ordinary and tiny, depths
over ten orders of magnitude, rotated and axis-aligned cameras, with and without
distortion, and sizes that end in partial blocks.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(33, 9), (64, 48), (1, 1)])
@pytest.mark.parametrize("voxel", [0.001, 0.0073, 1e-9, 1e6])
@pytest.mark.parametrize("k1,tilt", [(0.0, 0.3), (0.0, 0.0), (0.05, 0.3)])
def test_points_match_the_oracle(w, h, voxel, k1, tilt):
    import recon_mvs as M

    rng = np.random.default_rng(int(w + 1000 * k1))
    maps, poses, intr = [], [], []
    for i in range(2):
        depth = (10.0 ** rng.uniform(-5, 5, (h, w))).astype(np.float32)
        depth[rng.random((h, w)) < 0.1] = np.nan
        maps.append((depth, rng.integers(1, 6, (h, w)).astype(np.uint8), rng.uniform(0, 1, (h, w)).astype(np.float32)))
        c, s = np.cos(tilt + 0.1 * i * (tilt > 0)), np.sin(tilt + 0.1 * i * (tilt > 0))
        R = np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]]) @ np.array([[1, 0, 0], [0, c, -s], [0, s, c]])
        poses.append(np.concatenate([R.reshape(-1), [0.01 * i, -0.02, 0.0], [0.0]]))
        intr.append(np.array([1.1 * w, w, w / 2.0, h / 2.0, k1, -0.01 * (k1 > 0), 0, 0, 0, w, h], np.float64))
    want = O.fuse_depth_maps("oracle", maps, poses, intr, O.make_config(fusion_voxel_size_m=voxel))
    pc = M.FuseDepthMaps([M.DepthMap(*m) for m in maps], poses, intr, M.MvsConfig(fusion_voxel_size_m=voxel))
    order = np.lexsort((pc.positions[:, 2], pc.positions[:, 1], pc.positions[:, 0]))
    assert pc.size() == len(want[0])
    for got, ref in zip((pc.positions, pc.normals, pc.confidences), want):
        np.testing.assert_array_equal(got[order], ref)
