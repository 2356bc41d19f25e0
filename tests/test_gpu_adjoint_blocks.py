"""GPU: the adjoint's blocks of 32 hypotheses and its warps over source views.

A hypothesis' results do not depend on its neighbours in a block or on how many
views a warp takes, so a call over n hypotheses equals n calls of one, bit for
bit; its cost is the search's cost of the same plane within the cost parity bar
(1e-5 relative + 2e-6); and exactly the averaged views have a pose gradient.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 32, 33])
@pytest.mark.parametrize("sources,best_k", [(1, 4), (3, 2), (8, 4), (9, 0), (32, 8)])
def test_blocks_and_warps(n, sources, best_k):
    import recon_mvs as M
    import synthetic as S

    sc = S.sphere_on_backdrop(width=96, height=72, f=90.0, num_sources=sources, seed=sources)
    cams = [sc.ref.camera] + [s.camera for s in sc.sources]
    imgs = [sc.ref.image] + [s.image for s in sc.sources]
    views = M.ViewArgs.from_cameras(imgs[0], imgs[1:], cams[0], cams[1:])
    cfg = M.MvsConfig(min_depth_m=0.2, max_depth_m=0.6, patch_size=7)
    opts = M.Options(mode=M.MODE_PLANE, best_k=best_k, device=0)
    rng = np.random.default_rng(n)
    px, py = rng.integers(0, 96, n).astype(np.int32), rng.integers(0, 72, n).astype(np.int32)
    d = sc.ref.depth[py, px].astype(np.float32).astype(np.float64)
    nrm = sc.ref.normal[py, px]
    ang = np.stack([np.arccos(np.clip(nrm[:, 2], -1, 1)), np.arctan2(nrm[:, 1], nrm[:, 0])], -1)
    ang = ang.astype(np.float32).astype(np.float64)
    if n > 2:
        ang[2, 0] = 0.1  # a plane turned away: no hypothesis
    eng = M.Engine(opts)
    try:
        job = eng.stage(views, cfg)
        whole = eng.adjoint(job, px, py, d, ang, gn=True, pose=True)
        each = [eng.adjoint(job, px[i:i + 1], py[i:i + 1], d[i:i + 1], ang[i:i + 1], gn=True, pose=True)
                for i in range(n)]
        plain = eng.adjoint(job, px, py, d, ang)
    finally:
        eng.close()
    for k in range(4):
        assert np.array_equal(whole[k], np.concatenate([e[k] for e in each]))
    assert np.array_equal(whole[0], plain[0]) and np.array_equal(whole[1], plain[1])
    nv = np.stack([np.sin(ang[:, 0]) * np.cos(ang[:, 1]), np.sin(ang[:, 0]) * np.sin(ang[:, 1]), np.cos(ang[:, 0])], -1)
    cost, support, vc = M.Evaluate(views, cfg, opts, px, py, 1.0 / d, nv.astype(np.float32), per_view=True)
    ok = (cost < 1e29) & (whole[0] < 1e29)
    near = np.abs(whole[0] - cost) <= 1e-5 * np.abs(cost) + 2e-6
    assert ((whole[0] < 1e29) == (cost < 1e29)).mean() >= 0.9 and near[ok].mean() >= 0.9
    has = np.abs(whole[3]).max(-1) > 0
    averaged = np.minimum(support, best_k if 0 < best_k <= 8 else sources)
    assert (has.sum(1)[ok] <= averaged[ok]).mean() >= 0.9
    if n > 2:
        assert whole[0][2] >= 1e29 and not whole[1][2].any() and not whole[3][2].any()
