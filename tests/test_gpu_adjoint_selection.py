"""GPU: the views that the adjoint averages, and their pose gradients.

A hypothesis' views that have a pose gradient are the best_k of the search's own
per-view costs (recon_mvs_evaluate), neither more nor fewer, wherever those
costs say which they are: the two come from different window code (FP32, parity
bar 1e-5 relative + 2e-6), so hypotheses whose k-th and next cost are closer
than ten times that say nothing, nor do those that one of the two rejects.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sources,best_k", [(1, 4), (3, 2), (8, 4), (9, 0), (13, 5), (32, 8)])
def test_exactly_the_best_views_have_a_pose_gradient(sources, best_k):
    import recon_mvs as M
    import synthetic as S

    w, h, n = 96, 72, 300
    sc = S.sphere_on_backdrop(width=w, height=h, f=90.0, num_sources=sources, seed=sources)
    views = M.ViewArgs.from_cameras(sc.ref.image, [s.image for s in sc.sources], sc.ref.camera,
                                    [s.camera for s in sc.sources])
    cfg = M.MvsConfig(min_depth_m=0.2, max_depth_m=0.6, patch_size=7)
    opts = M.Options(mode=M.MODE_PLANE, best_k=best_k, device=0)
    rng = np.random.default_rng(sources)
    # windows well inside the reference image: a window at the edge of validity may differ
    px, py = rng.integers(6, w - 6, n).astype(np.int32), rng.integers(6, h - 6, n).astype(np.int32)
    d = sc.ref.depth[py, px].astype(np.float32).astype(np.float64)
    nrm = sc.ref.normal[py, px]
    ang = np.stack([np.arccos(np.clip(nrm[:, 2], -1, 1)), np.arctan2(nrm[:, 1], nrm[:, 0])], -1)
    ang = ang.astype(np.float32).astype(np.float64)
    eng = M.Engine(opts)
    try:
        cost, grad, H, pg = eng.adjoint(eng.stage(views, cfg), px, py, d, ang, gn=True, pose=True)
    finally:
        eng.close()
    nv = np.stack([np.sin(ang[:, 0]) * np.cos(ang[:, 1]), np.sin(ang[:, 0]) * np.sin(ang[:, 1]), np.cos(ang[:, 0])], -1)
    want, support, vc = M.Evaluate(views, cfg, opts, px, py, 1.0 / d, nv.astype(np.float32), per_view=True)
    has = np.abs(pg).max(-1) > 0
    checked = 0
    for i in range(n):
        valid = vc[i] < 1e29
        k = int(valid.sum())
        if 0 < best_k <= 8:
            k = min(k, best_k)
        order = np.argsort(vc[i], kind="stable")
        s = vc[i][order]
        if want[i] >= 1e29 or cost[i] >= 1e29 or (k < valid.sum() and s[k] - s[k - 1] < 1e-4 * s[k] + 2e-5):
            continue
        checked += 1
        best = np.zeros(sources, bool)
        best[order[:k]] = True
        assert np.array_equal(has[i], best), (i, np.nonzero(has[i])[0], np.nonzero(best)[0], s[:k + 1])
        assert abs(cost[i] - vc[i][best].mean()) <= 1e-5 * abs(cost[i]) + 2e-6
    assert checked > 0.7 * n
