"""GPU: the compat window kernels against the general compat path.

Whole 11x11 and 7x7 compat windows read each texel once and share its
interpolations between samples; recon_mvs_evaluate keeps the general loop, one
gather per sample.  Both do the same FP32 arithmetic in the same order, so the
bar is bit-identity: with one seed depth per 32-pixel cell and no iterations, a
compat map's costs are those of hypotheses known exactly.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# sizes around the 32 x 4 block (one short, exact, one over), images smaller than a window
@pytest.mark.parametrize("w,h", [(64, 48), (65, 49), (31, 33), (95, 35), (12, 12), (9, 40)])
@pytest.mark.parametrize("patch", [11, 7, 9, 5, 13, 15, 17, 21, 23])
def test_initial_costs_equal_the_general_path(w, h, patch):
    import recon_mvs as M
    import synthetic as S

    sc = S.sphere_on_backdrop(width=w, height=h, f=60.0, num_sources=3, seed=w + patch)
    cams = [sc.ref.camera] + [s.camera for s in sc.sources]
    imgs = [sc.ref.image] + [s.image for s in sc.sources]
    views = M.ViewArgs.from_cameras(imgs[0], imgs[1:], cams[0], cams[1:])
    cfg = M.MvsConfig(min_depth_m=0.2, max_depth_m=0.6, iterations=0, patch_size=patch)
    opts = M.Options(mode=M.MODE_COMPAT, device=0)
    rng = np.random.default_rng(patch)
    gx, gy = (w + 31) // 32, (h + 31) // 32
    depth = rng.uniform(0.21, 0.59, (gy, gx))
    seeds = [(min(32 * i + 1, w - 1), min(32 * j + 1, h - 1), depth[j, i]) for j in range(gy) for i in range(gx)]
    got = M.PatchMatchStereo(views, cfg, seeds, opts)
    y, x = [a.ravel() for a in np.mgrid[0:h, 0:w]]
    want, support = M.Evaluate(views, cfg, opts, x, y, 1.0 / depth[y // 32, x // 32])
    assert np.array_equal(got.cost.ravel(), want)
    ok = np.isfinite(got.depth.ravel())
    assert np.array_equal(got.support_count.ravel()[ok], support[ok])
    if min(w, h) > 2 * patch:
        assert (want < 1e29).mean() > 0.2
