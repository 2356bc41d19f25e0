"""GPU: compat windows at the ends of the sizes that are compiled whole.

The sizes from 3x3 (and 2x2, which is the same window) to 17x17 are compiled
whole, 1x1 and 19x19 take the general loop.  recon_mvs_evaluate runs the general
loop for every size, and both forms do the same FP32 arithmetic in the same
order, so a map's initial costs equal it bit for bit: with one seed depth per
32-pixel cell and no iterations they are those of hypotheses known exactly.  A
map that is searched and refined has to end with the costs of its own depths.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def views_of(M, S, w, h, seed):
    sc = S.sphere_on_backdrop(width=w, height=h, f=60.0, num_sources=3, seed=seed)
    cams = [sc.ref.camera] + [s.camera for s in sc.sources]
    imgs = [sc.ref.image] + [s.image for s in sc.sources]
    return M.ViewArgs.from_cameras(imgs[0], imgs[1:], cams[0], cams[1:])


@pytest.mark.parametrize("w,h", [(65, 49), (31, 33), (64, 4), (9, 40)])
@pytest.mark.parametrize("patch", [1, 2, 3, 17, 19])
def test_initial_costs_equal_the_general_path(w, h, patch):
    import recon_mvs as M
    import synthetic as S

    views = views_of(M, S, w, h, w + patch)
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


@pytest.mark.parametrize("patch", [3, 19])
def test_a_searched_map_has_the_costs_of_its_depths(patch):
    import recon_mvs as M
    import synthetic as S

    w, h = 95, 67
    views = views_of(M, S, w, h, patch)
    cfg = M.MvsConfig(min_depth_m=0.2, max_depth_m=0.6, iterations=2, patch_size=patch, subpixel_iterations=3)
    opts = M.Options(mode=M.MODE_COMPAT, device=0)
    got = M.PatchMatchStereo(views, cfg, options=opts)
    y, x = np.nonzero(np.isfinite(got.depth))
    assert len(x) > 0.5 * w * h
    # a map holds FP32 depths: the cost of the rounded depth is the cost within the slope of
    # the window's interpolation over 2^-24 of a depth, far below 1e-3 at these focal lengths
    want, _ = M.Evaluate(views, cfg, opts, x, y, 1.0 / got.depth[y, x].astype(np.float64))
    assert (np.abs(got.cost[y, x] - want) <= 1e-3).mean() >= 0.99


def test_views_of_a_hypothesis_out_of_range_have_no_cost():
    import recon_mvs as M
    import synthetic as S

    views = views_of(M, S, 65, 49, 3)
    cfg = M.MvsConfig(min_depth_m=0.2, max_depth_m=0.6, patch_size=7)
    inv = np.array([1.0 / 0.4, 1.0 / 0.1, 1.0 / 0.7, 0.0, -1.0])
    x, y = np.full(5, 32), np.full(5, 24)
    cost, sup, vc = M.Evaluate(views, cfg, M.Options(mode=M.MODE_COMPAT, device=0), x, y, inv, per_view=True)
    assert (cost[1:] >= 1e29).all() and (sup[1:] == 0).all() and (vc[1:] >= 1e29).all()
    assert sup[0] == (vc[0] < 1e29).sum()
