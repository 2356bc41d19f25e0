"""GPU: plane windows without an unrolled instance, read in groups of 3 or 4.

The sweep reads such windows in groups of 3 samples for 3x3, 5x5 and 9x9 and of
4 for the rest, recon_mvs_evaluate one sample at a time: the same samples in the
same order, so a searched map's costs are those of its hypotheses.  A map holds
depths (1 / inverse depth, two FP32 roundings: 1.2e-7 relative, 1e-5 px of
disparity here); a window's NCC changes by less than 20 per pixel on these
images, hence 1e-3 for all but a few windows of nearly no texture.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(65, 49), (33, 66)])
@pytest.mark.parametrize("patch,interp", [(3, 0), (5, 0), (9, 0), (3, 1), (13, 0)])
def test_a_searched_map_has_the_costs_of_its_planes(w, h, patch, interp):
    import recon_mvs as M
    import synthetic as S

    sc = S.sphere_on_backdrop(width=w, height=h, f=150.0 * w / 160, num_sources=3, seed=w + patch)
    views = M.ViewArgs.from_cameras(sc.ref.image, [s.image for s in sc.sources], sc.ref.camera,
                                    [s.camera for s in sc.sources])
    cfg = M.MvsConfig(min_depth_m=sc.min_depth, max_depth_m=sc.max_depth, iterations=2, patch_size=patch,
                      subpixel_iterations=0)
    opts = M.Options(mode=M.MODE_PLANE, best_k=2, refine=0, interp=interp, device=0)
    got = M.PatchMatchStereo(views, cfg, options=opts)
    y, x = np.nonzero(np.isfinite(got.depth))
    assert len(x) > 0.5 * w * h
    want, sup = M.Evaluate(views, cfg, opts, x, y, 1.0 / got.depth[y, x].astype(np.float64), got.normal[y, x])
    assert (np.abs(got.cost[y, x] - want) <= 1e-3).mean() >= 0.99
    assert (got.support_count[y, x] == sup).mean() >= 0.99
