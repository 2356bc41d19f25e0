"""GPU: the plane sweep's schedules over cut windows and ragged sizes.

Windows cut by an image border are read in groups of 4 samples by the
texture-read schedule and one sample at a time by the staged 7x7 schedule; tile
heights and the autotuner's pick change which warps run them.  All do the same
FP32 arithmetic on the same samples in the same order, so the bar is
bit-identity -- over sizes with partial tiles, windows with and without an
unrolled instance, both refinements, and batches whose jobs differ in sources
and iterations.  Small images keep most windows near a border.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene(w, h, n, seed):
    import synthetic as S

    return S.sphere_on_backdrop(width=w, height=h, f=150.0 * w / 160, num_sources=n, seed=seed)


def run(items, **opt):
    import recon_mvs as M

    eng = M.Engine(M.Options(mode=M.MODE_PLANE, device=0, **opt))
    try:
        jobs = []
        for sc, patch, iters in items:
            v = M.ViewArgs.from_cameras(sc.ref.image, [s.image for s in sc.sources], sc.ref.camera,
                                        [s.camera for s in sc.sources])
            jobs.append(eng.stage(v, M.MvsConfig(min_depth_m=sc.min_depth, max_depth_m=sc.max_depth, iterations=iters,
                                                 patch_size=patch, subpixel_iterations=3)))
        eng.run_many(jobs)
        return [eng.download(j) for j in jobs]
    finally:
        eng.close()


def same(a, b):
    for x, y in zip(a, b):
        assert x.filled == y.filled and x.filled > 0
        for k in ("depth", "support_count", "confidence", "normal", "cost"):
            assert np.array_equal(getattr(x, k), getattr(y, k), equal_nan=True), k


@pytest.mark.parametrize("w,h,n", [(160, 120, 4), (65, 49, 2), (97, 33, 3), (33, 66, 5), (128, 96, 9)])
@pytest.mark.parametrize("patch,interp,refine,best_k", [(11, 0, 1, 4), (7, 0, 1, 3), (9, 0, 1, 0), (11, 1, 2, 2)])
def test_schedules_give_the_same_maps(w, h, n, patch, interp, refine, best_k):
    items = [(scene(w, h, n, w + n), patch, 2)]
    opt = dict(interp=interp, refine=refine, best_k=best_k)
    fixed = run(items, tile_rows=4, **opt)
    same(run(items, **opt), fixed)
    if interp == 0 and patch != 9:
        same(run(items, tile_rows=4, window_staging=2, **opt), fixed)


def test_mixed_batch_and_coarse_level():
    items = [(scene(130, 98, 2, 1), 11, 3), (scene(96, 80, 7, 2), 11, 4), (scene(64, 64, 9, 3), 11, 2)]
    same(run(items, best_k=3), run(items, best_k=3, tile_rows=2))
    items = [(scene(200, 150, 5, 4), 7, 4)]
    same(run(items, coarse_iterations=2, exploration_iterations=1),
         run(items, coarse_iterations=2, exploration_iterations=1, tile_rows=8))
