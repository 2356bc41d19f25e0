"""GPU: ComputeNcc's two kernels -- a warp per window for few windows, a thread
per window for many -- give the same bits: the sums are the reference's serial
FP64 chains in both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 1 x 1 to several 128-sample chunks per window (even sizes take the next odd window), partial blocks of 4
@pytest.mark.parametrize("patch", [1, 4, 7, 11, 15, 21])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 37])
def test_few_windows_equal_many(patch, n):
    import recon_mvs as M

    rng = np.random.default_rng(patch * 100 + n)
    ref = rng.integers(0, 256, (41, 53)).astype(np.uint8)
    src = rng.integers(0, 256, (37, 60)).astype(np.uint8)
    src[:12, :14] = 90  # a flat corner: weak texture, no NCC
    c = np.stack([rng.uniform(-3, 56, n), rng.uniform(-3, 44, n), rng.uniform(-3, 63, n), rng.uniform(-3, 40, n)], 1)
    c[0] = (20.0, 15.0, 6.0, 5.0)
    few = M.ComputeNccBatch(ref, src, c, patch)
    reps = 152 * 4 * 32 // n + 1  # more windows than warps are taken for
    many = M.ComputeNccBatch(ref, src, np.tile(c, (reps, 1)), patch)
    for i in range(n):
        for j in (i, (reps - 1) * n + i):
            assert (few[i].valid, few[i].ncc, few[i].weak_texture, few[i].valid_samples) == \
                   (many[j].valid, many[j].ncc, many[j].weak_texture, many[j].valid_samples), (i, j)
