"""GPU: ComputeNcc on both sides of the window count from which a thread takes a
window instead of a warp -- the line depends on the window's size -- gives the
same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("patch", [1, 2, 3, 5, 11])
def test_both_sides_of_the_line(patch):
    import recon_mvs as M

    rng = np.random.default_rng(patch)
    ref = rng.integers(0, 256, (41, 53)).astype(np.uint8)
    src = rng.integers(0, 256, (37, 60)).astype(np.uint8)
    k = 17
    c = np.stack([rng.uniform(-3, 56, k), rng.uniform(-3, 44, k), rng.uniform(-3, 63, k), rng.uniform(-3, 40, k)], 1)
    row = lambda r: (r.valid, r.ncc, r.weak_texture, r.valid_samples)
    want = [row(r) for r in M.ComputeNccBatch(ref, src, c, patch)]
    line = 11000 * patch * patch // (patch * patch + 44)
    for n in (line, line + 1):
        got = M.ComputeNccBatch(ref, src, np.tile(c, (n // k + 1, 1))[:n], patch)
        assert all(row(got[i]) == want[i % k] for i in range(n)), n
