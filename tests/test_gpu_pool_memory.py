"""GPU: working memory from the pool, clouds handed over without a copy.

An array of a returned cloud stays valid and its own after the cloud object and
later calls; calls from several threads, each with its own stream, draw on the
same pool; and a call after a much larger one gives the same result.
"""
import gc
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def maps(M, w, h, seed):
    rng = np.random.default_rng(seed)
    d = rng.uniform(0.3, 0.5, (h, w)).astype(np.float32)
    m = M.DepthMap(d, np.full((h, w), 4, np.uint8), rng.uniform(0.2, 1.0, (h, w)).astype(np.float32))
    pose = np.concatenate([np.eye(3).reshape(-1), [0.0, 0.0, 0.0, 0.0]])
    intr = np.array([w, w, w / 2, h / 2, 0, 0, 0, 0, 0, w, h], np.float64)
    return [m], [pose], [intr], M.MvsConfig(fusion_voxel_size_m=0.002)


def test_cloud_arrays_outlive_the_cloud():
    import recon_mvs as M

    a = M.FuseDepthMaps(*maps(M, 64, 48, 1))
    keep, want = a.positions, a.positions.copy()
    keys = a.keys
    del a
    gc.collect()
    b = M.FuseDepthMaps(*maps(M, 640, 480, 2))
    assert b.size() > len(keep)
    assert np.array_equal(keep, want) and len(keys) == len(keep)
    keep[:] = 0.0  # the caller's to write
    c = M.FuseDepthMaps(*maps(M, 64, 48, 1))
    assert np.array_equal(c.positions, want)
    assert M.FuseDepthMaps(*maps(M, 64, 48, 1)[:3], M.MvsConfig(min_view_consistency=99)).size() == 0


def test_threads_share_the_pool():
    import recon_mvs as M

    args = [maps(M, 80 + 16 * i, 60, i) for i in range(4)]
    want = [M.FuseDepthMaps(*a) for a in args]
    bad = []

    def work(i):
        for _ in range(10):
            got = M.FuseDepthMaps(*args[i])
            if not (np.array_equal(got.positions, want[i].positions) and np.array_equal(got.keys, want[i].keys)
                    and np.array_equal(got.confidences, want[i].confidences)):
                bad.append(i)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_the_last_context_gives_the_memory_back():
    """In a process of its own: the contexts of a thread go with it, and with the
    last of them what the pool kept."""
    import subprocess
    import sys

    code = """
import os, sys, threading, time
sys.path[:0] = sys.argv[1:]
import torch
import recon_mvs as M
from test_gpu_pool_memory import maps
torch.zeros(1, device="cuda")
def call():
    m, p, i, cfg = maps(M, 1600, 1200, 1)
    M.FuseDepthMaps(m * 8, p * 8, i * 8, cfg)
    held.append(torch.cuda.mem_get_info()[0])
free, held = [], []
for _ in range(2):
    t = threading.Thread(target=call)
    t.start(); t.join()
    # join() returns before the system's thread and its contexts have ended
    end = time.time() + 20
    while torch.cuda.mem_get_info()[0] - held[-1] <= 8 * 1600 * 1200 * 8 and time.time() < end:
        time.sleep(0.05)
    free.append(torch.cuda.mem_get_info()[0])
print(free[0] - held[0], free[1] - free[0])
"""
    out = subprocess.run([sys.executable, "-c", code] + [p for p in sys.path if p], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    given_back, drift = map(int, out.stdout.split())
    # eight 1600x1200 maps' points, 8 bytes a pixel at the least
    assert given_back > 8 * 1600 * 1200 * 8
    assert abs(drift) < 64 << 20
