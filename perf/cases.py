"""The work that users of this engine have it do, as timed cases.

Every case goes through the Python face of the C ABI (recon_mvs.py), from what
a program has in hand (host images and maps, or jobs staged on the device) to
what it gets back (whole maps, clouds, gradients).  The scenes are the
package's own seeded synthetic ones, at the sizes of its tests and benchmark;
`draw` spreads the same kinds of call over their ranges.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "recon-scanner_gb300"))

import recon_mvs as M  # noqa: E402
import synthetic as S  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"

# MvsConfig / Options fields a map case may set
CFG_KEYS = ("patch_size", "iterations", "subpixel_iterations", "num_views", "num_threads", "fusion_voxel_size_m")
OPT_KEYS = ("mode", "storage", "best_k", "refine", "sampling", "prefilter", "interp", "coarse_iterations",
            "exploration_iterations")

PLANE_DEFAULT = dict(mode=M.MODE_PLANE, storage=M.STORAGE_FP32, best_k=4, refine=1, interp=0)
# the form the package's benchmark measures as its chosen one
PLANE_CHOSEN = dict(mode=M.MODE_PLANE, storage=M.STORAGE_FP16, best_k=4, refine=2, interp=1, coarse_iterations=2,
                    exploration_iterations=3)
COMPAT = dict(mode=M.MODE_COMPAT, storage=M.STORAGE_FP32, best_k=4, refine=1, interp=0)


def listed():
    return [
        # ComputeNcc on a few dozen window pairs: a program that scores single
        # matches, where a call's latency is all there is
        dict(name="ncc_64", kind="ncc", w=640, h=480, n=64, patch_size=11),
        # one small map through the stateless PatchMatchStereo with default
        # options: the size of the reference's own unit test
        dict(name="map_160", kind="map", w=160, h=120, sources=4, patch_size=11, iterations=4, subpixel_iterations=4,
             **PLANE_DEFAULT),
        # one VGA map, host images to host map, default options (exact FP32
        # reads, golden-section refinement): the ordinary call
        dict(name="map_640", kind="map", w=640, h=480, sources=4, patch_size=11, iterations=6, subpixel_iterations=4,
             **PLANE_DEFAULT),
        # full-resolution maps of a staged capture, in the form the benchmark
        # measures (FP16 textures, texture-unit interpolation, Gauss-Newton,
        # coarse-to-fine): the largest
        dict(name="capture_1920", kind="jobs", scene="tabletop", w=1920, h=1440, refs=2, sources=8, patch_size=11,
             iterations=8, subpixel_iterations=4, **PLANE_CHOSEN),
        # a batch of staged jobs of mixed sizes and 6-10 sources, default
        # options: the batched engine on an orbit capture
        dict(name="orbit_mixed", kind="orbit", w=960, h=720, refs=4, patch_size=11, iterations=4,
             subpixel_iterations=4, **PLANE_DEFAULT),
        # the whole MVS stage over a small capture, from host images to a fused
        # cloud, with the parameter registry's standard values (7x7 windows,
        # 3 iterations, 5 views)
        dict(name="stage_640", kind="stage", w=640, h=480, sources=8, consistency=2, **PLANE_DEFAULT),
        # the reference's own search on the device (compat mode)
        dict(name="compat_640", kind="map", w=640, h=480, sources=4, patch_size=11, iterations=2,
             subpixel_iterations=4, num_threads=8, **COMPAT),
        # RefineSubpixel on a map that another program made
        dict(name="refine_640", kind="refine", w=640, h=480, sources=4, patch_size=11, subpixel_iterations=4,
             **COMPAT),
        # cost, gradient, Gauss-Newton matrix and pose gradients of 10^4
        # hypotheses: one step of a program that optimises depths and poses
        dict(name="adjoint_10k", kind="adjoint", w=1280, h=960, sources=8, n=10000, patch_size=11, **PLANE_DEFAULT),
        # FuseDepthMaps of host maps behind keep masks into a 1 mm cloud
        dict(name="fuse_1280", kind="fuse", w=1280, h=960, maps=4, fusion_voxel_size_m=0.001),
        # the geometric consistency of one host map against the others
        dict(name="consistency_1280", kind="consistency", w=1280, h=960, maps=6),
        # a depth camera's scan: 8 frames into a 1 mm grid (31 M voxels), then
        # the surface points
        dict(name="tsdf_640", kind="tsdf", w=640, h=480, frames=8, voxel=0.001),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A width over [lo, hi] (logarithmic), odd ones among them, and a height of
    about 3/4 of it."""
    w = _log_int(rng, lo, hi)
    return w, max(lo * 3 // 4, int(w * rng.uniform(0.7, 0.8)))


def draw(rng):
    kind = rng.choice(["ncc", "map", "map", "map", "jobs", "jobs", "orbit", "stage", "compat", "refine", "adjoint",
                       "fuse", "consistency", "tsdf"])
    if kind == "ncc":
        w, h = _size(rng, 160, 1920)
        return dict(kind="ncc", w=w, h=h, n=_log_int(rng, 1, 2000), patch_size=rng.choice([3, 5, 7, 9, 11, 15]))
    if kind in ("map", "jobs"):
        interp = rng.choice([0, 0, 1])
        storage = rng.choice([M.STORAGE_FP32, M.STORAGE_FP16, M.STORAGE_U8] + ([] if interp else [M.STORAGE_BF16]))
        w, h = _size(rng, 150, 1000)
        iters = rng.randint(2, 6)
        c = dict(kind=kind, w=w, h=h, sources=rng.randint(2, 10), patch_size=rng.choice([5, 7, 7, 9, 11, 11, 11]),
                 iterations=iters, subpixel_iterations=rng.randint(2, 5), mode=M.MODE_PLANE, storage=storage,
                 best_k=rng.choice([0, 2, 3, 4, 4, 5]), refine=rng.choice([0, 1, 1, 2]), interp=interp,
                 sampling=rng.choice([0, 0, 0, 1]), coarse_iterations=rng.choice([0, 0, min(2, iters - 1)]),
                 exploration_iterations=rng.choice([0, 0, 2, 3]))
        if kind == "jobs":
            c.update(scene=rng.choice(["sphere", "tabletop"]), refs=rng.randint(1, 3))
            if c["scene"] == "sphere":
                c["refs"] = 1
        return c
    if kind == "orbit":
        return dict(kind="orbit", w=_log_int(rng, 320, 960), h=0, refs=rng.randint(2, 5),
                    patch_size=rng.choice([7, 11]), iterations=rng.randint(2, 4), subpixel_iterations=4,
                    **PLANE_DEFAULT)
    if kind == "stage":
        w, h = _size(rng, 240, 900)
        return dict(kind="stage", w=w, h=h, sources=rng.randint(3, 8), consistency=rng.choice([0, 1, 2]),
                    **rng.choice([PLANE_DEFAULT, PLANE_CHOSEN]))
    if kind == "compat":
        w, h = _size(rng, 120, 720)
        return dict(kind="map", w=w, h=h, sources=rng.randint(2, 6), patch_size=rng.choice([5, 7, 9, 11]),
                    iterations=rng.randint(1, 3), subpixel_iterations=4, num_threads=rng.randint(1, 8), **COMPAT)
    if kind == "refine":
        w, h = _size(rng, 120, 1000)
        return dict(kind="refine", w=w, h=h, sources=rng.randint(2, 6), patch_size=rng.choice([5, 7, 9, 11]),
                    subpixel_iterations=rng.randint(2, 6), **COMPAT)
    if kind == "adjoint":
        w, h = _size(rng, 320, 1280)
        return dict(kind="adjoint", w=w, h=h, sources=rng.randint(2, 10), n=_log_int(rng, 50, 20000),
                    patch_size=rng.choice([5, 7, 11]), **PLANE_DEFAULT)
    if kind in ("fuse", "consistency"):
        w, h = _size(rng, 160, 1280)
        c = dict(kind=kind, w=w, h=h, maps=rng.randint(2, 6))
        if kind == "fuse":
            c["fusion_voxel_size_m"] = rng.choice([0.0005, 0.001, 0.002, 0.005])
        return c
    w, h = _size(rng, 160, 640)
    return dict(kind="tsdf", w=w, h=h, frames=rng.randint(1, 8), voxel=rng.choice([0.001, 0.002, 0.004]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _config(case, sc=None):
    kw = {k: case[k] for k in CFG_KEYS if k in case}
    if sc is not None:
        kw.update(min_depth_m=sc.min_depth, max_depth_m=sc.max_depth)
    return M.MvsConfig(**kw)


def _options(case):
    return M.Options(**{k: case[k] for k in OPT_KEYS if k in case}, device=0)


def _sphere(case, seed):
    return S.sphere_on_backdrop(width=case["w"], height=case["h"], f=600.0 * case["w"] / 640,
                                num_sources=case["sources"], seed=seed, device=DEV)


def _tabletop(case, seed, n, distorted=True):
    k = dict(k1=0.05, k2=-0.01) if distorted else dict(k1=0.0, k2=0.0)
    return S.tabletop(width=case["w"], height=case["h"], f=1450.0 * case["w"] / 1920, num_sources=n, seed=seed,
                      device=DEV, **k)


def _views(sc):
    return M.ViewArgs.from_cameras(sc.ref.image, [s.image for s in sc.sources], sc.ref.camera,
                                   [s.camera for s in sc.sources])


def _maps(case, seed):
    """Depth maps of a capture as a program holds them: the surface with depth
    noise, outliers, holes and badly supported pixels.  When the cloud's size
    has to be the same for every seed (`fixed`), the depths and what is dropped
    are, and the supports and confidences are the seed's."""
    fixed = case["kind"] == "fuse"
    sc = _tabletop(case, 2 if fixed else seed, case["maps"] - 1, distorted=False)
    rng = np.random.default_rng(seed)
    geo = np.random.default_rng(2) if fixed else rng
    maps, keep = [], []
    for v in sc.views:
        h, w = v.depth.shape
        d = v.depth * (1.0 + geo.normal(0.0, 5e-4, v.depth.shape))
        out = geo.random(d.shape) < 0.02
        d[out] *= geo.uniform(0.8, 1.2, int(out.sum()))
        d[geo.random(d.shape) < 0.03] = np.nan
        sup = rng.integers(2, 9, (h, w)).astype(np.uint8)
        sup[geo.random(d.shape) < 0.1] = 1
        maps.append(M.DepthMap(d.astype(np.float32), sup, rng.uniform(0.2, 1.0, (h, w)).astype(np.float32)))
        keep.append((geo.random(d.shape) < 0.9).astype(np.uint8))
    cams = sc.cameras
    return maps, [c.pose_array() for c in cams], [c.intrinsics_array() for c in cams], keep


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "ncc":
        rng = np.random.default_rng(seed)
        w, h = case["w"], case["h"]
        yy, xx = np.mgrid[0:h, 0:w]
        base = 128 + 60 * np.sin(xx * 0.13 + rng.uniform(0, 6)) * np.cos(yy * 0.11) + rng.normal(0, 12, (h, w))
        st["ref"] = np.clip(base, 0, 255).astype(np.uint8)
        st["src"] = np.clip(np.roll(base, 3, 1) + rng.normal(0, 6, (h, w)), 0, 255).astype(np.uint8)
        c = np.stack([rng.uniform(-2, w + 2, case["n"]), rng.uniform(-2, h + 2, case["n"])], -1)
        st["coords"] = np.concatenate([c, c + [3.0, 0.0] + rng.uniform(-0.7, 0.7, c.shape)], 1)
    elif kind == "map":
        sc = _sphere(case, seed)
        st.update(views=_views(sc), cfg=_config(case, sc), opts=_options(case))
    elif kind == "jobs":
        if case["scene"] == "sphere":
            scenes = [_sphere(case, seed)]
        else:
            cap = _tabletop(case, seed, case["sources"])
            scenes = [S.as_reference(cap, k) for k in range(min(case["refs"], len(cap.views)))]
        eng = M.Engine(_options(case))
        cams = scenes[0].cameras
        imgs = [eng.stage_image(v.image, v.camera.intrinsics_array(), undistort=True) for v in scenes[0].views]
        poses = [c.pose_array() for c in cams]
        cfg = _config(case, scenes[0])
        st["eng"] = eng
        st["jobs"] = []
        for k in range(len(scenes)):
            others = [i for i in range(len(imgs)) if i != k]
            st["jobs"].append(eng.stage_images(imgs[k], [imgs[i] for i in others], poses[k],
                                               [poses[i] for i in others], cfg))
    elif kind == "orbit":
        w = case["w"]
        res = tuple((max(160, w * s // 6 + 1 - s % 2), max(120, w * s // 8)) for s in (2, 4, 6))
        # one rig (sizes, source counts) for every seed; each frame's pixel noise from the seed
        scenes = S.orbit_capture(n_frames=60, n_refs=case["refs"], seed=3, device=DEV, resolutions=res,
                                 noise_sigma=0.0)
        rng, noisy = np.random.default_rng(seed), set()
        for v in (v for sc in scenes for v in sc.views if id(v) not in noisy):
            noisy.add(id(v))
            v.image = np.clip(np.round(v.image + rng.normal(0.0, 1.0, v.image.shape)), 0, 255).astype(np.uint8)
        eng = M.Engine(_options(case))
        st["eng"] = eng
        st["jobs"] = [eng.stage(_views(sc), _config(case, sc)) for sc in scenes]
    elif kind == "stage":
        sc = _tabletop(case, seed, case["sources"])
        cfg = M.MvsConfig()
        cfg.apply_preset(1)
        cfg.min_depth_m, cfg.max_depth_m = sc.min_depth, sc.max_depth
        if case.get("coarse_iterations"):
            cfg.patch_size, cfg.iterations = 11, 6
        st.update(eng=M.Engine(_options(case)), cfg=cfg, images=[v.image for v in sc.views],
                  poses=[c.pose_array() for c in sc.cameras], intr=[c.intrinsics_array() for c in sc.cameras],
                  cloud=_cloud_buffers((case["sources"] + 1) * case["w"] * case["h"]))
    elif kind == "refine":
        sc = _sphere(case, seed)
        rng = np.random.default_rng(seed)
        d = (sc.ref.depth * (1.0 + rng.normal(0.0, 2e-3, sc.ref.depth.shape))).astype(np.float32)
        d[rng.random(d.shape) < 0.05] = np.nan
        st.update(views=_views(sc), cfg=_config(case, sc), opts=_options(case), depth=d)
    elif kind == "adjoint":
        sc = _tabletop(case, seed, case["sources"], distorted=False)
        rng = np.random.default_rng(seed)
        ys, xs = np.nonzero(np.isfinite(sc.ref.depth))
        pick = rng.choice(len(xs), case["n"])
        px, py = xs[pick].astype(np.int32), ys[pick].astype(np.int32)
        nrm = sc.ref.normal[py, px]
        depth = sc.ref.depth[py, px] * (1.0 + rng.uniform(-0.005, 0.005, len(px)))
        ang = np.stack([np.arccos(np.clip(nrm[:, 2], -1, 1)), np.arctan2(nrm[:, 1], nrm[:, 0])], -1)
        ang = ang + rng.uniform(-0.05, 0.05, ang.shape)
        # a program's depths and angles are FP32 maps
        depth, ang = depth.astype(np.float32).astype(np.float64), ang.astype(np.float32).astype(np.float64)
        eng = M.Engine(_options(case))
        st.update(eng=eng, job=eng.stage(_views(sc), _config(case, sc)), hyps=(px, py, depth, ang), scene=sc)
    elif kind in ("fuse", "consistency"):
        maps, poses, intr, keep = _maps(case, seed)
        st.update(maps=maps, poses=poses, intr=intr, keep=keep)
        if kind == "fuse":
            st["cfg"] = _config(case)
    else:
        cfg, frames = S.tsdf_capture(width=case["w"], height=case["h"], f=600.0 * case["w"] / 640,
                                     n_frames=case["frames"], seed=seed, voxel=case["voxel"],
                                     truncation=8 * case["voxel"])
        st.update(cfg=M.TsdfConfig(**cfg), frames=frames, cloud=_cloud_buffers(8 * case["w"] * case["h"]))
    return st


def _cloud_buffers(cap):
    """A program's own buffers for clouds of up to `cap` points."""
    return {"positions": np.zeros((cap, 3)), "normals": np.zeros((cap, 3)), "confidences": np.zeros(cap, np.float32),
            "keys": np.zeros(cap, np.int64), "counts": np.zeros(cap, np.int64), "points": 0}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _map_out(dm):
    out = {"depth": dm.depth, "support": dm.support_count, "confidence": dm.confidence, "cost": dm.cost,
           "filled": int(dm.filled)}
    if dm.normal is not None:
        out["normal"] = dm.normal
    return out


def _cloud_out(pc):
    return {"positions": pc.positions, "normals": pc.normals, "confidences": pc.confidences, "keys": pc.keys,
            "counts": pc.counts.astype(np.int64)}


def _cloud_into(buf, pc):
    """The cloud in the program's own buffers (their size does not depend on the
    number of points; what an earlier, larger cloud left is cleared)."""
    n, old = pc.size(), buf["points"]
    for k in ("positions", "normals", "confidences", "keys", "counts"):
        buf[k][:n] = getattr(pc, k)
        buf[k][n:old] = 0
    buf["points"] = n
    return dict(buf)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "ncc":
        r = M.ComputeNccBatch(st["ref"], st["src"], st["coords"], case["patch_size"])
        return {"valid": np.array([x.valid for x in r]), "ncc": np.array([x.ncc for x in r]),
                "weak": np.array([x.weak_texture for x in r]), "samples": np.array([x.valid_samples for x in r])}
    if kind == "map":
        return _map_out(M.PatchMatchStereo(st["views"], st["cfg"], options=st["opts"]))
    if kind in ("jobs", "orbit"):
        eng, jobs = st["eng"], st["jobs"]
        eng.run_many(jobs)
        return [_map_out(eng.download(j)) for j in jobs]
    if kind == "stage":
        pc, n = st["eng"].stage_run(st["images"], st["poses"], st["intr"], st["cfg"], undistort=True,
                                    consistency_views=case["consistency"])
        return dict(_cloud_into(st["cloud"], pc), maps=n)
    if kind == "refine":
        h, w = st["depth"].shape
        dm = M.DepthMap(st["depth"].copy(), np.zeros((h, w), np.uint8), np.zeros((h, w), np.float32))
        n = M.RefineSubpixel(st["views"], st["cfg"], dm, st["opts"])
        return {"depth": dm.depth, "confidence": dm.confidence, "refined": n}
    if kind == "adjoint":
        cost, grad, gn, pose = st["eng"].adjoint(st["job"], *st["hyps"], gn=True, pose=True)
        return {"cost": cost, "grad": grad, "gn": gn, "pose": pose}
    if kind == "fuse":
        return _cloud_out(M.FuseDepthMaps(st["maps"], st["poses"], st["intr"], st["cfg"], st["keep"]))
    if kind == "consistency":
        cnt, keep = M.GeometricConsistency(st["maps"], st["poses"], st["intr"], 0, 0.01, 1.0, 2)
        return {"count": cnt, "keep": keep}
    vol = M.TsdfVolume(st["cfg"])
    n = [vol.IntegrateDepthFrame(*f) for f in st["frames"]]
    pc = vol.ExtractPoints()
    vol.close()
    return dict(_cloud_into(st["cloud"], pc), integrated=np.array(n))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Bytes: each input read once, each output written once.  Flops: the
    window samples of the hypotheses that the search has to weigh (26 per
    sample: projection, interpolation, moments), over the views that are
    averaged; propagation from 8 regions and 5 perturbations a pixel and
    iteration."""
    kind = case["kind"]
    px = case["w"] * case["h"]
    out = 25.0  # depth, support, confidence, normal, cost
    if kind == "ncc":
        k2 = case["patch_size"] ** 2
        return {"bytes": 2.0 * px + 56.0 * case["n"], "flops": 30.0 * k2 * case["n"]}
    if kind in ("map", "jobs", "orbit", "stage"):
        k2 = case.get("patch_size", 7) ** 2
        ns = case.get("sources", 8)
        views = min(case["best_k"] or ns, ns)
        nmaps = case.get("refs", 1)
        if kind == "orbit":
            px = sum((case["w"] * s // 6) * (case["w"] * s // 8) for s in (2, 4, 6)) / 3
        if kind == "stage":
            nmaps, views = ns + 1, min(views, 5)
        if case["mode"] == M.MODE_COMPAT:
            hyps = 1 + case["iterations"] * 4 * 9
            return {"bytes": px * (1.0 + ns + 13.0), "flops": px * hyps * ns * 11.0 * k2}
        hyps = 1 + case.get("iterations", 3) * 13 + 2 + case.get("subpixel_iterations", 3)
        return {"bytes": nmaps * px * (out + 1.0) + ns * px, "flops": nmaps * px * hyps * views * 26.0 * k2}
    if kind == "refine":
        hyps = 5 + 1 + 2 + case["subpixel_iterations"] + 2
        return {"bytes": px * (1.0 + case["sources"] + 12.0),
                "flops": px * hyps * case["sources"] * 11.0 * case["patch_size"] ** 2}
    if kind == "adjoint":
        per = case["sources"] * case["patch_size"] ** 2 * 26.0 + 4 * case["patch_size"] ** 2 * 130.0
        return {"bytes": case["n"] * (24.0 + 8.0 + 40.0 + 24.0 * case["sources"]) + px * (1.0 + case["sources"]),
                "flops": case["n"] * per}
    if kind == "fuse":
        return {"bytes": case["maps"] * px * (10.0 + 30.0), "flops": case["maps"] * px * 60.0}
    if kind == "consistency":
        return {"bytes": px * (4.0 * case["maps"] + 2.0), "flops": px * (case["maps"] - 1) * 60.0}
    grid = (0.40 / case["voxel"]) * (0.32 / case["voxel"]) * (0.24 / case["voxel"])
    return {"bytes": 16.0 * grid + case["frames"] * px * (3.0 + 19 * 8.0), "flops": case["frames"] * px * 19 * 40.0}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _exact_ncc(case, st):
    ref = torch.as_tensor(st["ref"], dtype=torch.float64, device=DEV)
    src = torch.as_tensor(st["src"], dtype=torch.float64, device=DEV)
    c = torch.as_tensor(st["coords"], dtype=torch.float64, device=DEV)
    half = case["patch_size"] // 2
    o = torch.arange(-half, half + 1, device=DEV, dtype=torch.float64)
    dy, dx = [t.reshape(1, -1) for t in torch.meshgrid(o, o, indexing="ij")]

    def sample(img, u, v):
        h, w = img.shape
        ok = (u >= 0) & (v >= 0) & (u <= w - 1) & (v <= h - 1)
        x0 = torch.clamp(u.floor().long(), 0, w - 1)
        y0 = torch.clamp(v.floor().long(), 0, h - 1)
        x1, y1 = torch.clamp(x0 + 1, max=w - 1), torch.clamp(y0 + 1, max=h - 1)
        fx, fy = u - x0, v - y0
        top = img[y0, x0] * (1 - fx) + img[y0, x1] * fx
        bot = img[y1, x0] * (1 - fx) + img[y1, x1] * fx
        return top * (1 - fy) + bot * fy, ok

    a, oka = sample(ref, c[:, 0:1] + dx, c[:, 1:2] + dy)
    b, okb = sample(src, c[:, 2:3] + dx, c[:, 3:4] + dy)
    m = (oka & okb).double()
    n = m.sum(1)
    nn = n.clamp(min=1)
    ma, mb = (a * m).sum(1) / nn, (b * m).sum(1) / nn
    da, db = (a - ma[:, None]) * m, (b - mb[:, None]) * m
    den = torch.sqrt((da * da).sum(1) * (db * db).sum(1)) / nn
    ncc = torch.where((n >= case["patch_size"] ** 2 // 2) & (den >= 1e-9),
                      ((da * db).sum(1) / nn / den.clamp(min=1e-30)).clamp(-1, 1), torch.zeros_like(den))
    return {"valid": None, "ncc": ncc.cpu().numpy(), "weak": None, "samples": None}


def _exact_adjoint(case, st):
    """Cost, gradient and Gauss-Newton matrix of the mean of the best_k view
    costs 1 - NCC, from the per-sample derivatives, in FP64."""
    f8 = dict(dtype=torch.float64, device=DEV)
    sc = st["scene"]
    px, py, depth, ang = [torch.as_tensor(v, device=DEV) for v in st["hyps"]]
    px, py, d = px.double(), py.double(), depth.double()
    t, p = ang[:, 0], ang[:, 1]
    n = torch.stack([t.sin() * p.cos(), t.sin() * p.sin(), t.cos()], -1)
    nt = torch.stack([t.cos() * p.cos(), t.cos() * p.sin(), -t.sin()], -1)
    npp = torch.stack([-t.sin() * p.sin(), t.sin() * p.cos(), torch.zeros_like(t)], -1)
    cam = sc.ref.camera
    half = case["patch_size"] // 2
    o = torch.arange(-half, half + 1, **f8)
    dy, dx = [v.reshape(1, -1) for v in torch.meshgrid(o, o, indexing="ij")]
    N, K2 = len(px), dx.numel()
    ray = lambda x, y: torch.stack([(x + 0.5 - cam.cx) / cam.fx, (y + 0.5 - cam.cy) / cam.fy,  # noqa: E731
                                    torch.ones_like(x)], -1)
    qc = ray(px, py)
    q = ray((px[:, None] + dx), (py[:, None] + dy))
    kappa = (n * qc).sum(-1)
    m = (n[:, None] * q).sum(-1)
    X = q * (d * kappa)[:, None, None] / m[..., None]
    # dX/dn_i = q d (qc_i m - kappa q_i) / m^2
    dXn = q[..., :, None] * (d[:, None, None] * (qc[:, None] * m[..., None] - kappa[:, None, None] * q)
                             / (m * m)[..., None])[..., None, :]
    dX = torch.stack([X / d[:, None, None], (dXn * nt[:, None, None]).sum(-1), (dXn * npp[:, None, None]).sum(-1)], -1)
    ref = torch.as_tensor(sc.ref.image, **f8)
    rx, ry = (px[:, None] + dx).long(), (py[:, None] + dy).long()
    H0, W0 = ref.shape
    rok = (rx >= 0) & (ry >= 0) & (rx < W0) & (ry < H0) & (m < 0)
    r = ref[ry.clamp(0, H0 - 1), rx.clamp(0, W0 - 1)]
    R0, t0 = torch.as_tensor(cam.R, **f8), torch.as_tensor(cam.t, **f8)
    costs, grads, gns, poses = [], [], [], []
    for s in sc.sources:
        c = s.camera
        A = torch.as_tensor(c.R, **f8) @ R0.T
        b = torch.as_tensor(c.t, **f8) - A @ t0
        Y = X @ A.T + b
        z = Y[..., 2]
        u, v = c.fx * Y[..., 0] / z + c.cx - 0.5, c.fy * Y[..., 1] / z + c.cy - 0.5
        img = torch.as_tensor(s.image, **f8)
        h, w = img.shape
        ok = rok & (z > 1e-9) & (u >= 0) & (v >= 0) & (u <= w - 1) & (v <= h - 1)
        x0, y0 = u.floor().long().clamp(0, w - 1), v.floor().long().clamp(0, h - 1)
        x1, y1 = (x0 + 1).clamp(max=w - 1), (y0 + 1).clamp(max=h - 1)
        fu, fv = u - x0, v - y0
        p00, p10, p01, p11 = img[y0, x0], img[y0, x1], img[y1, x0], img[y1, x1]
        top, bot = p00 + fu * (p10 - p00), p01 + fu * (p11 - p01)
        val = top + fv * (bot - top)
        gu, gv = (p10 - p00) + fv * ((p11 - p01) - (p10 - p00)), bot - top
        G = torch.stack([gu * c.fx / z, gv * c.fy / z, -(gu * c.fx * Y[..., 0] + gv * c.fy * Y[..., 1]) / (z * z)], -1)
        mk = ok.double()
        cnt = mk.sum(1).clamp(min=1)
        rt = (r - (r * mk).sum(1, keepdim=True) / cnt[:, None]) * mk
        stl = (val - (val * mk).sum(1, keepdim=True) / cnt[:, None]) * mk
        srr, sss, srs = (rt * rt).sum(1), (stl * stl).sum(1), (rt * stl).sum(1)
        den = torch.sqrt(srr * sss)
        valid = (ok.sum(1) >= case["patch_size"] ** 2 // 2) & (den >= 1e-9 * cnt)
        den = den.clamp(min=1e-30)
        ncc = (srs / den).clamp(-1, 1)
        e = ((ncc * torch.sqrt(srr / sss.clamp(min=1e-30)))[:, None] * stl - rt)
        dk = ((G @ A)[..., None] * dX).sum(-2) * mk[..., None]
        pk = torch.cat([torch.linalg.cross(Y, G, dim=-1), G], -1) * mk[..., None]
        grads.append((e[..., None] * dk).sum(1) / den[:, None])
        poses.append((e[..., None] * pk).sum(1) / den[:, None])
        sd, ssd = dk.sum(1), (stl[..., None] * dk).sum(1)
        sdd = torch.einsum("nki,nkj->nij", dk, dk)
        sss = sss.clamp(min=1e-30)[:, None, None]
        Hm = (sdd - sd[:, :, None] * sd[:, None] / cnt[:, None, None] - ssd[:, :, None] * ssd[:, None] / sss) / sss
        gns.append(torch.stack([Hm[:, 0, 0], Hm[:, 0, 1], Hm[:, 0, 2], Hm[:, 1, 1], Hm[:, 1, 2], Hm[:, 2, 2]], -1))
        costs.append(torch.where(valid, 1 - ncc, torch.full_like(ncc, math.inf)))
    costs = torch.stack(costs, 1)
    nv = torch.isfinite(costs).sum(1)
    k = nv.clamp(max=case["best_k"] if case["best_k"] > 0 else len(sc.sources))
    rank = costs.argsort(dim=1, stable=True).argsort(dim=1, stable=True)
    rn = torch.sqrt((qc * qc).sum(-1))
    faces = (kappa < -0.05 * rn) & (nv > 0)
    sel = (rank < k[:, None]) & faces[:, None]
    wgt = sel.double() / k.clamp(min=1)[:, None]
    pick = lambda v: torch.where(sel[..., None], torch.stack(v, 1), torch.zeros((), **f8)) * wgt[..., None]  # noqa: E731
    cost = torch.where(faces, (torch.where(sel, costs, torch.zeros_like(costs)) * wgt).sum(1),
                       torch.full((N,), 1e30, **f8))
    assert K2 == case["patch_size"] ** 2 or case["patch_size"] % 2 == 0
    return {"cost": cost.cpu().numpy(), "grad": pick(grads).sum(1).cpu().numpy(),
            "gn": pick(gns).sum(1).cpu().numpy(), "pose": pick(poses).cpu().numpy()}


def _exact_fuse(case, st):
    """FuseDepthMaps: voxel means of the kept points in FP64, voxels in the
    order of their first points."""
    cfg = st["cfg"]
    pos, nrm, conf = [], [], []
    for m, p, k, keep in zip(st["maps"], st["poses"], st["intr"], st["keep"]):
        ok = np.isfinite(m.depth) & (m.support_count >= cfg.min_view_consistency) & (keep > 0)
        y, x = np.nonzero(ok)
        R, t = p[:9].reshape(3, 3), p[9:12]
        ray = [(x + 0.5 - k[2]) / k[0], (y + 0.5 - k[3]) / k[1], np.ones(len(x))]
        z = m.depth[ok].astype(np.float64)
        pc = [ray[i] * z - t[i] for i in range(3)]
        pos.append(np.stack([R[0, i] * pc[0] + R[1, i] * pc[1] + R[2, i] * pc[2] for i in range(3)], -1))
        nw = np.stack([R[0, i] * ray[0] + R[1, i] * ray[1] + R[2, i] * ray[2] for i in range(3)], -1)
        nrm.append(-nw / np.linalg.norm(nw, axis=1, keepdims=True))
        conf.append(m.confidence[ok].astype(np.float64))
    pos, nrm, conf = np.concatenate(pos), np.concatenate(nrm), np.concatenate(conf)
    v = np.floor(pos / cfg.fusion_voxel_size_m).astype(np.int64).astype(np.uint64)
    key = (v[:, 0] * np.uint64(73856093)) ^ (v[:, 1] * np.uint64(19349663)) ^ (v[:, 2] * np.uint64(83492791))
    _, first, inv, cnt = np.unique(key, return_index=True, return_inverse=True, return_counts=True)
    order = np.argsort(first, kind="stable")
    total = lambda a: np.bincount(inv.reshape(-1), weights=a, minlength=len(cnt))[order]  # noqa: E731
    c = cnt[order].astype(np.float64)
    n = np.stack([total(nrm[:, i]) for i in range(3)], -1)
    return {"positions": np.stack([total(pos[:, i]) for i in range(3)], -1) / c[:, None],
            "normals": n / np.linalg.norm(n, axis=1, keepdims=True),
            "confidences": np.minimum(1.0, total(conf) / c * np.sqrt(c)), "keys": None, "counts": None}


def exact(case, seed):
    """Searches (maps, the stage, RefineSubpixel) end at whichever of two nearly
    equal costs is lower, and the surface points of a grid are where its sign
    changes: they have no value in 64 bits apart from the search's own.
    Consistency counts are whole numbers."""
    fn = {"ncc": _exact_ncc, "adjoint": _exact_adjoint, "fuse": _exact_fuse}.get(case["kind"])
    return None if fn is None else fn(case, prepare(case, seed))
