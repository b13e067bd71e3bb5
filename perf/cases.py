"""Timed cases of the framework: what a user's program asks of it, from one
small solve to the largest scene, through the public entry points.

  solve   gba.solve / gba.solve_batch: host buffers in, host buffers out, the
          structure built, solved and thrown away (the drop-in call, and what
          the request server does for each micro-batch)
  plan    a resident plan (gba_plan_create in prepare), run again and read
          back through the C ABI into the caller's buffer, as a program does
          that solves the same structure repeatedly
  tri     gba.triangulate: batched multi-view triangulation, host buffers

Scenes are the benchmark's (ring windows, the grid seen from above, the random
walk), drawn here on the GPU from the seed with the same shapes and value
distributions.  Mixed-precision solves run a fixed number of LM iterations with
the stopping tests off, as the benchmark and the server do; FP64 solves use the
framework's default options (stop when converged).
"""
import ctypes
import math

import numpy as np
import torch

from hs_sfm_gb300 import abi, gba, synthetic

DEVICE = "cuda"
RADIAL, INTRINSIC = synthetic.COMPUTE_RADIAL, synthetic.COMPUTE_INTRINSIC


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one small adjustment with the default options: the reference's own test size
        {"name": "solve_ring_fp64", "call": "solve", "scene": "ring", "images": 10, "points": 1000,
         "lo": 5, "hi": 5, "count": 1, "precision": "fp64", "iterations": 50},
        # one local window of the request stream's median size
        {"name": "solve_window_mixed", "call": "solve", "scene": "ring", "images": 20, "points": 5000,
         "lo": 3, "hi": 8, "count": 1, "precision": "mixed", "iterations": 10},
        # a micro-batch of requests of different sizes
        {"name": "solve_batch_mixed", "call": "solve", "scene": "ring", "images": 20, "points": 5000,
         "lo": 3, "hi": 8, "count": 8, "precision": "mixed", "iterations": 10},
        # a small window solved again and again (tracking): launches and latency; odd sizes
        {"name": "plan_window_mixed", "call": "plan", "scene": "ring", "images": 13, "points": 2311,
         "lo": 3, "hi": 8, "count": 1, "precision": "mixed", "iterations": 10},
        # windows in the plain FP64 precision
        {"name": "plan_windows_fp64", "call": "plan", "scene": "ring", "images": 22, "points": 7500,
         "lo": 3, "hi": 8, "count": 24, "precision": "fp64", "iterations": 50},
        # the batch of local windows
        {"name": "plan_windows_mixed", "call": "plan", "scene": "ring", "images": 22, "points": 10250,
         "lo": 3, "hi": 8, "count": 512, "precision": "mixed", "iterations": 10},
        # the aerial grid, the benchmark's main workload
        {"name": "plan_grid_mixed", "call": "plan", "scene": "grid", "images": 200, "points": 100000,
         "lo": 4, "hi": 12, "count": 1, "precision": "mixed", "iterations": 20},
        # the same with the default precision and stopping tests
        {"name": "plan_grid_fp64", "call": "plan", "scene": "grid", "images": 200, "points": 100000,
         "lo": 4, "hi": 12, "count": 1, "precision": "fp64", "iterations": 50},
        # the grid with its camera calibrated along (shared intrinsics free)
        {"name": "plan_grid_free_mixed", "call": "plan", "scene": "grid_free", "images": 200, "points": 100000,
         "lo": 4, "hi": 12, "count": 1, "precision": "mixed", "iterations": 20},
        # the largest scene: long track, outliers, Huber loss, block-Jacobi PCG
        {"name": "plan_walk_pcg_mixed", "call": "plan", "scene": "walk", "images": 2000, "points": 1000000,
         "lo": 2, "hi": 60, "count": 1, "precision": "mixed", "iterations": 10},
        # a frame's new tracks, and a whole scene's
        {"name": "tri_3001", "call": "tri", "scene": "tracks", "images": 24, "points": 3001,
         "lo": 2, "hi": 8, "count": 1, "precision": "fp64", "iterations": 50},
        {"name": "tri_1m", "call": "tri", "scene": "tracks", "images": 200, "points": 1000000,
         "lo": 2, "hi": 12, "count": 1, "precision": "fp64", "iterations": 50},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "batch", "window", "windows", "grid", "grid_free", "walk", "tri"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    c = {"call": "plan", "scene": "ring", "images": 0, "points": 0, "lo": 3, "hi": 8, "count": 1,
         "precision": precision, "iterations": 50 if precision == "fp64" else 10}
    if kind in ("solve", "batch", "window", "windows"):
        c["images"] = _log(rng, 5, 40)
        c["points"] = _log(rng, 500, 20000)
        c["call"] = "solve" if kind in ("solve", "batch") else "plan"
        if kind == "batch":
            c["count"] = rng.randint(2, 16)
        if kind == "windows":
            c["count"] = _log(rng, 8, 32 if precision == "fp64" else 256)
    elif kind in ("grid", "grid_free"):
        c.update(scene=kind, images=_log(rng, 40, 200), points=_log(rng, 5000, 100000), lo=4, hi=12)
        if kind == "grid_free":
            c.update(precision="mixed", iterations=10)
    elif kind == "walk":
        c.update(scene="walk", images=_log(rng, 100, 2000), lo=2, hi=60, precision="mixed", iterations=10)
        c["points"] = _log(rng, 20000, min(1000000, 500 * c["images"]))
    else:
        c.update(call="tri", scene="tracks", images=rng.randint(16, 200), points=_log(rng, 1000, 1000000),
                 hi=rng.randint(5, 12), precision="fp64", iterations=50)
        c["lo"] = 2
    return c


def _options(case):
    mixed = case["precision"] == "mixed"
    kw = dict(max_iterations=case["iterations"],
              precision=abi.PRECISION_MIXED if mixed else abi.PRECISION_FP64)
    if mixed:   # a fixed number of iterations
        kw.update(eps1=0.0, eps2=0.0)
    if case["scene"] == "walk":
        kw.update(loss=abi.LOSS_HUBER, huber_delta=1.0, linear_solver=abi.LINEAR_PCG)
    return abi.make_options(**kw)


class _PlanState:
    """A resident plan and the caller's result buffer (every problem's x, one
    after the other)."""

    def __init__(self, case, seed):
        scenes = _scenes(case, seed)
        self.plan = gba.Plan(scenes, _options(case))
        sizes = [len(s.x0) for s in scenes]
        self.x = np.zeros(sum(sizes))
        at = self.x.ctypes.data + 8 * (np.cumsum(sizes) - sizes)
        dp = ctypes.POINTER(ctypes.c_double)
        self.xp = (dp * len(scenes))(*[ctypes.cast(int(a), dp) for a in at])
        self.reports = (abi.Report * len(scenes))()


class _SolveState:
    def __init__(self, case, seed):
        self.scenes = _scenes(case, seed)
        self.options = _options(case)


class _TriState:
    def __init__(self, case, seed):
        self.batch = _tracks(case, seed)


def prepare(case, seed):
    return {"plan": _PlanState, "solve": _SolveState, "tri": _TriState}[case["call"]](case, seed)


def run(state):
    if isinstance(state, _PlanState):
        state.plan.run()
        st = gba.lib().gba_plan_get_all(state.plan.h, state.xp, state.reports)
        if st != abi.GBA_OK:
            raise gba.GbaError(st, "gba_plan_get_all")
        return {"x": state.x, **_costs(state.reports)}
    if isinstance(state, _TriState):
        points, status = gba.triangulate(state.batch)
        return {"points": points, "status": status}
    if len(state.scenes) == 1:
        x, rep = gba.solve(state.scenes[0], state.options)
        return {"x": x, **_costs([rep])}
    xs, reps = gba.solve_batch(state.scenes, state.options)
    return {"x": xs, **_costs(reps)}


def _costs(reports):
    return {"initial": np.array([r.initial_cost for r in reports]),
            "final": np.array([r.final_cost for r in reports])}


def work(case):
    """Per LM iteration: every key's observation, indices and Jacobian work,
    the parameters read and written, the key pairs' products and the reduced
    system's factorization (or PCG products)."""
    n, p = case["count"], case["points"]
    if case["count"] > 1:      # sizes spread around the case's
        p = int(p * (1.0 if case["call"] == "plan" else 1.1))
    i = case["images"]
    if case["call"] == "tri":
        m = p * (case["lo"] + case["hi"]) / 2.0
        return {"bytes": 24.0 * m + 28.0 * p, "flops": 6 * 150.0 * m}
    k = 10.0 if case["scene"] == "walk" else min((case["lo"] + case["hi"]) / 2.0, i)
    keys = n * p * k
    iters = case["iterations"] if case["precision"] == "mixed" else 8
    unknowns = 6.0 * i + (8 if case["scene"] == "grid_free" else 0)
    solve = n * unknowns ** 3 / 3.0
    if case["scene"] == "walk":
        solve = 20 * 72.0 * i * min(i, 40)
    pairs = keys * (k + 1) / 2.0
    return {"bytes": iters * (24.0 * keys + n * (48.0 * p + 96.0 * i)),
            "flops": iters * (350.0 * keys + 216.0 * pairs + solve)}


# ---------------------------------------------------------------------------
# scenes (hs_sfm_gb300/synthetic.py's, drawn on the GPU)
# ---------------------------------------------------------------------------
def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)


def _skew(v):
    z = torch.zeros_like(v[:, 0])
    return torch.stack([z, -v[:, 2], v[:, 1], v[:, 2], z, -v[:, 0], -v[:, 1], v[:, 0], z], 1).view(-1, 3, 3)


def _rotation(r):
    """Rotation matrices of angle-axis vectors r [n, 3]."""
    t = r.square().sum(1).sqrt().clamp_min(1e-30)
    k = _skew(r / t[:, None])
    kk = (k[:, :, :, None] * k[:, None, :, :]).sum(2)
    return (torch.eye(3, dtype=r.dtype, device=r.device) + torch.sin(t)[:, None, None] * k
            + (1 - torch.cos(t))[:, None, None] * kk)


def _camera_points(images, img, X):
    R = _rotation(images[:, :3])
    return (R[img] * X[:, None, :]).sum(2) + images[img, 3:]


def _keys(images, img, X, cam):
    """Observations [n, 2] of the points X in the images img; cam = the full
    ten parameters [k1 k2 k3 d1 d2 f s cx cy a]."""
    y = _camera_points(images, img, X)
    n0, n1 = y[:, 0] / y[:, 2], y[:, 1] / y[:, 2]
    r2 = n0 * n0 + n1 * n1
    c = 1.0 + cam[0] * r2 + cam[1] * r2 * r2 + cam[2] * r2 * r2 * r2
    n0, n1 = c * n0, c * n1
    return torch.stack([cam[5] * n0 + cam[7], cam[5] * n1 + cam[8]], 1), y[:, 2]


def _full(mask, cam):
    out = [0.0] * 5 + [1.0, 0.0, 0.0, 0.0, 1.0]
    if mask & RADIAL:
        out[0:3] = list(cam[:3])
    if mask & INTRINSIC:
        out[5:10] = list(cam[-5:])
    return [float(v) for v in out]


def _scene(gen, rng, name, images, points, fm, mask, fix, cam, outliers=0.0):
    """Observed keys (1 px noise, rounded to float32), the perturbed initial x."""
    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=DEVICE, dtype=torch.float64)

    img = _t(images)
    obs = _keys(img, fm[:, 0], points[fm[:, 1]], _full(mask, cam))[0] + normal(len(fm), 2)
    if outliers:
        bad = torch.rand(len(fm), generator=gen, device=DEVICE) < outliers
        any_ = torch.rand(len(fm), 2, generator=gen, device=DEVICE, dtype=torch.float64)
        obs = torch.where(bad[:, None], any_ * torch.tensor([1920.0, 1080.0], dtype=torch.float64, device=DEVICE), obs)
    p0 = points + 0.05 * normal(len(points), 3)
    R = synthetic.rotvec_to_matrix(rng.normal(0, 0.01, (len(images), 3))) @ synthetic.rotvec_to_matrix(images[:, :3])
    i0 = np.concatenate([synthetic.matrix_to_rotvec(R), images[:, 3:] + rng.normal(0, 0.05, (len(images), 3))], 1)
    p0, pts = p0.cpu().numpy(), points.cpu().numpy()
    parts = [p0.reshape(-1), i0.reshape(-1)] + ([] if fix & synthetic.FIX_CAMERAS else [cam])
    true = [pts.reshape(-1), images.reshape(-1)] + ([] if fix & synthetic.FIX_CAMERAS else [cam])
    return synthetic.Scene(
        name=name, points=pts, images=images, cameras=cam[None, :],
        image_camera_map=np.zeros(len(images), np.int64), feature_maps=fm.cpu().numpy(), intrinsic_mask=mask,
        fix_mask=fix, near_y=obs.float().double().cpu().numpy().reshape(-1), x0=np.concatenate(parts),
        x_true=np.concatenate(true))


def _down(rng, centers):
    """Images at `centers` looking down, jittered by 0.02 rad."""
    R = synthetic.rotvec_to_matrix(rng.normal(0, 0.02, (len(centers), 3))) @ np.diag([1.0, -1.0, -1.0])
    return np.concatenate([synthetic.matrix_to_rotvec(R), -np.einsum("nij,nj->ni", R, centers)], 1)


def _ring(gen, rng, images, points, lo, hi, scale):
    phi = 2 * np.pi * np.arange(images) / images
    centers = np.stack([10 * scale * np.cos(phi), 10 * scale * np.sin(phi), np.zeros(images)], 1)
    R = synthetic.look_at(centers, np.zeros((images, 3)), np.array([0.0, 0.0, 1.0]))
    img = np.concatenate([synthetic.matrix_to_rotvec(R), -np.einsum("nij,nj->ni", R, centers)], 1)
    X = (torch.rand(points, 3, generator=gen, device=DEVICE, dtype=torch.float64) * 4 - 2) * scale
    order = (X[:, None, :] - _t(centers)[None]).square().sum(2).argsort(dim=1, stable=True)
    k = torch.randint(lo, hi + 1, (points,), generator=gen, device=DEVICE).clamp_max(images)
    take = torch.arange(images, device=DEVICE)[None, :] < k[:, None]
    rows = torch.repeat_interleave(torch.arange(points, device=DEVICE), k)
    fm = torch.stack([order[take], rows], 1)
    cam = synthetic.default_intrinsics(INTRINSIC)
    return _scene(gen, rng, "ring", img, X, fm, INTRINSIC, synthetic.FIX_CAMERAS, cam)


def _kept(points, rows, cols):
    """The points with at least two keys, renumbered, and their keys."""
    count = torch.bincount(rows, minlength=len(points))
    keep = count >= 2
    number = torch.cumsum(keep.long(), 0) - 1
    sel = keep[rows]
    return points[keep], torch.stack([cols[sel], number[rows[sel]]], 1)


def _grid(gen, rng, images, points, lo, hi, free):
    nx = int(round(math.sqrt(images * 2)))
    ny = max(1, images // nx)
    while nx * ny < images:
        ny += 1
    gx, gy = np.meshgrid(np.linspace(-19, 19, nx), np.linspace(-18, 18, ny), indexing="ij")
    centers = np.stack([gx.reshape(-1), gy.reshape(-1), np.full(nx * ny, 12.0)], 1)[:images]
    centers = centers + np.concatenate([rng.uniform(-0.5, 0.5, (images, 2)), rng.uniform(-0.3, 0.3, (images, 1))], 1)
    img = _down(rng, centers)
    mask = RADIAL | INTRINSIC
    cam = synthetic.default_intrinsics(mask, rng, 0.1)
    X = torch.rand(points, 3, generator=gen, device=DEVICE, dtype=torch.float64) * 2 - 1
    X = X * torch.tensor([20.0, 20.0, 2.0], dtype=torch.float64, device=DEVICE)
    want = torch.randint(lo, hi + 1, (points,), generator=gen, device=DEVICE)
    t, rows, cols = _t(img), [], []
    every = torch.arange(images, device=DEVICE)
    for a in range(0, points, 20000):
        b = min(points, a + 20000)
        r = torch.arange(a, b, device=DEVICE).repeat_interleave(images)
        c = every.repeat(b - a)
        key, depth = _keys(t, c, X[r], _full(mask, cam))
        vis = ((depth > 0.1) & (key[:, 0] > 0) & (key[:, 0] < 1920) & (key[:, 1] > 0) & (key[:, 1] < 1080)).view(b - a, images)
        pick = torch.rand(b - a, images, generator=gen, device=DEVICE, dtype=torch.float64)
        order = torch.where(vis, pick, torch.full_like(pick, 2.0)).argsort(dim=1, stable=True)
        k = torch.minimum(want[a:b], vis.sum(1))
        chosen = torch.zeros(b - a, images, dtype=torch.bool, device=DEVICE)
        chosen.scatter_(1, order, every[None, :] < k[:, None])
        got = chosen.nonzero()
        rows.append(got[:, 0] + a)
        cols.append(got[:, 1])
    X, fm = _kept(X, torch.cat(rows), torch.cat(cols))
    fix = 0 if free else synthetic.FIX_CAMERAS
    return _scene(gen, rng, "grid", img, X, fm, mask, fix, cam)


def _walk(gen, rng, images, points, longest):
    ang = rng.uniform(0, 2 * np.pi, images)
    xy = np.cumsum(np.stack([np.cos(ang), np.sin(ang)], 1), 0)
    img = _down(rng, np.concatenate([xy, np.full((images, 1), 15.0)], 1))
    u = torch.rand(points, generator=gen, device=DEVICE, dtype=torch.float64)
    k = 2 + torch.floor(torch.log1p(-u) / math.log(1 - 1.0 / 9.0)).long()      # 1 + geometric(1/9)
    k = k.clamp_max(min(longest, images))
    start = (torch.rand(points, generator=gen, device=DEVICE, dtype=torch.float64) * (images - k + 1)).long()
    sums = _t(np.concatenate([np.zeros((1, 2)), np.cumsum(xy, 0)], 0))
    mid = (sums[start + k] - sums[start]) / k[:, None]
    X = torch.randn(points, 2, generator=gen, device=DEVICE, dtype=torch.float64) * 1.5 + mid
    z = torch.rand(points, 1, generator=gen, device=DEVICE, dtype=torch.float64) * 4 - 2
    X = torch.cat([X, z], 1)
    rows = torch.repeat_interleave(torch.arange(points, device=DEVICE), k)
    cols = torch.arange(len(rows), device=DEVICE) - torch.repeat_interleave(torch.cumsum(k, 0) - k, k) + start[rows]
    cam = synthetic.default_intrinsics(INTRINSIC)
    key, depth = _keys(_t(img), cols, X[rows], _full(INTRINSIC, cam))
    vis = (depth > 0.1) & (key[:, 0] > -200) & (key[:, 0] < 2120) & (key[:, 1] > -200) & (key[:, 1] < 1280)
    X, fm = _kept(X, rows[vis], cols[vis])
    return _scene(gen, rng, "walk", img, X, fm, INTRINSIC, synthetic.FIX_CAMERAS, cam, outliers=0.01)


def _scenes(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    if case["scene"] in ("grid", "grid_free"):
        return [_grid(gen, rng, case["images"], case["points"], case["lo"], case["hi"], case["scene"] == "grid_free")]
    if case["scene"] == "walk":
        return [_walk(gen, rng, case["images"], case["points"], case["hi"])]
    if case["count"] == 1:
        return [_ring(gen, rng, case["images"], case["points"], case["lo"], case["hi"], float(rng.uniform(0.5, 2.0)))]
    out = []
    sizes = np.random.default_rng(12345)   # the batch's sizes are the case's, not the seed's
    for _ in range(case["count"]):
        if case["call"] == "plan":         # uniform around the case's size
            i = int(sizes.integers(max(5, case["images"] // 4), case["images"] * 7 // 4 + 1))
            p = int(sizes.integers(max(200, case["points"] // 20), case["points"] * 39 // 20 + 1))
        else:                              # log-normal requests around it
            i = int(np.clip(round(case["images"] * math.exp(sizes.normal(0, 0.5))), 5, 48))
            p = int(np.clip(round(case["points"] * math.exp(sizes.normal(0, 0.5))), 200, 40000))
        out.append(_ring(gen, rng, i, p, case["lo"], case["hi"], float(rng.uniform(0.5, 2.0))))
    return out


def _tracks(case, seed):
    """Views on a ring with their own intrinsics and distortion; each point
    seen by lo..hi views about 15 degrees apart, 0.5 px noise."""
    views = case["images"]
    t = synthetic.triangulation_batch(seed=seed, num_points=1, num_views=views)
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    n = case["points"]
    X = torch.rand(n, 3, generator=gen, device=DEVICE, dtype=torch.float64) * 4 - 2
    k = torch.randint(case["lo"], case["hi"] + 1, (n,), generator=gen, device=DEVICE).clamp_max(views)
    first = torch.randint(0, views, (n,), generator=gen, device=DEVICE)
    off = torch.cumsum(k, 0)
    pt = torch.repeat_interleave(torch.arange(n, device=DEVICE), k)
    pos = torch.arange(len(pt), device=DEVICE) - (off - k)[pt]
    view = (first[pt] + max(1, views // 24) * pos) % views
    key = _view_keys(_t(t.intrinsics), _t(t.extrinsics), view, X[pt])[0]
    key = key + 0.5 * torch.randn(len(pt), 2, generator=gen, device=DEVICE, dtype=torch.float64)
    return synthetic.TriangulationBatch(
        intrinsics=t.intrinsics, extrinsics=t.extrinsics,
        track_offsets=np.concatenate([[0], off.cpu().numpy()]).astype(np.int64), track_views=view.cpu().numpy(),
        track_keys=key.cpu().numpy(), points=X.cpu().numpy())


def _view_keys(intr, extr, view, X):
    """Keys and their derivatives with respect to X (sfm_utility's camera)."""
    R = _rotation(extr[:, :3])[view]
    c = (R * (X - extr[view, 3:])[:, None, :]).sum(2)
    f, s, cx, cy, a, k1, k2, k3, d1, d2 = intr[view].unbind(1)
    x, y, iz = c[:, 0] / c[:, 2], c[:, 1] / c[:, 2], 1.0 / c[:, 2]
    r2 = x * x + y * y
    q = 1 + k1 * r2 + k2 * r2 ** 2 + k3 * r2 ** 3
    dq = k1 + 2 * k2 * r2 + 3 * k3 * r2 ** 2                                   # d q / d r2
    ex = q * x + 2 * d1 * x * y + d2 * (r2 + 2 * x * x)
    ey = q * y + 2 * d2 * x * y + d1 * (r2 + 2 * y * y)
    exx = q + 2 * dq * x * x + 2 * d1 * y + 6 * d2 * x
    exy = 2 * dq * x * y + 2 * d1 * x + 2 * d2 * y
    eyy = q + 2 * dq * y * y + 2 * d2 * x + 6 * d1 * y
    key = torch.stack([f * ex + s * ey + cx, f * a * ey + cy], 1)
    n = torch.stack([torch.stack([f * exx + s * exy, f * exy + s * eyy], 1),
                     torch.stack([f * a * exy, f * a * eyy], 1)], 1)           # d key / d (x, y)
    z = torch.zeros_like(iz)
    p = torch.stack([torch.stack([iz, z, -x * iz], 1), torch.stack([z, iz, -y * iz], 1)], 1)
    return key, _mm(_mm(n, p), R)


# ---------------------------------------------------------------------------
# exact values: the same algorithms in torch FP64
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["call"] == "tri":
        return _exact_tracks(_tracks(case, seed))
    if case["scene"] == "walk" and case["points"] * case["images"] > 2e7:   # its reduced system is too large here
        return None
    if case["count"] > 64:
        return None
    got = [_exact_solve(s, _options(case)) for s in _scenes(case, seed)]
    x = [g[0] for g in got]
    if case["call"] == "plan" or len(x) == 1:
        x = np.concatenate(x)
    return {"x": x, "initial": np.array([g[1] for g in got]), "final": np.array([g[2] for g in got])}


def _mm(a, b):
    """Products of small matrices, elementwise (no reduced-precision units)."""
    return (a[:, :, :, None] * b[:, None, :, :]).sum(2)


def _exact_tracks(t):
    """The least-squares point of every track: Gauss-Newton from the truth."""
    intr, extr, view, key = _t(t.intrinsics), _t(t.extrinsics), _t(t.track_views), _t(t.track_keys)
    off = _t(t.track_offsets)
    n = len(off) - 1
    pt = torch.repeat_interleave(torch.arange(n, device=DEVICE), off[1:] - off[:-1])
    X = _t(t.points)
    for _ in range(30):
        k, J = _view_keys(intr, extr, view, X[pt])
        r = k - key
        N = torch.zeros(n, 3, 3, dtype=torch.float64, device=DEVICE).index_add_(0, pt, _mm(J.transpose(1, 2), J))
        g = torch.zeros(n, 3, dtype=torch.float64, device=DEVICE).index_add_(0, pt, (J * r[:, :, None]).sum(1))
        step = torch.linalg.solve(N, g)
        X = X - step
        if float(step.abs().max()) < 1e-14:
            break
    return {"points": X.cpu().numpy(), "status": None}


class _Problem:
    """Residuals, Jacobian blocks and normal equations of one scene in FP64."""

    def __init__(self, s, opt):
        self.opt, self.mask = opt, s.intrinsic_mask
        fm = _t(s.feature_maps)
        fm_key = fm[:, 1] * s.number_of_images + fm[:, 0]
        order = fm_key.argsort()
        self.img, self.pt = fm[order, 0], fm[order, 1]
        self.obs = _t(s.near_y.reshape(-1, 2))[order]
        self.P, self.I = s.number_of_points, s.number_of_images
        self.cams = 0 if s.fix_mask & synthetic.FIX_CAMERAS else s.cameras.shape[1]
        x = _t(s.x0)
        self.x0 = (x[:3 * self.P].view(-1, 3), x[3 * self.P:3 * self.P + 6 * self.I].view(-1, 6),
                   x[3 * self.P + 6 * self.I:] if self.cams else _t(s.cameras[0]))
        self.cols = [j for j in range(10) if (j < 3 and self.mask & RADIAL) or (j >= 5 and self.mask & INTRINSIC)]

    def residual(self, x):
        cam = torch.zeros(10, dtype=torch.float64, device=DEVICE)
        cam[5] = cam[9] = 1.0
        cam[self.cols] = x[2]
        y = _camera_points(x[1], self.img, x[0][self.pt])
        iz = 1.0 / y[:, 2]
        n0, n1 = y[:, 0] * iz, y[:, 1] * iz
        r2 = n0 * n0 + n1 * n1
        q = 1 + cam[0] * r2 + cam[1] * r2 ** 2 + cam[2] * r2 ** 3
        e0, e1 = q * n0, q * n1
        f, s, a = cam[5], cam[6], cam[9]
        r = torch.stack([f * e0 + s * e1 + cam[7], f * a * e1 + cam[8]], 1) - self.obs
        sq = r.square().sum(1)
        w = torch.ones_like(sq)
        rho = sq
        if self.opt.loss == abi.LOSS_HUBER:
            d = self.opt.huber_delta
            root = sq.sqrt()
            out = root > d
            rho = torch.where(out, 2 * d * root - d * d, sq)
            w = torch.where(out, d / root.clamp_min(1e-300), w)
        return float(rho.sum()), r, w, (cam, y, iz, n0, n1, r2, q, e0, e1)

    def jacobian(self, x, got):
        _, r, w, (cam, y, iz, n0, n1, r2, q, e0, e1) = got
        f, s, a = cam[5], cam[6], cam[9]
        dq = cam[0] + 2 * cam[1] * r2 + 3 * cam[2] * r2 ** 2
        d00, d01, d11 = q + 2 * dq * n0 * n0, 2 * dq * n0 * n1, q + 2 * dq * n1 * n1
        m = torch.stack([torch.stack([f * d00 + s * d01, f * d01 + s * d11], 1),
                         torch.stack([f * a * d01, f * a * d11], 1)], 1)
        z = torch.zeros_like(iz)
        p = torch.stack([torch.stack([iz, z, -n0 * iz], 1), torch.stack([z, iz, -n1 * iz], 1)], 1)
        jt = _mm(m, p)                                                        # d key / d (camera point)
        rot = x[1][:, :3]
        R = _rotation(rot)
        th2 = rot.square().sum(1)
        th = th2.sqrt()
        small = th < 1e-4
        t = torch.where(small, torch.ones_like(th), th)
        c1 = torch.where(small, 0.5 - th2 / 24, (1 - torch.cos(t)) / (t * t))
        c2 = torch.where(small, 1.0 / 6 - th2 / 120, (t - torch.sin(t)) / (t ** 3))
        k = _skew(rot)
        left = torch.eye(3, dtype=torch.float64, device=DEVICE) + c1[:, None, None] * k + c2[:, None, None] * _mm(k, k)
        turned = y - x[1][self.img, 3:]                                       # R X
        jr = -_mm(jt, _mm(_skew(turned), left[self.img]))                     # d (R X) / d r = -[R X]x J_l(r)
        ji = torch.cat([jr, jt], 2)
        jp = _mm(jt, R[self.img])
        sw = w.sqrt()[:, None]
        jc = None
        if self.cams:
            cols = []
            for j in self.cols:
                o, i0 = torch.ones_like(n0), torch.zeros_like(n0)
                if j < 3:
                    pw = r2 ** (j + 1)
                    cols.append(torch.stack([f * pw * n0 + s * pw * n1, f * a * pw * n1], 1))
                else:
                    cols.append(torch.stack([(e0, a * e1), (e1, i0), (o, i0), (i0, o), (i0, f * e1)][j - 5], 1))
            jc = torch.stack(cols, 2) * sw[:, :, None]
        return jp * sw[:, :, None], ji * sw[:, :, None], jc, r * sw

    def normal(self, x, got):
        jp, ji, jc, r = self.jacobian(x, got)

        def add(index, n, v):
            return torch.zeros(n, *v.shape[1:], dtype=torch.float64, device=DEVICE).index_add_(0, index, v)

        tp, ti = jp.transpose(1, 2), ji.transpose(1, 2)
        N = {"jp": jp, "ji": ji, "jc": jc,
             "V": add(self.pt, self.P, _mm(tp, jp)), "gp": add(self.pt, self.P, (jp * r[:, :, None]).sum(1)),
             "U": add(self.img, self.I, _mm(ti, ji)), "gi": add(self.img, self.I, (ji * r[:, :, None]).sum(1))}
        if jc is not None:
            tc = jc.transpose(1, 2)
            N.update(E=add(self.img, self.I, _mm(ti, jc)), Uc=_mm(tc, jc).sum(0), gc=(jc * r[:, :, None]).sum((0, 1)))
        return N

    def step(self, N, mu):
        """(N + mu I) delta = g by the Schur complement; None when it is not
        positive definite."""
        eye3 = torch.eye(3, dtype=torch.float64, device=DEVICE)
        C, bad = torch.linalg.cholesky_ex(N["V"] + mu * eye3)
        if int(bad.max()):
            return None
        Ci = torch.linalg.solve_triangular(C, eye3.expand_as(C), upper=False)
        h = _mm(Ci, N["gp"][:, :, None])[:, :, 0]
        Ck = Ci[self.pt]
        Z = _mm(Ck, _mm(N["jp"].transpose(1, 2), N["ji"]))
        I, c = self.I, self.cams
        blocks = torch.zeros(I * I, 36, dtype=torch.float64, device=DEVICE)
        d = 0
        while True:                                                           # keys d apart of the same point
            a = (self.pt[d:] == self.pt[:len(self.pt) - d]).nonzero()[:, 0]
            if not len(a):
                break
            for p0 in range(0, len(a), 2000000):
                q = a[p0:p0 + 2000000]
                blocks.index_add_(0, self.img[q + d] * I + self.img[q],
                                  _mm(Z[q + d].transpose(1, 2), Z[q]).view(-1, 36))
            d += 1
        low = -blocks.view(I, I, 6, 6)
        own = torch.arange(I, device=DEVICE)
        low[own, own] += N["U"]
        n = 6 * I + c
        S = torch.zeros(n, n, dtype=torch.float64, device=DEVICE)
        S[:6 * I, :6 * I] = low.permute(0, 2, 1, 3).reshape(6 * I, 6 * I)
        b = torch.zeros(n, dtype=torch.float64, device=DEVICE)
        zh = (Z * h[self.pt][:, :, None]).sum(1)
        b[:6 * I] = (N["gi"] - torch.zeros_like(N["gi"]).index_add_(0, self.img, zh)).reshape(-1)
        if c:
            W = torch.zeros(self.P, 3, c, dtype=torch.float64, device=DEVICE)
            W.index_add_(0, self.pt, _mm(N["jp"].transpose(1, 2), N["jc"]))
            Zc = _mm(Ci, W)
            E = N["E"] - torch.zeros_like(N["E"]).index_add_(0, self.img, _mm(Z.transpose(1, 2), Zc[self.pt]))
            S[6 * I:, :6 * I] = E.reshape(6 * I, c).T
            S[6 * I:, 6 * I:] = N["Uc"] - _mm(Zc.transpose(1, 2), Zc).sum(0)
            b[6 * I:] = N["gc"] - (Zc * h[:, :, None]).sum((0, 1))
        S.diagonal().add_(mu)
        L, bad = torch.linalg.cholesky_ex(S)                                  # reads the lower triangle
        if int(bad):
            return None
        y = torch.cholesky_solve(b[:, None], L)[:, 0]
        di, dc = y[:6 * I].view(-1, 6), y[6 * I:]
        t = h - torch.zeros_like(h).index_add_(0, self.pt, (Z * di[self.img][:, None, :]).sum(2))
        if c:
            t = t - (Zc * dc[None, None, :]).sum(2)
        return (Ci * t[:, :, None]).sum(1), di, dc

    def grad(self, N):
        return [N["gp"], N["gi"]] + ([N["gc"]] if self.cams else [])


def _exact_solve(s, opt):
    """Levenberg-Marquardt (Madsen, Nielsen & Tingleff 2004, Alg. 3.16) with
    the framework's stopping tests: x, initial and final cost."""
    P = _Problem(s, opt)
    x = P.x0
    got = P.residual(x)
    F = first = got[0]
    N = P.normal(x, got)
    diag = [N["V"].diagonal(dim1=1, dim2=2), N["U"].diagonal(dim1=1, dim2=2)] + ([N["Uc"].diagonal()] if P.cams else [])
    mu, nu = opt.tau * max(float(v.max()) for v in diag), 2.0
    free = 3 if P.cams else 2
    for _ in range(opt.max_iterations):
        g = P.grad(N)
        if max(float(v.abs().max()) for v in g) <= opt.eps1:
            break
        d = P.step(N, mu)
        if d is None:
            mu, nu = mu * nu, nu * 2
            continue
        dn2 = sum(float(v.square().sum()) for v in d[:free])
        xn2 = sum(float(v.square().sum()) for v in x[:free])
        if math.sqrt(dn2) <= opt.eps2 * (math.sqrt(xn2) + opt.eps2):
            break
        gd = sum(float((u * v).sum()) for u, v in zip(g, d))
        new = tuple(x[j] - d[j] if j < free else x[j] for j in range(3))
        got = P.residual(new)
        denom = mu * dn2 + gd
        rho = (F - got[0]) / denom if denom else -1.0
        if math.isfinite(got[0]) and denom > 0 and rho > 0:
            x, F = new, got[0]
            mu, nu = mu * max(1.0 / 3.0, 1 - (2 * rho - 1) ** 3), 2.0
            N = P.normal(x, got)
        else:
            mu, nu = mu * nu, nu * 2
    return torch.cat([v.reshape(-1) for v in x[:free]]).cpu().numpy(), first, F
