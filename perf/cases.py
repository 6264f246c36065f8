"""Workloads of the bundle adjuster for timing and for comparing two builds.

Every case is work a user's program gives the library through its public
entry points: a complete robust adjustment from the handle API or from
CalcPLSA, a batch of scenes, the partitioned branch, the per-point refinement,
the Exteval evaluation.  The scenes are those of ``rpba_b200.scenes`` (arc,
street, aerial grid, city: the same cameras, track lengths, noise, outliers
and start perturbations), drawn on the GPU with torch so that a scene of any
size is made in well under a second.

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  inputs, handles and weights a program has in hand
  run(state)           one pass through the public entry points
  work(case)           bytes and operations the path cannot do without
  exact(case, seed)    64-bit values of the outputs that have closed ones
"""
from __future__ import annotations

import math

import numpy as np
import torch

import rpba_b200 as rb
from rpba_b200 import scenes, train_precond
from rpba_b200.block import Block

SOLVERS = {"pcg": rb.SOLVER_PCG, "direct": rb.SOLVER_DIRECT, "learned": rb.SOLVER_LEARNED}
PRECISIONS = {"fp64": rb.PREC_FP64, "mixed": rb.PREC_MIXED}
TRACK_MEAN = {"arc": 4.0, "street": 5.0, "aerial": 5.3, "city": 6.5}
PTS_PER_CAM = {"arc": 160, "street": 190, "aerial": 103, "city": 328}
CITY_CLUSTER = 274  # cameras of one city cluster


def _solve(name, scene, cams, solver, precision, tol=0.0, robust=True, k2=True, k4=True, f=True, points=0):
    return {"name": name, "op": "solve", "scene": scene, "cams": cams, "points": points or cams * PTS_PER_CAM[scene],
            "solver": solver, "precision": precision, "tol": tol, "robust": robust, "k2": k2, "k4": k4, "f": f}


def listed():
    return [
        # the smallest call: one in-place CalcPLSA of a dozen cameras, handle
        # creation and release included; latency, launches and host work
        {"name": "call_arc_12", "op": "call", "scene": "arc", "cams": 12, "points": 1500, "solver": "pcg",
         "precision": "fp64", "tol": 0.0, "robust": True, "k2": True, "k4": True, "f": True},
        # the basic object scan: drop-in FP64 form on a resident handle
        _solve("arc_50_fp64_pcg", "arc", 50, "pcg", "fp64", points=8000),
        # the street drive with the sparse direct form
        _solve("street_1000_fp64_direct", "street", 1000, "direct", "fp64", points=190_000),
        # the aerial survey in each form a user picks for it: drop-in FP64,
        # mixed precision with the direct solve, mixed two-level PCG
        _solve("aerial_3000_fp64_pcg", "aerial", 3000, "pcg", "fp64", points=310_000),
        _solve("aerial_3000_mixed_direct", "aerial", 3000, "direct", "mixed", points=310_000),
        _solve("aerial_3000_learned", "aerial", 3000, "learned", "mixed", tol=3e-5, points=310_000),
        # a district of the city in the drop-in form
        _solve("city_1370_fp64_pcg", "city", 5 * CITY_CLUSTER, "pcg", "fp64", points=450_000),
        # the whole city: the largest adjustment, the learned mixed form
        _solve("city_13700_learned", "city", 50 * CITY_CLUSTER, "learned", "mixed", tol=3e-5, points=4_500_000),
        # many uneven scans on one GPU (photo collections split into objects)
        {"name": "batch_24_mixed", "op": "batch", "scene": "arc", "scenes": 24, "cmin": 20, "cmax": 400,
         "solver": "pcg", "precision": "mixed", "tol": 0.0, "robust": True, "workers": 8},
        # the reference's Threads = 0 branch: partitioned RPBA of two city clusters
        {"name": "partitioned_548", "op": "partitioned", "scene": "city", "cams": 2 * CITY_CLUSTER, "points": 45_000,
         "parts": 8},
        # per-point refinement against fixed cameras with robust deletion
        {"name": "triangulate_310k", "op": "triangulate", "scene": "aerial", "cams": 3000, "points": 310_000,
         "mode": 2, "parts": 0},
        # Exteval: back-projection errors of every observation
        {"name": "exteval_190k", "op": "exteval", "scene": "street", "cams": 1000, "points": 190_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["solve"] * 6 + ["call", "batch", "partitioned", "triangulate", "exteval"])
    if op == "batch":
        lo = rng.randint(8, 60)
        return {"op": "batch", "scene": "arc", "scenes": rng.randint(3, 24), "cmin": lo,
                "cmax": lo + rng.randint(20, 300), "solver": "pcg", "precision": rng.choice(["mixed", "fp64"]),
                "tol": 0.0, "robust": True, "workers": rng.choice([1, 4, 8])}
    if op == "partitioned":
        n = rng.randint(2, 4)
        return {"op": "partitioned", "scene": "city", "cams": n * CITY_CLUSTER, "points": rng.randint(20_000, 90_000),
                "parts": rng.randint(2, 8)}
    if op == "triangulate":
        cams = _log(rng, 150, 3000)
        return {"op": "triangulate", "scene": "aerial", "cams": cams, "points": _log(rng, 2000, 400_000),
                "mode": rng.choice([0, 1, 2]), "parts": rng.choice([0, 0, 1, 4, 8])}
    if op == "exteval":
        return {"op": "exteval", "scene": "street", "cams": _log(rng, 300, 1500),
                "points": _log(rng, 10_000, 400_000)}
    scene = "arc" if op == "call" else rng.choice(["arc", "arc", "street", "aerial", "aerial", "city"])
    robust = rng.random() < 0.85
    adds = rng.choice([(True, True, True)] * 3 + [(False, False, True), (True, False, True), (False, False, False)])
    # the forms each scene family is adjusted with
    if scene == "arc":
        cams = _log(rng, 8, 400) if op == "solve" else _log(rng, 6, 60)
        per = rng.randint(100, 200)
        form = rng.choice([("pcg", "fp64"), ("pcg", "mixed"), ("direct", "fp64"), ("direct", "mixed")])
        tol, robust_adds = 0.0, adds
        robust = robust or cams > 60  # a large plain fit is pulled apart by its outliers
    elif scene == "street":
        cams, per, robust_adds = rng.randint(700, 1200), rng.randint(150, 250), (True, True, True)
        form, tol, robust = ("direct", "fp64"), 0.0, True
    elif scene == "aerial":
        cams, per, robust_adds = _log(rng, 150, 3000), rng.randint(90, 160), adds
        form = rng.choice([("pcg", "fp64"), ("direct", "mixed"), ("learned", "mixed"), ("direct", "fp64")])
        tol = rng.choice([3e-5, 1e-5]) if form[0] == "learned" else 0.0
    else:
        form = rng.choice([("learned", "mixed"), ("learned", "mixed"), ("pcg", "fp64")])
        cl = _log(rng, 2, 40) if form[0] == "learned" else rng.randint(2, 5)
        cams, per, robust_adds = cl * CITY_CLUSTER, rng.randint(150, 328), (True, True, True)
        robust = True
        tol = rng.choice([3e-5, 1e-5]) if form[0] == "learned" else 0.0
    k2, k4, f = robust_adds
    c = _solve("", scene, cams, form[0], form[1], tol, robust, k2, k4, f, points=cams * per + rng.randint(0, 63))
    del c["name"]
    c["op"] = op
    return c


# ------------------------------------------------------------------ scenes

def _cameras(scene, n, rng):
    """Rotations, centres, focal lengths and distortions of a scene's cameras
    (``rpba_b200.scenes``), and what its points are drawn from."""
    up = np.array([0.0, 1.0, 0.0])
    if scene == "arc":
        th = np.linspace(-0.5 * np.pi, 0.5 * np.pi, n) + rng.normal(0, 0.01, n)
        C = np.stack([10.0 * np.sin(th), 1.5 + rng.normal(0, 0.1, n), 10.0 * np.cos(th)], 1)
        T, fr = rng.normal(0, 0.2, (n, 3)), (400, 600)
        geo = {}
    elif scene == "street":
        C = np.stack([np.arange(n) * 3.0, 2.0 + rng.normal(0, 0.05, n), rng.normal(0, 0.3, n)], 1)
        T = C + np.stack([np.full(n, 20.0), rng.normal(0, 0.3, n), rng.normal(0, 0.5, n)], 1)
        fr, geo = (400, 600), {}
    elif scene == "aerial":
        nx = max(3, int(round(math.sqrt(1.2 * n))))
        h = 100.0 + 50.0 * (np.arange(n) // nx % 3) / 2.0
        sp = 45.0
        gx = (np.arange(n) % nx) * sp + rng.normal(0, 2, n)
        gy = (np.arange(n) // nx) * sp + rng.normal(0, 2, n)
        C = np.stack([gx, h + rng.normal(0, 1, n), gy], 1)
        T = np.stack([gx + rng.normal(0, 3, n), np.zeros(n), gy + rng.normal(0, 3, n)], 1)
        up, fr = np.array([0.0, 0.0, 1.0]), (1000, 3000)
        geo = {"nx": nx, "ny": (n + nx - 1) // nx, "sp": sp}
    else:
        ncl = n // CITY_CLUSTER
        cid = np.repeat(np.arange(ncl), CITY_CLUSTER)
        cc = np.stack([(np.arange(ncl) % 10) * 90.0, np.zeros(ncl), (np.arange(ncl) // 10) * 90.0], 1)
        th, rad = rng.uniform(0, 2 * np.pi, n), rng.uniform(35.0, 55.0, n)
        C = cc[cid] + np.stack([rad * np.cos(th), rng.uniform(2, 25, n), rad * np.sin(th)], 1)
        T = cc[cid] + rng.normal(0, 8.0, (n, 3)) * np.array([1.0, 0.3, 1.0])
        gx, gy = np.arange(ncl) % 10, np.arange(ncl) // 10
        nbr = [[d for d in range(ncl) if d != c and abs(gx[d] - gx[c]) <= 1 and abs(gy[d] - gy[c]) <= 1] or [c]
               for c in range(ncl)]
        geo = {"centers": cc, "nbr": np.array([(v * 8)[:8] for v in nbr])}
        fr = (400, 600)
    R = scenes.look_at(C, T, up)
    return R, C, rng.uniform(*fr, n), np.stack([rng.normal(0, 1e-2, n), rng.normal(0, 1e-4, n)], 1), geo


_MAX_TRACK = {"arc": 12, "street": 30, "aerial": 30, "city": 100}
_MAX_P = {"arc": 1.5, "street": 1.2, "aerial": 0.45, "city": 1.0}
_MIN_DEPTH = {"arc": 0.5, "street": 3.0, "aerial": 10.0, "city": 2.0}
_OUTLIERS = {"arc": 0.03, "street": 0.05, "aerial": 0.03, "city": 0.03}


def _project(R, t, f, k, X, cam):
    """BAL projection of X [.., 3] through the cameras cam."""
    P = torch.einsum("...ij,...j->...i", R[cam], X) + t[cam]
    z = torch.where(P[..., 2].abs() < 1e-9, torch.full_like(P[..., 2], -1e-9), P[..., 2])
    p = -P[..., :2] / z[..., None]
    r2 = (p * p).sum(-1)
    d = 1.0 + k[cam, 0] * r2 + k[cam, 1] * r2 * r2
    return f[cam, None] * d[..., None] * p if p.dim() == 2 else None, P[..., 2], p.abs().amax(-1)


def _observations(scene, n_cams, n_pts):
    """Observations of a scene: a little under the mean track length (geometric
    from 2 on, cut at the scene's longest track) that its cameras see."""
    if scene == "aerial":
        return int(2.8 * n_pts)  # the footprints end most tracks early
    q, longest = 1.0 - 1.0 / (TRACK_MEAN[scene] - 1.0), min(_MAX_TRACK[scene], n_cams)
    return int(0.95 * n_pts * (2.0 + sum(q ** i for i in range(1, longest - 1))))


def _points(scene, n_cams, n, geo, C, u):
    """Point positions and, for chosen rows, K proposed cameras per point."""
    dev = "cuda"
    r = lambda *s: torch.rand(*s, generator=u, device=dev, dtype=torch.float64)
    ints = lambda lo, hi, *s: torch.randint(lo, hi, s, generator=u, device=dev)
    if scene == "arc":
        X = r(n, 3) * 4.0 - 2.0
        return X, lambda rows, K: torch.rand(rows.numel(), n_cams, generator=u, device=dev).argsort(1)[:, :K]
    if scene == "street":
        L = n_cams * 3.0
        X = torch.stack([5.0 + r(n) * (L - 3.0 + 105.0), r(n) * 10.0, r(n) * 20.0 - 10.0], 1)

        def props(rows, K):
            hi = torch.floor((X[rows, 0] - 5.0) / 3.0).long()
            return (hi[:, None] - ints(0, 35, rows.numel(), K)).clamp(0, n_cams - 1)
        return X, props
    if scene == "aerial":
        lo, hi = C.amin(0), C.amax(0)
        px, pz = lo[0] + r(n) * (hi[0] - lo[0]), lo[2] + r(n) * (hi[2] - lo[2])
        y = (8.0 * torch.sin(px / 170.0) * torch.cos(pz / 230.0) + 5.0 * torch.sin(px / 61.0 + 1.3) * torch.sin(pz / 83.0)
             + 2.0 * torch.cos(px / 23.0 - pz / 31.0) + 15.0)
        X = torch.stack([px, y, pz], 1)

        def props(rows, K):
            ix = torch.round(X[rows, 0] / geo["sp"]).long()[:, None] + ints(-2, 3, rows.numel(), K)
            iy = torch.round(X[rows, 2] / geo["sp"]).long()[:, None] + ints(-2, 3, rows.numel(), K)
            return (iy.clamp(0, geo["ny"] - 1) * geo["nx"] + ix.clamp(0, geo["nx"] - 1)).clamp(0, n_cams - 1)
        return X, props
    cc = torch.as_tensor(geo["centers"], device=dev)
    nbr = torch.as_tensor(geo["nbr"], device=dev)
    home = ints(0, cc.shape[0], n)
    X = cc[home] + torch.stack([r(n) * 60.0 - 30.0, r(n) * 20.0, r(n) * 60.0 - 30.0], 1)
    inter = r(n) < 0.2

    def props(rows, K):
        m = rows.numel()
        own = home[rows, None] * CITY_CLUSTER + ints(0, CITY_CLUSTER, m, K)
        oc = nbr[home[rows], ints(0, 8, m)]
        oth = oc[:, None] * CITY_CLUSTER + ints(0, CITY_CLUSTER, m, K)
        return torch.where(inter[rows, None] & (torch.rand(m, K, generator=u, device=dev) < 0.3), oth, own)
    return X, props


def _scene(scene, n_cams, n_pts, seed, perturb_cameras=True):
    """A seeded scene as a Block (host arrays, as InputBlock leaves them)."""
    rng = np.random.default_rng(seed)
    u = torch.Generator(device="cuda").manual_seed(seed)
    Rn, Cn, fn, kn, geo = _cameras(scene, n_cams, rng)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
    R, C, f, k = dev(Rn), dev(Cn), dev(fn), dev(kn)
    t = -torch.einsum("nij,nj->ni", R, C)
    n_drawn = n_pts + n_pts // 8 + 16  # some points are seen less than twice
    X, props = _points(scene, n_cams, n_drawn, geo, C, u)
    # geometric track lengths from 2 on
    p = 1.0 / (TRACK_MEAN[scene] - 2 + 1.0)
    want = 2 + torch.floor(torch.log(torch.rand(n_drawn, generator=u, device="cuda", dtype=torch.float64).clamp_min(1e-12))
                           / math.log(1.0 - p)).long()
    want = want.clamp_max(min(_MAX_TRACK[scene], n_cams))
    cams, pts = [], []
    # short tracks need few proposals; the rows of a chunk are drawn together
    short = 12
    for rows_all, K in ((torch.nonzero(want <= short).flatten(), 3 * short), (torch.nonzero(want > short).flatten(),
                                                                              3 * _MAX_TRACK[scene] // 2)):
        K = min(K, n_cams) if scene == "arc" else K
        for s in range(0, rows_all.numel(), 400_000):
            rows = rows_all[s:s + 400_000]
            prop = props(rows, K)
            _, pz, pinf = _project(R, t, f, k, X[rows, None, :].expand(-1, prop.shape[1], -1), prop)
            vis = (pz < -_MIN_DEPTH[scene]) & (pinf < _MAX_P[scene])
            sp, order = torch.sort(prop, dim=1, stable=True)
            first = torch.ones_like(vis)
            first[:, 1:] = sp[:, 1:] != sp[:, :-1]
            keep = torch.zeros_like(vis).scatter_(1, order, first) & vis
            take = keep & (keep.cumsum(1) <= want[rows, None])
            take &= (take.sum(1) >= 2)[:, None]
            i, j = torch.nonzero(take, as_tuple=True)
            cams.append(prop[i, j])
            pts.append(rows[i])
    cam, pt = torch.cat(cams), torch.cat(pts)
    key, _ = torch.sort(pt * n_cams + cam)  # point major, cameras ascending in a track
    cam, pt = key % n_cams, key // n_cams
    # the case's number of points and of observations: the first n_pts points
    # seen twice, and the last observation of as many longer tracks as needed dropped
    used = torch.zeros(n_drawn, dtype=torch.bool, device="cuda")
    used[pt] = True
    new_id = used.cumsum(0) - 1
    keep = new_id[pt] < n_pts
    cam, pt = cam[keep], new_id[pt[keep]]
    X = X[used][:n_pts]
    n_obs = _observations(scene, n_cams, n_pts)
    while cam.numel() > n_obs:
        length = torch.bincount(pt, minlength=n_pts)
        long = torch.nonzero(length > 2).flatten()
        long = long[torch.randperm(long.numel(), generator=u, device="cuda")[:cam.numel() - n_obs]]
        stay = torch.ones_like(cam, dtype=torch.bool)
        stay[length.cumsum(0)[long] - 1] = False
        cam, pt = cam[stay], pt[stay]
    no = cam.numel()
    if no != n_obs or X.shape[0] != n_pts:
        raise RuntimeError(f"the scene has {X.shape[0]} points and {no} observations, not {n_pts} and {n_obs}")
    xy = torch.empty(no, 2, dtype=torch.float64, device="cuda")
    for s in range(0, no, 4_000_000):
        e = min(no, s + 4_000_000)
        xy[s:e] = _project(R, t, f, k, X[pt[s:e]], cam[s:e])[0]
    xy += 0.5 * torch.randn(no, 2, generator=u, device="cuda", dtype=torch.float64)
    out = torch.rand(no, generator=u, device="cuda") < _OUTLIERS[scene]
    xy += out[:, None] * (torch.rand(no, 2, generator=u, device="cuda", dtype=torch.float64) * 100.0 - 50.0)
    # start state
    if perturb_cameras:
        Rn = np.einsum("nij,njk->nik", scenes.small_rotation(rng, n_cams, 0.01), Rn)
        Cn = Cn + rng.normal(scale=0.05 / math.sqrt(3.0), size=Cn.shape)
        fn = fn * (1.0 + rng.normal(scale=0.02, size=n_cams))
    X = X + (0.05 / math.sqrt(3.0)) * torch.randn(X.shape, generator=u, device="cuda", dtype=torch.float64)
    # the block
    pmat = np.zeros((n_cams, 3, 4), np.float32)
    pmat[:, :, :3] = Rn
    pmat[:, :, 3] = -np.einsum("nij,nj->ni", Rn, Cn)
    K = np.zeros((n_cams, 3, 3), np.float32)
    K[:, 0, 0] = K[:, 1, 1] = fn
    K[:, 2, 2] = 1.0
    _, order = torch.sort(cam, stable=True)
    img_off = torch.zeros(n_cams + 1, dtype=torch.long, device="cuda")
    img_off[1:] = torch.bincount(cam, minlength=n_cams).cumsum(0)
    slot = torch.empty_like(cam)
    slot[order] = torch.arange(no, device="cuda") - img_off[cam[order]]
    pt_off = torch.zeros(X.shape[0] + 1, dtype=torch.long, device="cuda")
    pt_off[1:] = torch.bincount(pt, minlength=X.shape[0]).cumsum(0)
    i32 = lambda a: a.to(torch.int32).cpu().numpy()
    one = np.ones(no, np.float32)
    return Block(pmat.reshape(n_cams, 12), K.reshape(n_cams, 9), kn.astype(np.float32),
                 X.to(torch.float32).cpu().numpy(), i32(img_off), (-xy[order]).to(torch.float32).cpu().numpy(), one,
                 one.copy(), np.zeros(no, np.float32), i32(pt_off), i32(cam), i32(slot))


# -------------------------------------------------------------------- cases

_CHANGED = ("pmat", "K", "distpara", "XX", "pt_obs_off", "pt_obs_image", "pt_obs_slot")


def _pinned_like(b):
    """A block that receives results in page-locked arrays."""
    pin = lambda a: torch.zeros(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True).numpy()
    return Block(*(pin(getattr(b, n)) if n in _CHANGED else getattr(b, n)
                   for n in ("pmat", "K", "distpara", "XX", "img_obs_off", "xg", "wx", "wy", "wxy", "pt_obs_off",
                             "pt_obs_image", "pt_obs_slot")))


def _work_copy(b):
    """A block that CalcPLSA may change, the constant arrays shared."""
    return Block(*(getattr(b, n).copy() if n in _CHANGED else getattr(b, n)
                   for n in ("pmat", "K", "distpara", "XX", "img_obs_off", "xg", "wx", "wy", "wxy", "pt_obs_off",
                             "pt_obs_image", "pt_obs_slot")))


def _out(b):
    return {n: getattr(b, n) for n in _CHANGED}


def prepare(case, seed):
    op = case["op"]
    s = {"case": case}
    if op == "batch":
        # camera counts spread over the case's range, shuffled
        m, span = case["scenes"], case["cmax"] - case["cmin"]
        s["blocks"] = []
        for i in range(m):
            n = case["cmin"] + (span * ((7 * i) % m)) // max(m - 1, 1)
            s["blocks"].append(_scene("arc", n, 150 * n, seed * 1000 + i))
        return s
    b = s["block"] = _scene(case["scene"], case["cams"], case["points"], seed,
                            perturb_cameras=op not in ("triangulate",))
    if op == "solve":
        S = s["solver"] = rb.Solver(b, robust=case["robust"], k2=case["k2"], k4=case["k4"], f=case["f"],
                                    solver=SOLVERS[case["solver"]], precision=PRECISIONS[case["precision"]],
                                    pcg_tolerance=case["tol"])
        if case["solver"] == "learned":
            S.set_preconditioner(train_precond.load())
        s["out"] = _pinned_like(b)
    elif op == "triangulate":
        # the images' thresholds of a refined scene: 1 / (2.1981 median |r|^2), noise 0.5 px
        s["sig0w"] = np.full(b.n_images, 1.3, np.float32)
        if case["parts"]:
            s["part"] = rb.partition_images(b, case["parts"])
    elif op == "partitioned":
        s["part"] = rb.partition_images(b, case["parts"])
    return s


def run(s):
    case, op = s["case"], s["case"]["op"]
    if op == "solve":
        st, rep = s["solver"].solve()
        return {"status": st, **_out(s["solver"].state(out=s["out"])), "sigma0": np.float32(rep["sigma0_out"]),
                "rms": rep["rms"]}
    if op == "call":
        b = _work_copy(s["block"])
        st, _, rep = rb.CalcPLSA(b, robust=case["robust"], addflags=(case["k2"], case["k4"], case["f"]),
                                 solver=SOLVERS[case["solver"]], precision=PRECISIONS[case["precision"]])
        return {"status": st, **_out(b), "sigma0": np.float32(rep["sigma0_out"]), "rms": rep["rms"]}
    if op == "batch":
        bs = [_work_copy(b) for b in s["blocks"]]
        st, reps, _ = rb.solve_batch(bs, workers=case["workers"], robust=case["robust"],
                                     solver=SOLVERS[case["solver"]], precision=PRECISIONS[case["precision"]])
        outs = [_out(b) for b in bs]
        return {"status": np.array(st), "rms": np.float32([r["rms"] for r in reps]),
                **{k: np.concatenate([o[k] for o in outs]) for k in outs[0]}}
    if op == "partitioned":
        st, b, stats, _ = rb.calc_plsa_parallel(s["block"], s["part"], case["parts"])
        out = {"status": st, **_out(b), "sig0opt": stats["sig0opt"]}
        for n in ("pt_obs_image", "pt_obs_slot"):  # the tracks come trimmed to what was kept
            out[n] = np.zeros_like(getattr(s["block"], n))
            out[n][:getattr(b, n).size] = getattr(b, n)
        return out
    if op == "triangulate":
        w = s["sig0w"] if case["mode"] == 2 else None
        if case["parts"]:
            return rb.triangulate_parts(s["block"], s["part"], case["parts"], sig0w=w, robustmode=case["mode"])
        return rb.triangulate(s["block"], sig0w=w, robustmode=case["mode"])
    with rb.Solver(s["block"], exteval=True) as S:
        r, rep = S.exteval()
    return {"resid": r, "sigma0": np.float32(rep["exteval_sigma0"]), "nrobs": rep["exteval_nrobs"],
            "redundancy": rep["exteval_redundancy"]}


def work(case):
    op = case["op"]
    if op == "batch":
        cams = case["scenes"] * (case["cmin"] + case["cmax"]) / 2
        pts = 150 * cams
    else:
        cams, pts = case["cams"], case["points"]
    obs = _observations(case["scene"], cams, pts)
    t = obs / pts
    # the block in (20 B of xg and weights, 8 B of track entry per
    # observation; 16 B a point; 92 B a camera) and the changed part out
    block = 28 * obs + 16 * pts + 92 * cams
    changed = 8 * obs + 16 * pts + 92 * cams
    if op == "exteval":
        return {"bytes": block + 16 * obs, "flops": 50 * obs}
    if op == "triangulate":
        return {"bytes": block + 24 * pts + 5 * obs + pts + 24 * pts * case["parts"], "flops": 4 * 150 * obs}
    # at least two linearisations: Jacobians, the point elimination and the
    # pair products (a track of t observations has about t^2 of them with the
    # geometric spread of the lengths)
    return {"bytes": block + changed, "flops": 2 * (400 * obs + 400 * obs * t)}


def exact(case, seed):
    if case["op"] != "exteval":
        return None  # an iteration's result has no closed 64-bit value
    b = _scene(case["scene"], case["cams"], case["points"], seed)
    g = lambda a: torch.as_tensor(a, device="cuda").double()
    n = b.n_obs
    im = torch.as_tensor(b.pt_obs_image[:n], device="cuda").long()
    pt = torch.repeat_interleave(torch.arange(b.n_points, device="cuda"),
                                 torch.as_tensor(np.diff(b.pt_obs_off), device="cuda").long())
    P = g(b.pmat).reshape(-1, 3, 4)[im]
    h = torch.einsum("nij,nj->ni", P[:, :, :3], g(b.XX)[pt]) + P[:, :, 3]
    z = h[:, 2]
    inv = torch.where(z.abs() < 1e-3, torch.where(z > 0, 1e3, -1e3).double(), 1.0 / z)
    p = h[:, :2] * inv[:, None]
    r2 = (p * p).sum(1)
    d = g(b.distpara)[im]
    p = p * ((1.0 + d[:, 0] * r2 + d[:, 1] * r2 * r2) * g(b.K)[im, 0])[:, None]
    sl = torch.as_tensor(b.track_slots(), device="cuda").long()
    return {"resid": g(b.xg)[sl] - p, "sigma0": None, "nrobs": None, "redundancy": None}
