"""Performance cases: the work that a user of the framework has it do.

Each case goes through the package's public entry points with host arrays in
and host arrays out, as a sparse-stage caller uses them: whole bundle
adjustments in both precision forms (the smallest survey to a large oblique
one, and a batch of models), one round of the sparse stage on a device
context, the adjoint, triangulation, RANSAC, the pair check and the summary.

``listed()`` are the named cases, ``draw(rng)`` gives more of the same ranges.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "aerial-3d-model_gb300"))

import stitch_ba  # noqa: E402
from stitch_ba import Context, Options, Problem, Tracks, survey  # noqa: E402


def listed():
    return [
        # The reference's own test is a 12-camera block: the smallest survey
        # that is adjusted in earnest.  Launches and latency are all there is.
        dict(name="solve_fp64_12", kind="solve", form="fp64", cams=12, points=1501, loss="cauchy",
             groups=1, refine=True, pcg="stored", oblique=0.0, iters=60),
        # An ordinary flight (77 photos), the library's defaults: the drop-in
        # for the reference's bundle_adjust.
        dict(name="solve_fp64_77", kind="solve", form="fp64", cams=77, points=40_000,
             loss="cauchy", groups=1, refine=True, pcg="stored", oblique=0.0, iters=60),
        # A large flight in the parity form.
        dict(name="solve_fp64_500", kind="solve", form="fp64", cams=500, points=400_000,
             loss="cauchy", groups=1, refine=True, pcg="stored", oblique=0.0, iters=60),
        # The same survey in the fast form, with the settings that the
        # integration notes give for it: the benchmark's workload.
        dict(name="solve_mixed_500", kind="solve", form="mixed", cams=500, points=400_000,
             loss="cauchy", groups=1, refine=True, pcg="stored", oblique=0.0, iters=60),
        # The largest single model here: nadir rows and an oblique ring.
        dict(name="solve_mixed_1200", kind="solve", form="mixed", cams=1200, points=1_000_003,
             loss="cauchy", groups=1, refine=True, pcg="stored", oblique=0.3, iters=60),
        # Many models of uneven size in one call.
        dict(name="batch_mixed_32", kind="batch", models=32, cams_lo=20, cams_hi=400),
        # One round of the sparse stage on a context: triangulate and gate the
        # tracks, build the problem, solve it, read it back, summarise it.
        dict(name="round_fp64_77", kind="round", cams=77, points=40_000, thr=10.0),
        # Backward: gradient of the cost for the intrinsics, and a VJP.
        dict(name="adjoint_500", kind="adjoint", cams=500, points=400_000, loss="cauchy"),
        # Triangulation and gating of a large flight's tracks.
        dict(name="triangulate_400k", kind="triangulate", cams=500, points=400_000, thr=10.0),
        # Match verification: 8-point RANSAC of the photo pairs of a flight.
        dict(name="ransac_150", kind="ransac", cams=150, points=90_000, iters=600),
        # Pair check of a larger flight under its poses.
        dict(name="pair_fits_300", kind="pair_fits", cams=300, points=180_000),
        # Fields of cameras.json and the points of sparse.ply.
        dict(name="summary_500", kind="summary", cams=500, points=400_000, neighbours=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "round", "adjoint", "triangulate",
                       "ransac", "pair_fits", "summary"])
    loss = rng.choice(["cauchy", "cauchy", "huber"])
    if kind == "solve":
        form = rng.choice(["fp64", "mixed"])
        cams = _log(rng, 8, 220) if form == "fp64" else _log(rng, 40, 1000)
        points = int(cams * rng.uniform(150, 800))
        pcg = "matrix_free" if form == "mixed" and cams < 400 and rng.random() < 0.15 else "stored"
        groups = rng.choice([1, 1, 1, 2]) if pcg == "stored" and cams <= 90 else 1
        iters = 60 if form == "mixed" else rng.choice([10, 20])
        return dict(kind=kind, form=form, cams=cams, points=points, loss=loss, groups=groups,
                    refine=rng.random() < 0.8, pcg=pcg, oblique=rng.choice([0.0, 0.0, 0.3]),
                    iters=iters)
    if kind == "batch":
        return dict(kind=kind, models=_log(rng, 3, 32), cams_lo=20, cams_hi=_log(rng, 40, 300))
    if kind == "round":
        cams = _log(rng, 16, 200)
        return dict(kind=kind, cams=cams, points=int(cams * rng.uniform(150, 700)),
                    thr=rng.choice([6.0, 10.0, 20.0]))
    if kind == "adjoint":
        cams = _log(rng, 20, 500)
        return dict(kind=kind, cams=cams, points=int(cams * rng.uniform(150, 800)), loss=loss)
    if kind == "triangulate":
        cams = _log(rng, 20, 500)
        return dict(kind=kind, cams=cams, points=int(cams * rng.uniform(150, 800)),
                    thr=rng.choice([4.0, 10.0, 40.0]))
    if kind == "ransac":
        cams = _log(rng, 12, 150)
        return dict(kind=kind, cams=cams, points=int(cams * rng.uniform(200, 600)),
                    iters=rng.choice([200, 600, 600]))
    if kind == "pair_fits":
        cams = _log(rng, 16, 300)
        return dict(kind=kind, cams=cams, points=int(cams * rng.uniform(150, 600)))
    cams = _log(rng, 12, 500)
    return dict(kind="summary", cams=cams, points=int(cams * rng.uniform(100, 800)),
                neighbours=rng.choice([8, 8, 5, 16]))


# ---- inputs -------------------------------------------------------------------

SIGMA = 1.0   # px, the surveys' loss scale
VIEWS_MAX, PAIRS_MAX = 16, 48   # capacity of an output, per point


def _params(case, seed, **kw):
    obl = case.get("oblique", 0.0)
    base = survey.PRESETS["oblique2000" if obl else "single500"]
    d = dict(seed=seed % (1 << 31) + 1, n_cams=case["cams"], n_points=case["points"],
             oblique_frac=obl, refine_intrinsics=case.get("refine", True))
    d.update(kw)
    return base, d


def _survey(case, seed, **kw):
    base, d = _params(case, seed, **kw)
    p, truth = survey.generate(base, **d)
    g = case.get("groups", 1)
    if g > 1:  # several lenses on one flight: the cameras take turns
        p = Problem(intr=np.repeat(p.intr, g, 0), rot=p.rot, center=p.center,
                    cam_group=np.arange(p.n_cams, dtype=np.uint32) % g, points=p.points,
                    obs_cam=p.obs_cam, obs_pt=p.obs_pt, obs_uv=p.obs_uv,
                    prior_mask=p.prior_mask, prior=p.prior,
                    refine_intrinsics=p.refine_intrinsics)
    return p, truth


def _refined(case, seed):
    """A survey whose poses an earlier round has brought close."""
    return _survey(case, seed, rot_perturb_deg=0.02, centre_perturb_m=0.05, f_scale_init=1.001)


def _tracks(p):
    cnt = np.bincount(p.obs_pt, minlength=p.n_points)
    ptr = np.concatenate([[0], np.cumsum(cnt)]).astype(np.uint32)
    return Tracks(ptr, p.obs_cam, p.obs_uv, p.cam_group, p.n_groups)


def _mixed(cams, **kw):
    """The fast form's settings (integration notes): two-level PCG, 40
    iterations per step (60 above 1000 cameras), 100 in the end game."""
    return Options(precision="mixed", coarse=True, pcg_max_iter=40 if cams <= 1000 else 60,
                   stop_patience=2, pcg_end_max_iter=100, pcg_end_rel=1e-5, **kw)


class _Solve:
    """A problem and a copy of its initial state: every pass adjusts it anew."""

    def __init__(self, p):
        self.p = p
        self.start = p.state()

    def again(self):
        self.p.set_state(self.start)
        return self.p


def prepare(case, seed):
    k = case["kind"]
    if k == "solve":
        p, _ = _survey(case, seed)
        if case["form"] == "fp64":
            opt = Options(loss=case["loss"])
        else:
            opt = _mixed(case["cams"], loss=case["loss"], matrix_free=case["pcg"])
        return dict(kind=k, solve=_Solve(p), opt=opt, iters=case["iters"])
    if k == "batch":
        rs = np.random.default_rng(case["models"])   # sizes are the case's, the surveys the seed's
        ps = []
        for m in range(case["models"]):
            nc = int(rs.integers(case["cams_lo"], case["cams_hi"] + 1))
            per_cam = int(rs.integers(500, 1001))
            ps.append(survey.generate("single500", seed=(seed + 7919 * m) % (1 << 31) + 1,
                                      n_cams=nc, n_points=max(50, math.ceil(nc * per_cam / 6.5)))[0])
        # One buffer per state array, a slice of it per model.
        flat = {f: np.concatenate([getattr(p, f) for p in ps]) for f in
                ("rot", "center", "intr", "points")}
        for f, a in flat.items():
            at = 0
            for p in ps:
                n = len(getattr(p, f))
                setattr(p, f, a[at:at + n])
                at += n
        opt = _mixed(case["cams_hi"], pcg_kernel="cluster")
        return dict(kind=k, problems=ps, flat=flat, start={f: a.copy() for f, a in flat.items()},
                    opt=opt)
    if k == "round":
        p, _ = _refined(case, seed)
        return dict(kind=k, p=p, tracks=_tracks(p), thr=case["thr"], ctx=Context(),
                    points=np.zeros((p.n_points, 3)),
                    points_f32=np.zeros((p.n_points, 3), np.float32))
    if k == "adjoint":
        p, _ = _survey(case, seed)
        ctx = Context()
        ctx.upload(p)
        rng = np.random.default_rng(seed)
        return dict(kind=k, p=p, ctx=ctx, opt=Options(loss=case["loss"]),
                    cot=rng.standard_normal((p.n_obs, 2)),
                    cot_prior=rng.standard_normal((p.n_cams, 3)))
    if k == "triangulate":
        p, _ = _refined(case, seed)
        return dict(kind=k, p=p, tracks=_tracks(p), thr=case["thr"],
                    good=np.zeros(VIEWS_MAX * case["points"], bool))
    if k in ("ransac", "pair_fits"):
        p, _ = _refined(case, seed)
        pairs = survey.pair_matches(p, seed=seed)
        cap = p.n_cams * (p.n_cams - 1) // 2
        return dict(kind=k, p=p, pairs=pairs, iters=case.get("iters", 600),
                    inlier=np.zeros(PAIRS_MAX * case["points"], bool), median=np.zeros(cap),
                    per_pair=np.zeros((3, cap), np.int32))
    p, _ = _refined(case, seed)
    return dict(kind="summary", p=p, neighbours=case["neighbours"])


# ---- one pass -----------------------------------------------------------------

# The number of observations, matches or LM iterations depends on the seed: where
# an output has one value for each, it stands at the front of a buffer of the
# case's capacity, with zeros after it.

def _front(buffer, values):
    buffer[:len(values)] = values
    buffer[len(values):] = 0
    return buffer


def _state_of(p):
    return dict(rot=p.rot, center=p.center, intr=p.intr, points=p.points)


def run(state):
    k = state["kind"]
    if k == "solve":
        p = state["solve"].again()
        st, info = stitch_ba.bundle_adjust(p, state["iters"], SIGMA, state["opt"],
                                            return_info=True)
        return dict(_state_of(p), iterations=st.iterations, initial_rms=st.initial_rms,
                    final_rms=st.final_rms, final_cost=info.final_cost,
                    trial_costs=_front(np.zeros(state["iters"]), info.new_cost),
                    accepted=_front(np.zeros(state["iters"], bool), info.accepted))
    if k == "batch":
        for f, a in state["start"].items():
            np.copyto(state["flat"][f], a)
        infos = stitch_ba.bundle_adjust_batch(state["problems"], 60, SIGMA, state["opt"])
        return dict(state["flat"], iterations=np.array([i.iterations for i in infos]),
                    initial_rms=np.array([i.initial_rms for i in infos]),
                    final_cost=np.array([i.final_cost for i in infos]))
    if k == "round":
        p, ctx, thr = state["p"], state["ctx"], state["thr"]
        n_pts, n_obs = ctx.upload_tracks(state["tracks"], p.rot, p.center, p.intr, thr,
                                         prior_mask=p.prior_mask, prior=p.prior)
        info = ctx.solve(20, thr / 2.0)[0]
        out = Problem.empty(p.n_cams, n_pts, n_obs, p.n_groups)
        ctx.download(out)
        s = ctx.sparse_summary(80.0)
        return dict(rot=out.rot, center=out.center, intr=out.intr,
                    points=_front(state["points"], out.points), n_points=n_pts, n_obs=n_obs,
                    iterations=info.iterations, final_rms=info.final_rms,
                    neighbours=s.neighbours, shared=s.shared, depth_range=s.depth_range,
                    points_f32=_front(state["points_f32"], s.points_f32))
    if k == "adjoint":
        ctx = state["ctx"]
        grad = ctx.intrinsics_grad(SIGMA, state["opt"])
        gc, gp, gi = ctx.vjp(SIGMA, state["cot"], state["cot_prior"], state["opt"])
        return dict(grad=grad, cameras=gc, points=gp, intrinsics=gi)
    if k == "triangulate":
        p = state["p"]
        kept, points, good = stitch_ba.triangulate(state["tracks"], p.rot, p.center, p.intr,
                                                   state["thr"])
        return dict(kept=kept, points=points, good=_front(state["good"], good))
    if k == "ransac":
        inlier, n, best, refit = stitch_ba.ransac_fundamental(state["pairs"], 1.5, state["iters"])
        for row, values in zip(state["per_pair"], (n, best, refit)):
            _front(row, values)
        return dict(inlier=_front(state["inlier"], inlier), per_pair=state["per_pair"])
    if k == "pair_fits":
        p = state["p"]
        return dict(median=_front(state["median"], stitch_ba.pair_fits(
            state["pairs"], p.rot, p.center, p.intr, p.cam_group)))
    s = stitch_ba.sparse_summary(state["p"], 80.0, state["neighbours"])
    return dict(neighbours=s.neighbours, shared=s.shared, count=s.n_neighbours,
                depth_range=s.depth_range, points_f32=s.points_f32)


# ---- what a pass cannot do without ----------------------------------------------

VIEWS = 7.4       # observations per point of these surveys
PAIR_SHARE = 30   # co-observations (camera pairs) per point
LM_ITERS = 12


def work(case):
    k = case["kind"]
    if k == "batch":
        cams = case["models"] * (case["cams_lo"] + case["cams_hi"]) / 2
        points = cams * 750 / 6.5
    else:
        cams, points = case["cams"], case["points"]
    obs = points * VIEWS
    problem = 24.0 * obs + 24.0 * points + 200.0 * cams   # observations, points, cameras
    state = 24.0 * points + 96.0 * cams
    if k in ("solve", "batch", "round"):
        # linearisation and sums per observation, 6x3 by 3x6 per camera pair
        flops = LM_ITERS * (obs * 700.0 + points * (PAIR_SHARE + VIEWS) * 216.0)
        return dict(bytes=problem + state, flops=flops)
    if k == "adjoint":
        return dict(bytes=2 * problem + 16.0 * obs + state, flops=2 * obs * 250.0)
    if k == "triangulate":
        return dict(bytes=problem + 25.0 * points + obs, flops=obs * 350.0 + points * 1500.0)
    matches = points * PAIR_SHARE
    if k == "ransac":
        return dict(bytes=33.0 * matches, flops=case["iters"] * (matches * 30.0 + cams * 10 * 1500.0))
    if k == "pair_fits":
        return dict(bytes=32.0 * matches, flops=matches * 250.0)
    return dict(bytes=8.0 * obs + 24.0 * points + 12.0 * points + 96.0 * cams, flops=obs * 10.0)


# ---- the same results in plain numpy, 64 bits -------------------------------------

def _linearise(p):
    """Per observation: residual e (n, 2), Jacobians of the prediction for the
    camera (rotation as a left perturbation, centre), the point and the
    intrinsics (f, cx, cy, k1, k2), and whether the point is in front."""
    R, K = p.rot[p.obs_cam], p.intr[p.cam_group[p.obs_cam]]
    xc = np.einsum("nij,nj->ni", R, p.points[p.obs_pt] - p.center[p.obs_cam])
    front = xc[:, 2] > 1e-6
    z = np.where(front, xc[:, 2], 1.0)
    px, py = xc[:, 0] / z, xc[:, 1] / z
    f, k1, k2 = K[:, 0], K[:, 3], K[:, 4]
    r2 = px * px + py * py
    d = 1.0 + k1 * r2 + k2 * r2 * r2
    e = p.obs_uv - np.stack([f * d * px + K[:, 1], f * d * py + K[:, 2]], 1)
    c = 2.0 * (k1 + 2.0 * k2 * r2)
    A = np.empty((len(z), 2, 2))
    A[:, 0, 0], A[:, 1, 1] = f * (d + c * px * px), f * (d + c * py * py)
    A[:, 0, 1] = A[:, 1, 0] = f * c * px * py
    B = np.zeros((len(z), 2, 3))
    B[:, 0, 0] = B[:, 1, 1] = 1.0 / z
    B[:, 0, 2], B[:, 1, 2] = -px / z, -py / z
    du = A @ B
    S = np.zeros((len(z), 3, 3))
    S[:, 0, 1], S[:, 0, 2], S[:, 1, 2] = -xc[:, 2], xc[:, 1], -xc[:, 0]
    S -= S.transpose(0, 2, 1)
    Jp = du @ R
    Jc = np.concatenate([-du @ S, -Jp], 2)
    Ji = np.zeros((len(z), 2, 5))
    Ji[:, 0, 0], Ji[:, 1, 0] = px * d, py * d
    Ji[:, 0, 1] = Ji[:, 1, 2] = 1.0
    Ji[:, 0, 3], Ji[:, 1, 3] = f * px * r2, f * py * r2
    Ji[:, 0, 4], Ji[:, 1, 4] = f * px * r2 * r2, f * py * r2 * r2
    for J in (Jc, Jp, Ji):
        J[~front] = 0.0
    return e, Jc, Jp, Ji, front


def _sum_by(index, values, n):
    return np.stack([np.bincount(index, values[:, i], n) for i in range(values.shape[1])], 1)


def _exact_adjoint(case, seed):
    p, _ = _survey(case, seed)
    rng = np.random.default_rng(seed)
    cot, cot_prior = rng.standard_normal((p.n_obs, 2)), rng.standard_normal((p.n_cams, 3))
    e, Jc, Jp, Ji, front = _linearise(p)
    e2 = (e * e).sum(1)
    if case["loss"] == "huber":
        a = np.sqrt(e2)
        w = np.where(a <= SIGMA, 1.0, SIGMA / np.maximum(a, 1e-300))
    else:
        w = 1.0 / (1.0 + e2 / SIGMA**2)
    lam = np.where(front[:, None], 2.0 * w[:, None] * e, 0.0)
    grp = p.cam_group[p.obs_cam].astype(np.int64)
    grad = _sum_by(grp, -np.einsum("nri,nr->ni", Ji, lam), p.n_groups)
    gc = _sum_by(p.obs_cam, -np.einsum("nri,nr->ni", Jc, cot), p.n_cams)
    gc[:, 3:] += np.where(p.prior_mask[:, None] != 0, cot_prior / p.prior[:, 3:], 0.0)
    return dict(grad=grad, cameras=gc,
                points=_sum_by(p.obs_pt, -np.einsum("nri,nr->ni", Jp, cot), p.n_points),
                intrinsics=_sum_by(grp, -np.einsum("nri,nr->ni", Ji, cot), p.n_groups))


def _undistort(K, uv):
    q = (uv - K[:, 1:3]) / K[:, :1]
    x = q.copy()
    for _ in range(8):
        r2 = (x * x).sum(1)
        x = q / (1.0 + K[:, 3] * r2 + K[:, 4] * r2 * r2)[:, None]
    return x


def _exact_triangulate(case, seed):
    p, _ = _refined(case, seed)
    n = p.n_points
    K = p.intr[p.cam_group[p.obs_cam]]
    x = _undistort(K, p.obs_uv)
    Pm = np.concatenate([p.rot, -(p.rot @ p.center[:, :, None])], 2)[p.obs_cam]
    rows = x[:, :, None] * Pm[:, 2:3] - Pm[:, :2]
    M = np.einsum("nri,nrj->nij", rows, rows).reshape(-1, 16)
    M = _sum_by(p.obs_pt, M, n).reshape(n, 4, 4)
    v = np.linalg.eigh(M)[1][:, :, 0]
    cnt = np.bincount(p.obs_pt, minlength=n)
    ok = (cnt >= 2) & (np.abs(v[:, 3]) >= 1e-12)
    X = np.where(ok[:, None], v[:, :3] / np.where(ok, v[:, 3], 1.0)[:, None], 0.0)
    C = p.center[p.obs_cam]
    xc = np.einsum("nij,nj->ni", p.rot[p.obs_cam], X[p.obs_pt] - C)
    front = xc[:, 2] > 1e-6
    y = xc[:, :2] / np.where(front, xc[:, 2], 1.0)[:, None]
    r2 = (y * y).sum(1)
    u = K[:, :1] * (1.0 + K[:, 3] * r2 + K[:, 4] * r2 * r2)[:, None] * y + K[:, 1:3]
    good = ok[p.obs_pt] & front & (np.sqrt(((u - p.obs_uv) ** 2).sum(1)) < case["thr"])
    ray = X[p.obs_pt] - C
    ray /= np.linalg.norm(ray, axis=1)[:, None]
    first = np.concatenate([[0], np.cumsum(cnt)])
    least = np.ones(n)
    for m in np.unique(cnt[cnt >= 2]):
        t = np.nonzero(cnt == m)[0]
        at = first[t][:, None] + np.arange(m)
        r, g = ray[at], good[at]
        dot = np.einsum("tia,tja->tij", r, r)
        dot[~(g[:, :, None] & g[:, None, :])] = 1.0
        least[t] = np.minimum(dot.reshape(len(t), -1).min(1), 1.0)
    ng = np.bincount(p.obs_pt, good, n)
    deg = np.degrees(np.arccos(np.maximum(least, -1.0)))
    kept = (ng >= 2) & np.where(ng >= 3, deg > 2.0, deg > 6.0)
    return dict(kept=None, points=np.where(kept[:, None], X, 0.0), good=None)


def _exact_pair_fits(case, seed):
    p, _ = _refined(case, seed)
    q = survey.pair_matches(p, seed=seed)
    ptr = q.match_ptr.astype(np.int64)
    med = np.full(len(ptr) - 1, np.finfo(np.float64).max)
    for k, (a, b) in enumerate(q.pair_cam.astype(np.int64)):
        uv = q.uv[ptr[k]:ptr[k + 1]]
        if len(uv) == 0:
            continue
        Ka, Kb = p.intr[p.cam_group[a]], p.intr[p.cam_group[b]]
        x1 = np.column_stack([_undistort(np.repeat(Ka[None], len(uv), 0), uv[:, :2]),
                              np.ones(len(uv))])
        x2 = np.column_stack([_undistort(np.repeat(Kb[None], len(uv), 0), uv[:, 2:]),
                              np.ones(len(uv))])
        t = p.rot[b] @ (p.center[a] - p.center[b])
        E = np.array([[0, -t[2], t[1]], [t[2], 0, -t[0]], [-t[1], t[0], 0]]) @ p.rot[b] @ p.rot[a].T
        fa, gb = x1 @ E.T, x2 @ E
        e = (x2 * fa).sum(1)
        d = fa[:, 0]**2 + fa[:, 1]**2 + gb[:, 0]**2 + gb[:, 1]**2
        err = np.sqrt(np.where(d < 1e-18, np.finfo(np.float64).max, e * e / np.maximum(d, 1e-18)))
        med[k] = np.partition(err * Ka[0], len(uv) // 2)[len(uv) // 2]
    out = np.zeros(p.n_cams * (p.n_cams - 1) // 2)
    out[:len(med)] = med
    return dict(median=out)


def _exact_summary(case, seed):
    p, _ = _refined(case, seed)
    z = np.einsum("nj,nj->n", p.rot[p.obs_cam, 2], p.points[p.obs_pt] - p.center[p.obs_cam])
    out = np.tile([0.3 * 80.0, 3.0 * 80.0], (p.n_cams, 1))
    order = np.lexsort((z, p.obs_cam))
    n = np.bincount(p.obs_cam, minlength=p.n_cams)
    at = np.concatenate([[0], np.cumsum(n)])
    for c in np.nonzero(n >= 10)[0]:
        d = z[order[at[c]:at[c + 1]]]
        out[c] = d[n[c] // 20] * 0.8, d[n[c] * 19 // 20] * 1.25
    return dict(neighbours=None, shared=None, count=None, depth_range=out,
                points_f32=p.points.astype(np.float32))


def _exact_solve(case, seed):
    """A bundle adjustment stops before it has converged (its stop rule, its
    capped inner solves): only the error that it starts from has such a value."""
    p, _ = _survey(case, seed)
    e, _, _, _, front = _linearise(p)
    out = dict.fromkeys(("rot", "center", "intr", "points", "iterations", "final_rms",
                         "final_cost", "trial_costs", "accepted"))
    return dict(out, initial_rms=math.sqrt((e[front] ** 2).sum() / max(int(front.sum()), 1)))


def exact(case, seed):
    """What run() returns, in plain numpy."""
    f = dict(solve=_exact_solve, adjoint=_exact_adjoint, triangulate=_exact_triangulate,
             pair_fits=_exact_pair_fits, summary=_exact_summary).get(case["kind"])
    return f(case, seed) if f else None
