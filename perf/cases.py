"""The work that users of this framework have it do, as timed cases.

Every case goes through the public entry points the way a compiled client of
the library does: the drop-in ``pfcore_filter_update`` / ``pfcore_gl_localize``
host layer, the fused and the staged ``pfc_*`` calls, batched filters, the
``pfgl_*`` scorers and localizers and the learned proposal.  Inputs that a
client holds as C records (observations, odometry) are built once, in
``prepare``.

Filters run on a closed circle of poses, so a pass can be repeated: step k's
odometry and observations are those of the k-th pose, and after the last pose
comes the first again.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import cuda_pf_localization_b200 as pkg
from cuda_pf_localization_b200 import sim

LOOP = 256        # poses of a single filter's circle
BATCH_LOOP = 32   # poses of a batched filter's circle


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # a robot's tracker with the default particle count and a dozen landmarks, all
        # seen in every update, no gate: the smallest call, latency is all of it
        dict(name="update_4096", kind="update", n=4096, landmarks=12, nobs=0, outliers=0.0,
             box=20.0, gate=0.0, inject=0.0, mode="cart"),
        # the drop-in update at an ordinary large count, with a dense sensor suite: 256
        # observations of 64 landmarks, a tenth of them outliers
        dict(name="update_100k", kind="update", n=100003, landmarks=64, nobs=256,
             outliers=0.1, box=50.0, gate=3.0, inject=0.01, mode="cart"),
        # the benchmark's workload, observations already on the device, one fused call
        dict(name="cycle_1m", kind="cycle_device", n=1000000, landmarks=64, nobs=256,
             outliers=0.1, box=50.0, gate=3.0, inject=0.01, mode="cart"),
        # the largest filter, fused call from host observations
        dict(name="cycle_4m", kind="cycle", n=3999999, landmarks=64, nobs=256,
             outliers=0.1, box=50.0, gate=3.0, inject=0.01, mode="cart"),
        # weighting and estimate of a given cloud from range-bearing observations (radar,
        # camera bearings): the staged calls a client makes that resamples by itself
        dict(name="weigh_bearing_500k", kind="weigh", n=500009, landmarks=40, nobs=150,
             gate=3.0, mode="bearing"),
        # the same with few observations of a large map, hardly a landmark seen twice
        dict(name="weigh_sparse_200k", kind="weigh", n=200003, landmarks=500, nobs=96,
             gate=3.0, mode="cart"),
        # many robots, or many hypotheses of one: filters of uneven size in one call
        dict(name="batch_128", kind="batch", filters=128, n_min=1000, n_max=200000,
             gate=3.0, inject=0.01),
        # the drop-in global localization with its default parameters
        dict(name="localize_50k", kind="localize", hyps=50000, rays=360, span=2 * math.pi,
             topk=10, width=200, height=200, boxes=30),
        # candidate poses of a client's own scored against a 270 degree lidar's scan on a
        # map that is not square
        dict(name="score_20k_270deg", kind="score", hyps=20011, rays=271, span=1.5 * math.pi,
             topk=64, width=401, height=299, boxes=60),
        # a million poses (positions x 16 headings) through the fused localizer
        dict(name="localize_fused_1m", kind="localize_fused", hyps=1000000, rays=360,
             span=2 * math.pi, topk=64, width=200, height=200, boxes=30),
        # a thousand scans through the learned proposal, 250 samples each
        dict(name="learned_queries", kind="learned_queries", queries=1000, samples=250,
             topk=64, rays=360, batch=1024),
        # training of the proposal network, weights read back
        dict(name="learned_train", kind="learned_train", batch=8192, steps=32, pairs=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update", "cycle", "cycle_device", "weigh", "weigh", "batch", "localize",
                       "score", "localize_fused", "learned_queries", "learned_train"])
    if kind in ("update", "cycle", "cycle_device"):
        every = rng.random() < 0.3
        return dict(kind=kind, n=_log_int(rng, 1000, 2000000),
                    landmarks=_log_int(rng, 6, 32 if every else 160),
                    nobs=0 if every else _log_int(rng, 4, 256),
                    outliers=rng.choice([0.0, 0.1]), box=rng.choice([20.0, 50.0]),
                    gate=rng.choice([0.0, 3.0]), inject=rng.choice([0.0, 0.01, 0.05]),
                    mode=rng.choice(["cart", "cart", "cart", "bearing", "mixed"]))
    if kind == "weigh":
        return dict(kind=kind, n=_log_int(rng, 2000, 500000), landmarks=_log_int(rng, 6, 600),
                    nobs=_log_int(rng, 4, 200), gate=rng.choice([0.0, 3.0]),
                    mode=rng.choice(["cart", "cart", "bearing", "mixed"]))
    if kind == "batch":
        return dict(kind=kind, filters=_log_int(rng, 8, 128), n_min=1000,
                    n_max=_log_int(rng, 4000, 200000), gate=rng.choice([0.0, 3.0]),
                    inject=rng.choice([0.0, 0.01]))
    if kind in ("localize", "score", "localize_fused"):
        top = 200000 if kind != "localize_fused" else 600000
        return dict(kind=kind, hyps=_log_int(rng, 4000, top), rays=_log_int(rng, 60, 500),
                    span=rng.choice([math.pi, 1.5 * math.pi, 2 * math.pi]),
                    topk=_log_int(rng, 1, 100), width=rng.randint(120, 420),
                    height=rng.randint(120, 420), boxes=rng.randint(5, 60))
    if kind == "learned_queries":
        return dict(kind=kind, queries=_log_int(rng, 30, 1000), samples=_log_int(rng, 60, 600),
                    topk=_log_int(rng, 1, 60), rays=rng.randint(90, 384), batch=1024)
    return dict(kind=kind, batch=128 * _log_int(rng, 4, 64), steps=rng.randint(8, 32), pairs=65536)


# ------------------------------------------------------------------- filters

def _circle(case, seed):
    """A closed circle of poses with its odometry and observations."""
    n = LOOP
    nobs = case["nobs"] or None
    sc = sim.helix_scenario(n, case["landmarks"], (case["box"], case["box"], 10.0), nobs,
                            case["outliers"], seed + 1, radius=5.0, climb=0.0,
                            arc=2 * math.pi * 5.0 / n)
    if case["mode"] != "cart":
        rb = sim.as_range_bearing(sc)
        for k, st in enumerate(sc.steps):
            to_rb = np.ones(len(st.obs), bool) if case["mode"] == "bearing" \
                else np.arange(len(st.obs)) % 3 == 0
            st.obs = np.where(to_rb[:, None], rb.steps[k].obs, st.obs)
    return sc


def _odom(st, sc):
    o = pkg.PfcOdom()
    o.t[:] = list(map(float, st.odom_t))
    o.q[:] = list(map(float, st.odom_q))
    o.tstd[:] = list(sc.trans_noise)
    o.rstd[:] = list(sc.rot_noise)
    return o


class _Update:
    """``ParticleFilter::update`` of the drop-in host layer."""

    def __init__(self, case, seed):
        sc = _circle(case, seed)
        self.pf = pkg.ParticleFilter(case["n"], seed=seed + 42, resample_ess_ratio=0.5,
                                     random_inject_ratio=case["inject"],
                                     gate_sigma=case["gate"])
        self.pf.set_map(sc.landmark_dict())
        self.pf.reinitialize(np.r_[sc.prior_p, sc.prior_q], [0.3] * 3, [0.1] * 3)
        self.odom = [pkg.make_core_odom(s.odom_t, s.odom_q, sc.trans_noise, sc.rot_noise)
                     for s in sc.steps]
        self.obs = [pkg.make_core_obs(s.obs) for s in sc.steps]
        self.count = [len(s.obs) for s in sc.steps]
        self.k = 0

    def run(self):
        k, self.k = self.k, (self.k + 1) % LOOP
        est = pkg.PfcoreEstimate()
        if pkg.core().pfcore_filter_update(self.pf._h, C.byref(self.odom[k]), self.obs[k],
                                           self.count[k], C.byref(est)) != 0:
            raise RuntimeError(pkg.core().pfcore_last_error().decode())
        return pkg.estimate_dict(est)


class _Cycle:
    """The fused cycle on a raw handle, from host or device observations."""

    def __init__(self, case, seed):
        sc = _circle(case, seed)
        self.lib = pkg.kernels()
        self.h = self.lib.pfc_create(256)
        if not self.h or self.lib.pfc_init(self.h, case["n"], seed + 42) != 0:
            raise RuntimeError(pkg.last_error())
        lm = np.ascontiguousarray(sc.landmarks, np.float32).reshape(-1)
        self.lib.pfc_upload_landmarks(self.h, pkg.fptr(lm), len(sc.landmarks))
        spread = np.full(3, 0.3, np.float32), np.full(3, 0.1, np.float32)
        prior = np.r_[sc.prior_p, sc.prior_q].astype(np.float32)
        self.lib.pfc_reinit(self.h, *map(float, prior), pkg.fptr(spread[0]), pkg.fptr(spread[1]))
        self.odom = [_odom(s, sc) for s in sc.steps]
        self.obs = [pkg.make_cobs(s.obs) for s in sc.steps]
        self.count = [len(s.obs) for s in sc.steps]
        self.prm = pkg.PfcCycleParams(0.05, 0.02, case["gate"], 0.5, case["inject"], 0)
        self.device = case["kind"] == "cycle_device"
        if self.device:
            flat = np.concatenate([pkg.cobs_records(s.obs) for s in sc.steps])
            self.d_obs = torch.from_numpy(flat.view(np.uint8).copy()).cuda()
            starts = np.concatenate([[0], np.cumsum(self.count)])
            self.at = [C.c_void_p(self.d_obs.data_ptr() + 24 * int(s)) for s in starts[:-1]]
        torch.cuda.synchronize()
        self.k = 0

    def run(self):
        k, self.k = self.k, (self.k + 1) % LOOP
        est = np.zeros(pkg.PFC_EST_LEN)
        if self.device:
            rc = self.lib.pfc_cycle_device(self.h, C.byref(self.odom[k]), self.at[k],
                                           self.count[k], C.byref(self.prm), pkg.dptr(est))
        else:
            rc = self.lib.pfc_cycle(self.h, C.byref(self.odom[k]), self.obs[k], self.count[k],
                                    C.byref(self.prm), pkg.dptr(est))
        if rc != 0:
            raise RuntimeError(pkg.last_error())
        return est

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.pfc_destroy(self.h)
            self.h = None


def _cloud(case, seed):
    """A cloud about a true pose, a map and observations of it (numpy, f32)."""
    r = np.random.default_rng(seed)
    n, nl, no = case["n"], case["landmarks"], case["nobs"]
    lm = r.uniform([-25, -25, 0], [25, 25, 10], (nl, 3)).astype(np.float32)
    truth = r.uniform([-5, -5, 2], [5, 5, 6])
    yaw = r.uniform(0, 2 * math.pi)
    q = np.array([math.cos(yaw / 2), 0.0, 0.0, math.sin(yaw / 2)])
    pos = (truth + r.normal(0, 0.05, (n, 3))).astype(np.float32)
    v = r.normal(0, 0.01, (n, 3))
    dq = np.c_[np.ones(n), v]
    dq /= np.linalg.norm(dq, axis=1, keepdims=True)
    quat = np.stack([q[0] * dq[:, 0] - q[3] * dq[:, 3], q[0] * dq[:, 1] - q[3] * dq[:, 2],
                     q[0] * dq[:, 2] + q[3] * dq[:, 1], q[0] * dq[:, 3] + q[3] * dq[:, 0]],
                    1).astype(np.float32)
    ids = r.permutation(nl)[:no] if no <= nl else r.integers(0, nl, no)
    world = lm[ids].astype(np.float64) - truth
    c, s = math.cos(yaw), math.sin(yaw)
    body = np.stack([c * world[:, 0] + s * world[:, 1], c * world[:, 1] - s * world[:, 0],
                     world[:, 2]], 1) + r.normal(0, 0.05, (no, 3))
    out = r.random(no) < 0.1
    body[out] += r.normal(0, 3.0, (int(out.sum()), 3))
    rows = np.zeros((no, 6))
    rows[:, 0] = ids
    rows[:, 2:5] = body
    rb = {"cart": np.zeros(no, bool), "bearing": np.ones(no, bool),
          "mixed": np.arange(no) % 3 == 0}[case["mode"]]
    rng_ = np.linalg.norm(body, axis=1)
    rows[rb, 1] = 1
    rows[rb, 5] = rng_[rb]
    rows[rb, 2:5] = -body[rb] / rng_[rb, None]
    return lm, pos, quat, rows


class _Weigh:
    """Weighting, estimate sums and covariances of a cloud the client set."""

    def __init__(self, case, seed):
        lm, pos, quat, rows = _cloud(case, seed)
        self.lib = pkg.kernels()
        self.h = self.lib.pfc_create(256)
        if not self.h or self.lib.pfc_init(self.h, case["n"], 42) != 0:
            raise RuntimeError(pkg.last_error())
        self.lib.pfc_upload_landmarks(self.h, pkg.fptr(lm.reshape(-1)), len(lm))
        self.lib.pfc_set_state(self.h, pkg.fptr(pos.reshape(-1)), pkg.fptr(quat.reshape(-1)), None)
        self.obs, self.count, self.gate = pkg.make_cobs(rows), len(rows), case["gate"]

    def run(self):
        sums, cov, q = np.zeros(14), np.zeros(12), np.zeros(4)
        bad = self.lib.pfc_weight(self.h, self.obs, self.count, 0.05, 0.02, self.gate)
        bad = bad or self.lib.pfc_est_sums(self.h, pkg.dptr(sums))
        pkg.core().pfcore_quat_mean(pkg.dptr(sums[3:13]), pkg.dptr(q))
        bad = bad or self.lib.pfc_covs(self.h, *map(float, np.float32(sums[:3])),
                                       *map(float, np.float32(q)), pkg.dptr(cov))
        if bad:
            raise RuntimeError(pkg.last_error())
        return dict(sums=sums, attitude=q, covariances=cov)

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.pfc_destroy(self.h)
            self.h = None


def _batch_plan(case, seed):
    r = np.random.default_rng(seed)
    nf = case["filters"]
    sizes = np.exp(r.uniform(math.log(case["n_min"]), math.log(case["n_max"]), nf)).astype(int)
    return r, sizes, r.integers(8, 65, nf), r.integers(4, 65, (nf, BATCH_LOOP))


class _Batch:
    """One cycle of every filter of a batch, from host inputs."""

    def __init__(self, case, seed):
        r, sizes, landmarks, counts = _batch_plan(case, seed)
        nf = case["filters"]
        scen = [sim.helix_scenario(BATCH_LOOP, int(landmarks[f]), (20.0, 20.0, 5.0), 64, 0.0,
                                   int(r.integers(1, 1 << 31)), radius=1.0, climb=0.0,
                                   arc=2 * math.pi / BATCH_LOOP,
                                   phase=float(r.uniform(0, 2 * math.pi))) for f in range(nf)]
        self.b = pkg.BatchPF(sizes, seeds=np.arange(1, nf + 1) + seed, obs_cap=64 * nf)
        self.b.set_params(gate=case["gate"], inject=case["inject"])
        self.b.set_landmarks([s.landmarks for s in scen])
        self.b.reinit([np.r_[s.prior_p, s.prior_q] for s in scen], np.full((nf, 3), 0.3),
                      np.full((nf, 3), 0.1))
        self.inputs = []
        for k in range(BATCH_LOOP):
            rows = np.concatenate([scen[f].steps[k].obs[:counts[f, k]] for f in range(nf)])
            self.inputs.append(((pkg.PfcOdom * nf)(*[_odom(s.steps[k], s) for s in scen]),
                                pkg.make_cobs(rows), counts[:, k].astype(np.int32)))
        self.nf, self.k = nf, 0

    def run(self):
        odom, obs, nobs = self.inputs[self.k]
        self.k = (self.k + 1) % BATCH_LOOP
        est = np.zeros((self.nf, pkg.PFC_EST_LEN))
        if pkg.kernels().pfc_batch_cycle(self.b.handle, odom, obs, pkg.iptr(nobs),
                                         pkg.dptr(est)) != 0:
            raise RuntimeError(pkg.last_error())
        return est


# ------------------------------------------------------- global localization

RES, RMAX = 0.05, 10.0


def _map(case, seed):
    """Walled room with box obstacles, and a true pose in it."""
    r = np.random.default_rng(seed)
    w, h = case.get("width", 200), case.get("height", 200)
    cells = np.zeros((h, w), np.uint8)
    cells[0, :] = cells[-1, :] = 1
    cells[:, 0] = cells[:, -1] = 1
    for _ in range(case.get("boxes", 30)):
        bw, bh = r.integers(4, 21, 2)
        x, y = int(r.integers(1, w - bw)), int(r.integers(1, h - bh))
        trial = cells.copy()
        trial[y:y + bh, x:x + bw] = 1
        if (trial == 0).mean() >= 0.6:
            cells = trial
    return r, cells


def _poses(r, cells, n):
    ys, xs = np.nonzero(cells == 0)
    at = r.integers(0, len(xs), n)
    return np.stack([(xs[at] + r.random(n)) * RES, (ys[at] + r.random(n)) * RES,
                     r.uniform(-math.pi, math.pi, n)], 1).astype(np.float32)


def _scan(gl, pose, case, seed):
    return pkg.render_scans(gl, pose, case["rays"], RMAX, case.get("span", 2 * math.pi), 0.01, seed)


def _fed(case, seed):
    """A client's own candidates: a uniform set, some of them near the truth."""
    r, cells = _map(case, seed)
    truth = _poses(r, cells, 1)
    hyps = _poses(r, cells, case["hyps"])
    near = case["hyps"] // 10
    hyps[:near] = truth + r.normal(0, [0.3, 0.3, 0.2], (near, 3))
    return cells, truth, hyps


class _GL:
    def __init__(self, case, seed, cap):
        self.case, self.lib = case, pkg.kernels()
        r, self.cells = _map(case, seed)
        self.r = r
        hh, w = self.cells.shape
        self.h = self.lib.pfgl_create(w, hh, RES, 0.0, 0.0, pkg.u8ptr(self.cells), cap)
        if not self.h:
            raise RuntimeError(pkg.last_error())

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.pfgl_destroy(self.h)
            self.h = None


class _Localize:
    """``CudaGlobalLoc::localize`` of the drop-in host layer."""

    def __init__(self, case, seed):
        r, cells = _map(case, seed)
        self.g = pkg.GlobalLoc(cells, RES, hypotheses=case["hyps"], rays=case["rays"], rmax=RMAX,
                               ang_span=case["span"], topk=case["topk"], seed=seed + 7)
        self.scan = _scan(self.g.handle, _poses(r, cells, 1), case, seed)[0]

    def run(self):
        return np.array(self.g.localize(self.scan))[:, :3]


class _Score(_GL):
    """CAER of fed hypotheses and the best of them."""

    def __init__(self, case, seed):
        super().__init__(case, seed, case["hyps"])
        _, truth, hyps = _fed(case, seed)
        if self.lib.pfgl_set_hyps(self.h, pkg.fptr(hyps.reshape(-1)), len(hyps)) != 0:
            raise RuntimeError(pkg.last_error())
        self.scan = _scan(self.h, truth, case, seed)[0]

    def run(self):
        c, k = self.case, self.case["topk"]
        pose, caer, idx = np.zeros((k, 3), np.float32), np.zeros(k, np.float32), np.zeros(k, np.int32)
        if self.lib.pfgl_score(self.h, pkg.fptr(self.scan), c["rays"], RMAX, c["span"]) != 0 or \
                self.lib.pfgl_topk_ex(self.h, k, pkg.fptr(pose), pkg.fptr(caer), pkg.iptr(idx)) != k:
            raise RuntimeError(pkg.last_error())
        return dict(caer=caer, index=idx, pose=pose)


class _LocalizeFused(_GL):
    """Dispersion (positions x 16 headings) and the fused, pruned localizer."""

    def __init__(self, case, seed):
        super().__init__(case, seed, case["hyps"])
        self.scan = _scan(self.h, _poses(self.r, self.cells, 1), case, seed)[0]
        self.seed = seed + 7

    def run(self):
        c, k = self.case, self.case["topk"]
        pose, caer, idx = np.zeros((k, 3), np.float32), np.zeros(k, np.float32), np.zeros(k, np.int32)
        if self.lib.pfgl_generate_yaws(self.h, c["hyps"] // 16, 16, self.seed) != 0 or \
                self.lib.pfgl_localize(self.h, pkg.fptr(self.scan), c["rays"], RMAX, c["span"], k,
                                       pkg.fptr(pose), pkg.fptr(caer), pkg.iptr(idx)) != k:
            raise RuntimeError(pkg.last_error())
        return dict(caer=caer, index=idx, pose=pose)


class _LearnedQueries(_GL):
    """A batch of scans through the learned proposal.  The network's weights
    are set by the client: random hidden layers and, as training leaves them,
    narrow mixture components spread over the map."""

    def __init__(self, case, seed):
        super().__init__(case, seed, case["queries"] * case["samples"])
        self.net = pkg.LearnedProposal(self.h, batch=case["batch"], seed=3)
        flat, at = [], 0
        for layer in range(pkg.LP_LAYERS):
            i = pkg.LP_IN if layer == 0 else pkg.LP_HIDDEN
            o = pkg.LP_OUT if layer == pkg.LP_LAYERS - 1 else pkg.LP_HIDDEN
            last = layer == pkg.LP_LAYERS - 1
            b = math.sqrt(6.0 / i) * (0.1 if last else 1.0)
            flat.append(self.r.uniform(-b, b, o * i).astype(np.float32))
            bias = np.zeros(o, np.float32)
            if last:
                bias[32:160] = self.r.uniform(-0.8, 0.8, 128)
                bias[160:288] = -2.0
            flat.append(bias)
        self.net.set_params(np.concatenate(flat))
        self.scans = _scan(self.h, _poses(self.r, self.cells, case["queries"]), case, seed)

    def run(self):
        c = self.case
        pose, caer, idx, info = self.net.localize_batch(self.scans, c["samples"], 0, c["topk"], RMAX)
        return dict(caer=caer, index=idx, pose=pose, info=info)

    def __del__(self):
        if getattr(self, "net", None):
            self.net.close()
        super().__del__()


class _LearnedTrain(_GL):
    """Adam steps over generated pairs; the loss of each and the weights."""

    def __init__(self, case, seed):
        super().__init__(case, seed, 1024)
        self.net = pkg.LearnedProposal(self.h, batch=case["batch"], seed=seed + 3)
        self.net.make_data(max(case["pairs"], case["batch"]), seed=seed + 7)

    def run(self):
        loss = self.net.train(self.case["steps"], 1200, 2e-3)
        return dict(loss=loss, weights=self.net.params())

    def __del__(self):
        if getattr(self, "net", None):
            self.net.close()
        super().__del__()


_KINDS = dict(update=_Update, cycle=_Cycle, cycle_device=_Cycle, weigh=_Weigh, batch=_Batch,
              localize=_Localize, score=_Score, localize_fused=_LocalizeFused,
              learned_queries=_LearnedQueries, learned_train=_LearnedTrain)


def prepare(case, seed):
    return _KINDS[case["kind"]](case, int(seed))


def run(state):
    return state.run()


# ---------------------------------------------------------------------- work

def _pf_work(n, landmarks, nobs, mode, move):
    """A pose is read (and, moved, written) once; a landmark is rotated into a
    particle's frame once (33 operations) and every observation compared with
    it: 10 operations, about 40 with the bearing's quotient and arc cosine."""
    seen = min(landmarks, nobs)
    per = {"cart": 10, "bearing": 40, "mixed": 20}[mode]
    return dict(bytes=n * (56 if move else 28) + 24 * nobs + 12 * landmarks,
                flops=n * (33 * seen + per * nobs + (200 if move else 80)))


def work(case):
    kind = case["kind"]
    if kind in ("update", "cycle", "cycle_device"):
        return _pf_work(case["n"], case["landmarks"], case["nobs"] or case["landmarks"],
                        case["mode"], True)
    if kind == "weigh":
        return _pf_work(case["n"], case["landmarks"], case["nobs"], case["mode"], False)
    if kind == "batch":
        _, sizes, landmarks, counts = _batch_plan(case, 0)
        parts = [_pf_work(int(sizes[f]), int(landmarks[f]), int(counts[f].mean()), "cart", True)
                 for f in range(case["filters"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind in ("localize", "score", "localize_fused", "learned_queries"):
        # a ray crosses some 50 cells of such a room, four operations each
        n = case["hyps"] if kind != "learned_queries" else case["queries"] * case["samples"]
        need = dict(bytes=12 * n, flops=n * case["rays"] * 50 * 4)
        if kind == "learned_queries":
            need["bytes"] += 4 * case["queries"] * case["rays"] + 2 * 3932160
            need["flops"] += 2 * 3932160 * case["queries"]
        return need
    rows = case["batch"] * case["steps"]
    # forward, and for the backward both gradients of each layer but the first
    return dict(bytes=rows * (384 * 2 + 16) + 2 * 4 * 3936256,
                flops=rows * 2 * (3 * 3932160 - 384 * 1024))


# --------------------------------------------------------------------- exact

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _qrot(qc, v):
    w, x, y, z = qc
    tx, ty, tz = 2 * (y * v[2] - z * v[1]), 2 * (z * v[0] - x * v[2]), 2 * (x * v[1] - y * v[0])
    return (v[0] + w * tx + y * tz - z * ty, v[1] + w * ty + z * tx - x * tz,
            v[2] + w * tz + x * ty - y * tx)


def _exact_weigh(case, seed):
    lm, pos, quat, rows = _cloud(case, seed)
    d = _dev()
    P, Q = torch.from_numpy(pos).to(d).double(), torch.from_numpy(quat).to(d).double()
    obs = np.float32(rows).astype(np.float64)
    sr, sb, g = float(np.float32(0.05)), float(np.float32(0.02)), case["gate"]
    at = torch.from_numpy(lm[rows[:, 0].astype(int)]).to(d).double()
    o = torch.from_numpy(obs).to(d)
    ll = torch.empty(len(pos), dtype=torch.float64, device=d)
    for a in range(0, len(pos), 32768):
        p, q = P[a:a + 32768], Q[a:a + 32768]
        v = [at[None, :, k] - p[:, k:k + 1] for k in range(3)]
        e = _qrot((q[:, 0:1], -q[:, 1:2], -q[:, 2:3], -q[:, 3:4]), v)
        r2 = sum((e[k] - o[None, :, 2 + k]) ** 2 for k in range(3))
        cart = -r2 / (2 * sr * sr)
        if g > 0:
            cart = torch.where(r2 > g * g * 3 * sr * sr, torch.full_like(cart, -1.5 * g * g), cart)
        rn = torch.sqrt(sum(x * x for x in e)).clamp_min(1e-9)
        er2 = (rn - o[None, :, 5]) ** 2
        eb2 = torch.arccos((-sum(e[k] * o[None, :, 2 + k] for k in range(3)) / rn).clamp(-1, 1)) ** 2
        tr, tb = -er2 / (2 * sr * sr), -eb2 / (2 * sb * sb)
        if g > 0:
            tr = torch.where(er2 > g * g * sr * sr, torch.full_like(tr, -0.5 * g * g), tr)
            tb = torch.where(eb2 > g * g * sb * sb, torch.full_like(tb, -0.5 * g * g), tb)
        ll[a:a + 32768] = torch.where(o[None, :, 1] == 0, cart, tr + tb).sum(1)
    w = torch.softmax(ll, 0)
    mean = (w[:, None] * P).sum(0)
    M = torch.einsum("n,ni,nj->ij", w, Q, Q)
    up = [(i, j) for i in range(4) for j in range(i, 4)]
    sums = torch.cat([mean, torch.stack([M[i, j] for i, j in up]), (w * w).sum()[None]])
    qm = torch.linalg.eigh(M)[1][:, 3]
    qm = qm if qm[0] >= 0 else -qm
    dp = P - mean
    a = _qrel(qm, Q)
    s = torch.where(a[0] < 0, -1.0, 1.0)
    vec = torch.stack([a[k] * s for k in (1, 2, 3)], 1)
    nv = vec.norm(dim=1)
    f = torch.where(nv > 1e-12, 2 * torch.atan2(nv, a[0] * s) / nv.clamp_min(1e-300), 0.0)
    rv = vec * f[:, None]
    up3 = [(i, j) for i in range(3) for j in range(i, 3)]
    cov = [(w * x[:, i] * x[:, j]).sum() for x in (dp, rv) for i, j in up3]
    return dict(sums=sums.cpu().numpy(), attitude=qm.cpu().numpy(),
                covariances=torch.stack(cov).cpu().numpy())


def _qrel(m, Q):
    w, x, y, z = m[0], -m[1], -m[2], -m[3]
    a, b, c, d = Q[:, 0], Q[:, 1], Q[:, 2], Q[:, 3]
    return (w * a - x * b - y * c - z * d, w * b + x * a + y * d - z * c,
            w * c - x * d + y * a + z * b, w * d + x * c - y * b + z * a)


def _exact_score(case, seed):
    """CAERs of the best hypotheses by stepping every ray through the grid."""
    cells, truth, hyps = _fed(case, seed)
    d = _dev()
    if d.type == "cpu" and case["hyps"] * case["rays"] > 200000:
        return None
    state = _Score(case, seed)
    scan = torch.from_numpy(state.scan).to(d).double()
    del state
    rays, (hh, ww) = case["rays"], cells.shape
    occ = torch.from_numpy(np.pad(cells, 1, constant_values=2).reshape(-1)).to(d)
    res = float(np.float32(RES))
    H = torch.from_numpy(hyps).to(d).double()
    best = []
    for a in range(0, len(hyps), 8192):
        h = H[a:a + 8192]
        th = h[:, 2:3] + case["span"] * torch.arange(rays, device=d, dtype=torch.float64) / (rays - 1)
        dx, dy = torch.cos(th), torch.sin(th)
        fx, fy = (h[:, 0] / res)[:, None].expand_as(th), (h[:, 1] / res)[:, None].expand_as(th)
        cx, cy = torch.floor(fx), torch.floor(fy)
        inside = (cx >= 0) & (cy >= 0) & (cx < ww) & (cy < hh)
        tdx, tdy = res / dx.abs().clamp_min(1e-300), res / dy.abs().clamp_min(1e-300)
        tmx = torch.where(dx > 0, 1 - (fx - cx), fx - cx) * tdx
        tmy = torch.where(dy > 0, 1 - (fy - cy), fy - cy) * tdy
        sx, sy = torch.where(dx > 0, 1, -1), torch.where(dy > 0, ww + 2, -(ww + 2))
        at = ((cy + 1) * (ww + 2) + cx + 1).long()
        dist = torch.full_like(th, RMAX)
        open_ = inside.clone()
        at = torch.where(open_, at, 0)
        while bool(open_.any()):
            px = tmx <= tmy
            t = torch.where(px, tmx, tmy)
            tmx, tmy = torch.where(px, tmx + tdx, tmx), torch.where(px, tmy, tmy + tdy)
            at = torch.where(open_, at + torch.where(px, sx, sy), at)
            v = occ[at]
            dist = torch.where(open_ & (v == 1) & (t <= RMAX), t, dist)
            open_ = open_ & (v == 0) & (t <= RMAX)
        best.append((scan[None, :] - dist).abs().sum(1))
    caer = torch.sort(torch.cat(best))[0][:case["topk"]]
    # the order of near ties is a matter of rounding, so poses have no such value
    return dict(caer=caer.cpu().numpy(), index=None, pose=None)


def exact(case, seed):
    """Values in 64 bits where the inputs are the client's own.  Filters move
    by the library's noise streams and resample by its offsets, dispersions
    and mixture samples are its draws: those outputs have no value outside."""
    if case["kind"] == "weigh":
        return _exact_weigh(case, int(seed))
    if case["kind"] == "score":
        return _exact_score(case, int(seed))
    return None
