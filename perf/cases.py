"""The workloads that this library's speed is measured on.

Each case is one call (or the few calls that belong together) a user's program
makes through the public Python binding, with its problem already analysed:
batches of QPs with new vectors, a warm-started parametric batch, one large
QP, one KKT system with new values, and the active-set model's forward pass
and gradients.  Problems come from nasoq_gb300.problems (seeded synthetic).
"""
import functools
import math

import numpy as np
import torch

import nasoq_gb300 as nq
from nasoq_gb300 import learn
from nasoq_gb300 import problems as P

EPS = 1e-8
MODEL_SIZES = (32, 256, 256, 900)  # the active-set model of the horizon-50 MPC family
THRESHOLD = 1.5                    # logit above which it proposes a constraint


def listed():
    return [
        # one small control problem at a time: the latency of a call (default settings: FP64, reference refinement)
        {"name": "mpc10_one_fp64", "kind": "batch", "family": "mpc", "count": 1, "horizon": 10, "mixed": False},
        # parametric MPC, learned warm start: the main workload, theta on the host to solutions on the host
        {"name": "mpc50_warm_4096", "kind": "warm", "count": 4096},
        # the same family without a model: labelling training data, first deployment
        {"name": "mpc50_cold_mixed_2048", "kind": "batch", "family": "mpc", "count": 2048, "horizon": 50,
         "mixed": True},
        # the plain path of the default settings on a batch
        {"name": "mpc50_cold_fp64_1024", "kind": "batch", "family": "mpc", "count": 1024, "horizon": 50,
         "mixed": False},
        # MPC problems of uneven horizons 10..100, every problem with matrices of its own
        {"name": "mpc_uneven_mixed_1024", "kind": "batch", "family": "uneven", "count": 1024, "horizon": 100,
         "mixed": True},
        # small general QPs, every one with a sparsity pattern of its own
        {"name": "random_fp64_96", "kind": "batch", "family": "random", "count": 96, "horizon": 12, "mixed": False},
        # one QP through the host's active-set loop, analysis included: a random convex one and a bounded mesh one
        {"name": "single_random_n576", "kind": "single", "family": "random", "grid": 24},
        {"name": "single_mesh_n1600", "kind": "single", "family": "mesh", "grid": 40},
        # one KKT system, new values and right-hand side: FP32 factor with FP64 refinement, and plain FP64
        {"name": "kkt_40cube_fp32", "kind": "kkt", "grid": 40, "fp32": True},
        {"name": "kkt_20cube_fp64", "kind": "kkt", "grid": 20, "fp32": False},
        # the active-set model: logits of a batch of parameters, and the gradients of a mini-batch
        {"name": "model_forward_4096", "kind": "forward", "rows": 4096},
        {"name": "model_gradient_1024", "kind": "gradient", "rows": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["batch", "batch", "batch", "warm", "single", "kkt", "forward", "gradient"])
    if kind == "batch":
        family = rng.choice(["mpc", "mpc", "uneven", "random"])
        if family == "random":
            return {"kind": kind, "family": family, "count": _log_int(rng, 1, 96), "horizon": rng.randint(6, 14),
                    "mixed": rng.random() < 0.3}
        horizon = rng.randint(10, 100)
        most = min(2048, int(1024 * (50 / horizon) ** 2)) if family == "mpc" else int(1024 * 100 / horizon)
        return {"kind": kind, "family": family, "count": _log_int(rng, 1, min(most, 1024)), "horizon": horizon,
                "mixed": rng.random() < 0.5}
    if kind == "warm":
        return {"kind": kind, "count": _log_int(rng, 16, 4095)}
    if kind == "single":
        family = rng.choice(["random", "mesh"])
        return {"kind": kind, "family": family, "grid": rng.randint(7, 24) if family == "random" else rng.randint(12, 40)}
    if kind == "kkt":
        fp32 = rng.random() < 0.5
        return {"kind": kind, "grid": rng.randint(8, 39) if fp32 else rng.randint(6, 23), "fp32": fp32}
    return {"kind": kind, "rows": _log_int(rng, 1, 4096) if kind == "forward" else _log_int(rng, 32, 1024)}


# ---- the problems -------------------------------------------------------------

def _batch_problems(case, seed):
    """The QPs of a batch.  The plants are the program's own (the "mpc"
    family's one, the "uneven" family's horizons, the "random" family's
    matrices); an uneven plant's matrices come from the seed."""
    count, h = case["count"], case["horizon"]
    if case["family"] == "mpc":
        return [P.qp_mpc(0, h)] * count
    if case["family"] == "uneven":
        horizons = np.random.default_rng(count).integers(min(10, h), h + 1, size=count)
        horizons[0] = h
        return [P.qp_mpc(seed * 100003 + i, int(k)) for i, k in enumerate(horizons)]
    n = h * h
    return [P.qp_random_convex(i, grid=h, meq=max(1, n // 7), mineq=max(4, n * 5 // 6)) for i in range(count)]


def _batch_vectors(case, qps, seed):
    """q, b, d of every problem, stacked: this step's vectors."""
    rng = np.random.default_rng([seed, 5])
    if case["family"] == "mpc":
        base = qps[0]
        # costs and box shifts of the size that the parametric family has; a box moves as a whole
        q = 0.6 * rng.standard_normal((len(qps), base.n))
        shift = 0.6 * rng.standard_normal((len(qps), base.n))
        d = np.repeat(base.d[None, :], len(qps), axis=0)
        d[:, 0::2] += shift
        d[:, 1::2] -= shift
        return q.ravel(), None, d.ravel()
    q = np.concatenate([p.q for p in qps])
    return q * (1.0 + 0.05 * rng.standard_normal(q.size)), np.concatenate([p.b for p in qps]), \
        np.concatenate([p.d for p in qps])


def _single(case, seed):
    g = case["grid"]
    if case["family"] == "mesh":
        return P.bilaplacian_bounded(seed, grid=g, pins=max(4, g * g // 80))
    n = g * g
    return P.qp_random_convex(seed, grid=g, meq=max(1, n * 200 // 2025), mineq=max(1, n * 1000 // 2025))


def _kkt(case, seed):
    g = case["grid"]
    return P.lbl_kkt(seed, grid3d=g, m=max(8, g ** 3 * 20000 // 64 ** 3), per_row=6, delta=1e-8)


@functools.lru_cache(maxsize=1)
def _family():
    return P.mpc_parametric(0)


@functools.lru_cache(maxsize=1)
def _model_weights():
    """Weights of the family's active-set model, trained once per process on
    solved instances (plain torch, so that the weights are those of any model
    a user brings); rounded to BF16, the precision the library keeps them in."""
    fam = _family()
    theta = np.random.default_rng(3).standard_normal((49152, MODEL_SIZES[0]))
    labels, _, _ = learn.solve_labels(fam, theta, variant=0, eps_abs=EPS, precision=nq.NQG_FP32, refine=1,
                                      refine_tol=1e-10)
    gen = torch.Generator().manual_seed(7)
    ws, bs = [], []
    for i, o in zip(MODEL_SIZES[:-1], MODEL_SIZES[1:]):
        ws.append((torch.randn((o, i), generator=gen) * math.sqrt(2.0 / i)).cuda().requires_grad_())
        bs.append(torch.zeros(o, device="cuda", requires_grad=True))
    x, y = torch.from_numpy(theta.astype(np.float32)).cuda(), torch.from_numpy(labels).cuda()
    weight = torch.clamp((1 - y.mean()) / y.mean().clamp(min=1e-6), max=50.0)
    opt = torch.optim.Adam(ws + bs, lr=1e-3)
    for _ in range(60):
        for rows in torch.randperm(x.shape[0], generator=gen).cuda().split(1024):
            h = x[rows]
            for l, (w, b) in enumerate(zip(ws, bs)):
                h = torch.nn.functional.linear(h, w, b)
                h = torch.relu(h) if l + 1 < len(ws) else h
            loss = torch.nn.functional.binary_cross_entropy_with_logits(h, y[rows], pos_weight=weight,
                                                                        reduction="sum") / rows.numel()
            opt.zero_grad()
            loss.backward()
            opt.step()
    w = np.concatenate([t.detach().bfloat16().float().cpu().numpy().ravel() for t in ws])
    return w, np.concatenate([t.detach().cpu().numpy() for t in bs])


def _random_weights(seed):
    """He-initialised weights at BF16 values, small biases."""
    rng = np.random.default_rng([seed, 9])
    w = np.concatenate([(rng.standard_normal(i * o) * math.sqrt(2.0 / i)) for i, o in
                        zip(MODEL_SIZES[:-1], MODEL_SIZES[1:])])
    w = torch.from_numpy(w).bfloat16().float().numpy()
    return w, (0.1 * rng.standard_normal(sum(MODEL_SIZES[1:]))).astype(np.float32)


def _model_rows(case, seed):
    rng = np.random.default_rng([seed, 10])
    x = rng.standard_normal((case["rows"], MODEL_SIZES[0])).astype(np.float32)
    return x, (rng.random((case["rows"], MODEL_SIZES[-1])) < 0.05).astype(np.float32)


# ---- what a program has in hand, and the call ------------------------------------

def prepare(case, seed):
    torch.cuda.init()
    kind = case["kind"]
    if kind == "batch":
        qps = _batch_problems(case, seed)
        s = dict(precision=nq.NQG_FP32, refine=1, refine_tol=1e-10) if case["mixed"] else {}
        batch = nq.QPBatch([(p.H, p.q, p.A, p.b, p.C, p.d) for p in qps], settings=nq.batch_settings(eps_abs=EPS, **s))
        return kind, batch, _batch_vectors(case, qps, seed)
    if kind == "warm":
        fam = _family()
        batch = learn.family_batch(fam, case["count"], variant=0, eps_abs=EPS, precision=nq.NQG_FP32, refine=1,
                                   refine_tol=1e-10)
        model = nq.MLP(MODEL_SIZES)
        model.set_weights(*_model_weights())
        theta = np.random.default_rng([seed, 1]).standard_normal((case["count"], MODEL_SIZES[0]))
        return kind, learn.WarmStarter(batch, model, fam, threshold=THRESHOLD), theta
    if kind == "single":
        return kind, _single(case, seed)
    if kind == "kkt":
        K, rhs = _kkt(case, seed)
        if case["fp32"]:
            s = nq.default_settings(precision=nq.NQG_FP32, solve_precision=nq.NQG_FP32, req_ref_iter=1,
                                    max_inner_iter=8, tol_abs=1e-12 * float(np.linalg.norm(rhs)), tol_rel=1.0,
                                    reg_diag=1e-9)
        else:
            s = nq.default_settings(req_ref_iter=2, max_inner_iter=2, reg_diag=1e-9)
        return kind, nq.Plan(K.ncol, K.p, K.i, K.x, settings=s), K.x, rhs
    model = nq.MLP(MODEL_SIZES)
    model.set_weights(*_random_weights(seed))
    x, y = _model_rows(case, seed)
    if kind == "forward":
        return kind, model, torch.from_numpy(x).cuda(), torch.empty(y.shape, dtype=torch.float32, device="cuda")
    return kind, model, x, y


def _solution(x, y, z, stats):
    return {"x": x, "y": y, "z": z, "objective": np.array([s.objective for s in stats]),
            "status": np.array([s.status for s in stats], np.int32)}


def run(state):
    kind = state[0]
    if kind == "batch":
        _, batch, (q, b, d) = state
        batch.set_vectors(q, b, d)
        batch.solve()
        return _solution(*batch.results())
    if kind == "warm":
        _, starter, theta = state
        return _solution(*starter.solve(theta))
    if kind == "single":
        qp = state[1]
        x, y, z, _, r = nq.qp_solve(qp.H, qp.q, qp.A, qp.b, qp.C, qp.d, settings=nq.qp_settings(variant=0, eps_abs=EPS))
        return {"x": x, "y": y, "z": z, "objective": float(r.objective), "status": int(r.status)}
    if kind == "kkt":
        _, plan, values, rhs = state
        plan.set_values(values)
        plan.factor()
        return plan.solve(rhs)
    if kind == "forward":
        _, model, x, out = state
        model.forward_device(x.shape[0], x.data_ptr(), out.data_ptr())
        return out
    _, model, x, y = state
    loss, gw, gb = model.loss_grad(x, y, pos_weight=8.0)
    return {"loss": np.float32(loss), "weights": gw, "biases": gb}  # the loss is a sum of FP32 terms


# ---- what a pass cannot do without ------------------------------------------------

@functools.lru_cache(maxsize=64)
def _factor_work(kind, family, size):
    """(bytes of the values, FLOPs of one factorization and solve) of a
    system, from the symbolic factor that its ordering gives."""
    if kind == "kkt":
        K, _ = _kkt({"grid": size}, 0)
        n, p, i, hidden = K.ncol, K.p, K.i, None
    else:
        qp = P.qp_mpc(0, size) if family == "mpc" else _single({"family": family, "grid": size}, 0) \
            if kind == "single" else _batch_problems({"family": "random", "count": 1, "horizon": size}, 0)[0]
        K = P.kkt_lower_fast(qp.H, qp.A, 1e-9)  # the equality-constrained system: where the iteration starts
        n, p, i, hidden = K.ncol, K.p, K.i, None
    sym = nq.Symbolic(n, p, i, extra_cols=hidden)
    rows = np.diff(sym.lpi).astype(np.float64)
    wide = np.diff(sym.super).astype(np.float64)
    k = rows - (wide - 1) / 2
    return 8.0 * len(i), float((wide * k * k).sum() + 4.0 * (wide * k).sum())


def work(case):
    kind = case["kind"]
    if kind in ("forward", "gradient"):
        nw = sum(i * o for i, o in zip(MODEL_SIZES[:-1], MODEL_SIZES[1:]))
        if kind == "forward":
            return {"bytes": 4 * case["rows"] * (MODEL_SIZES[0] + MODEL_SIZES[-1]) + 2 * nw + 4 * sum(MODEL_SIZES[1:]),
                    "flops": 2 * case["rows"] * nw}
        return {"bytes": 4 * case["rows"] * (MODEL_SIZES[0] + MODEL_SIZES[-1]) + 6 * nw + 8 * sum(MODEL_SIZES[1:]),
                "flops": 2 * case["rows"] * (3 * nw - MODEL_SIZES[0] * MODEL_SIZES[1])}
    if kind == "kkt":
        values, flops = _factor_work("kkt", "", case["grid"])
        n = case["grid"] ** 3 + max(8, case["grid"] ** 3 * 20000 // 64 ** 3)
        return {"bytes": values + 16 * n, "flops": flops}
    if kind == "single":
        values, flops = _factor_work("single", case["family"], case["grid"])
        qp = _single(case, 0)
        return {"bytes": values + 8 * len(qp.C.x) + 8 * (2 * qp.n + 2 * qp.A.nrow + 2 * qp.C.nrow), "flops": flops}
    # a batch: vectors in, solutions out, every distinct matrix read once; one factorization and solve per QP
    count = case["count"]
    if kind == "warm":
        values, flops = _factor_work("batch", "mpc", 50)
        base = _family().base
        n, me, mi = base.n, base.A.nrow, base.C.nrow
        return {"bytes": 8.0 * count * (MODEL_SIZES[0] + n + me + mi) + values + 8 * 32 * (n + mi),
                "flops": count * (flops + 2 * 32 * (n + mi))}
    if case["family"] == "uneven":
        mid = (min(10, case["horizon"]) + case["horizon"]) // 2
        values, flops = _factor_work("batch", "mpc", mid)
        n, me, mi, distinct = 9 * mid, 6 * mid, 18 * mid, count
    elif case["family"] == "mpc":
        values, flops = _factor_work("batch", "mpc", case["horizon"])
        n, me, mi, distinct = 9 * case["horizon"], 6 * case["horizon"], 18 * case["horizon"], 1
    else:
        values, flops = _factor_work("batch", "random", case["horizon"])
        n = case["horizon"] ** 2
        me, mi, distinct = max(1, n // 7), max(4, n * 5 // 6), count
    return {"bytes": 8.0 * count * (2 * n + 2 * me + 2 * mi) + distinct * (values + 16.0 * mi), "flops": count * flops}


# ---- the same in 64 bits, by plain torch --------------------------------------------

class _KKT:
    """(H + C' w C) dx + A' dy = r1, A dx = r2 for a stack of problems;
    C None stands for the rows x_v, -x_v, x_v', -x_v', ... of a box and H is
    then a diagonal."""

    def __init__(self, H, A, C):
        self.H, self.A, self.C = H, A, C

    def c(self, x):
        return torch.stack((x, -x), -1).flatten(-2) if self.C is None else (self.C @ x[..., None])[..., 0]

    def ct(self, z):
        return z[..., 0::2] - z[..., 1::2] if self.C is None else (self.C.mT @ z[..., None])[..., 0]

    def h(self, x):
        return self.H * x if self.C is None else (self.H @ x[..., None])[..., 0]

    def a(self, x):
        return (self.A @ x[..., None])[..., 0]

    def at(self, y):
        return (self.A.mT @ y[..., None])[..., 0]

    def factor(self, w):
        if self.C is None:
            m = self.H + w[..., 0::2] + w[..., 1::2]
            self.inv = lambda r: r / (m if r.dim() == m.dim() else m[..., None])
        else:
            L = torch.linalg.cholesky(self.H + (self.C.mT * w[..., None, :]) @ self.C)
            self.inv = lambda r: torch.cholesky_solve(r if r.dim() == L.dim() else r[..., None], L).reshape(r.shape)
        self.S = torch.linalg.cholesky(self.A @ self.inv(self.A.mT.expand(w.shape[0], -1, -1)))

    def solve(self, r1, r2):
        dy = torch.cholesky_solve((self.a(self.inv(r1)) - r2)[..., None], self.S)[..., 0]
        return self.inv(r1 - self.at(dy)), dy


def _optimum(H, q, A, b, C, d):
    """min 1/2 x'Hx + q'x, Ax = b, Cx <= d for a stack of problems (see
    _KKT): Mehrotra's predictor-corrector interior point, then the
    equality-constrained solution on the active set it finds."""
    k = _KKT(H, A, C)
    x, y = torch.zeros_like(q), torch.zeros_like(b)
    z = torch.ones_like(d)
    s = torch.clamp(d - k.c(x), min=1.0)

    def room(v, dv):
        return torch.where(dv < 0, -v / dv, torch.full_like(v, 1e30)).amin(-1, keepdim=True).clamp(max=1.0)

    for _ in range(80):
        rd, rp, rc = k.h(x) + q + k.at(y) + k.ct(z), k.a(x) - b, k.c(x) + s - d
        mu = (s * z).mean(-1, keepdim=True)
        todo = (mu > 1e-12) | (rp.abs().amax(-1, keepdim=True) > 1e-9) | (rc.abs().amax(-1, keepdim=True) > 1e-9)
        if not bool(todo.any()):
            break
        k.factor(z / s)

        def direction(rm):
            dx, dy = k.solve(-rd - k.ct((z * rc - rm) / s), -rp)
            ds = -rc - k.c(dx)
            return dx, dy, (-rm - z * ds) / s, ds

        _, _, dz, ds = direction(s * z)
        a = torch.minimum(room(s, ds), room(z, dz))
        sigma = (((s + a * ds) * (z + a * dz)).mean(-1, keepdim=True) / mu) ** 3
        dx, dy, dz, ds = direction(s * z + ds * dz - sigma * mu)
        a = (0.995 * torch.minimum(room(s, ds), room(z, dz))) * todo
        x, y, z, s = x + a * dx, y + a * dy, z + a * dz, s + a * ds
    active = (z > s).to(q.dtype)
    z = z * active
    w = 1e6 * active
    k.factor(w)
    for _ in range(12):  # refinement by the active rows' augmented system
        r1, r3 = -(k.h(x) + q + k.at(y) + k.ct(z)), (d - k.c(x)) * active
        dx, dy = k.solve(r1 + k.ct(w * r3), b - k.a(x))
        dz = w * (k.c(dx) - r3)
        x, y, z = x + dx, y + dy, z + dz
    objective = (0.5 * x * k.h(x) + q * x).sum(-1) + ((k.c(x) - d) * z).sum(-1)
    return x, y, z, objective


def _dense(M):
    out = torch.zeros((M.nrow, M.ncol), dtype=torch.float64)
    out[torch.from_numpy(M.i.astype(np.int64)), torch.from_numpy(np.repeat(np.arange(M.ncol), np.diff(M.p)))] = \
        torch.from_numpy(np.asarray(M.x, np.float64))
    return out.cuda()


def _dense_sym(M):
    t = _dense(M)
    return t + t.mT - torch.diag(torch.diag(t))


def _to(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float64)).cuda()


def _stack_answers(rows):
    x, y, z, o = (torch.cat([r[k].reshape(-1) for r in rows]).cpu().numpy() for k in range(4))
    return {"x": x, "y": y, "z": z, "objective": o, "status": None}


def _exact_mpc_shared(base, q, d, chunk=1024):
    """A stack of problems over one plant's matrices (diagonal H, box rows)."""
    H, A = torch.diag(_dense(base.H))[None], _dense(base.A)[None]
    return _stack_answers([_optimum(H, _to(q[i:i + chunk]), A, _to(base.b).expand(len(q[i:i + chunk]), -1), None,
                                    _to(d[i:i + chunk])) for i in range(0, len(q), chunk)])


def _exact_mpc_uneven(qps, q_all, chunk=64):
    """Problems of different horizons: stacked in order of size, the smaller
    ones filled up with separate variables held at zero."""
    order = sorted(range(len(qps)), key=lambda i: qps[i].n)
    at = np.cumsum([0] + [p.n for p in qps])
    found = [None] * len(qps)
    for c0 in range(0, len(order), chunk):
        ids = order[c0:c0 + chunk]
        n, me = qps[ids[-1]].n, qps[ids[-1]].A.nrow
        H, q = torch.ones((len(ids), n), dtype=torch.float64).cuda(), torch.zeros((len(ids), n), dtype=torch.float64).cuda()
        A, b = torch.zeros((len(ids), me, n), dtype=torch.float64).cuda(), torch.zeros((len(ids), me), dtype=torch.float64).cuda()
        d = torch.ones((len(ids), 2 * n), dtype=torch.float64).cuda()
        for r, i in enumerate(ids):
            p = qps[i]
            m = p.A.nrow
            H[r, :p.n], q[r, :p.n], b[r, :m] = _to(p.H.x), _to(q_all[at[i]:at[i + 1]]), _to(p.b)
            A[r, :m, :p.n], d[r, :2 * p.n] = _dense(p.A), _to(p.d)
            A[r, torch.arange(m, me), p.n + torch.arange(me - m)] = 1.0
        x, y, z, o = _optimum(H, q, A, b, None, d)
        for r, i in enumerate(ids):
            found[i] = (x[r, :qps[i].n], y[r, :qps[i].A.nrow], z[r, :qps[i].C.nrow], o[r:r + 1])
    return _stack_answers(found)


def _exact_general(qp, q):
    """One QP with dense matrices."""
    x, y, z, o = _optimum(_dense_sym(qp.H)[None], _to(q)[None], _dense(qp.A)[None], _to(qp.b)[None],
                          _dense(qp.C)[None], _to(qp.d)[None])
    return x[0], y[0], z[0], o


def _exact_kkt(case, seed):
    """x of [H A'; A -delta I] x = rhs by the Schur complement of H, the 3-D
    Laplacian, whose inverse the sine transform gives."""
    K, rhs = _kkt(case, seed)
    g = case["grid"]
    n, m = g ** 3, K.ncol - g ** 3
    col = np.repeat(np.arange(K.ncol), np.diff(K.p))
    below = (K.i >= n) & (col < n)
    A = torch.zeros((m, n), dtype=torch.float64)
    A[torch.from_numpy(K.i[below].astype(np.int64) - n), torch.from_numpy(col[below])] = torch.from_numpy(K.x[below])
    A = A.cuda()
    k = torch.arange(1, g + 1, dtype=torch.float64).cuda()
    S = torch.sin(math.pi / (g + 1) * k[:, None] * k[None, :]) * math.sqrt(2.0 / (g + 1))
    lam = 2.0 - 2.0 * torch.cos(math.pi * k / (g + 1))
    lam = lam[:, None, None] + lam[None, :, None] + lam[None, None, :]

    def transform(v):
        for ax in (1, 2, 3):
            v = torch.tensordot(v, S, dims=([ax], [0])).movedim(-1, ax)
        return v

    def h_inv(v):
        return (transform(transform(v.reshape(-1, g, g, g)) / lam)).reshape(-1, n)

    def h_mul(v):
        u = v.reshape(g, g, g)
        out = 6.0 * u
        for ax in range(3):
            lo, hi = [slice(None)] * 3, [slice(None)] * 3
            lo[ax], hi[ax] = slice(0, g - 1), slice(1, g)
            out[tuple(hi)] -= u[tuple(lo)]
            out[tuple(lo)] -= u[tuple(hi)]
        return out.reshape(-1)

    schur = torch.empty((m, m), dtype=torch.float64, device="cuda")
    for r in range(0, m, 512):
        schur[r:r + 512] = h_inv(A[r:r + 512]) @ A.mT
    delta = 1e-8
    low = torch.linalg.cholesky(schur + delta * torch.eye(m, dtype=torch.float64, device="cuda"))
    f, h = _to(rhs[:n]), _to(rhs[n:])
    x, y = torch.zeros_like(f), torch.zeros_like(h)
    for _ in range(3):
        r1, r2 = f - h_mul(x) - A.mT @ y, h - A @ x + delta * y
        dy = torch.cholesky_solve((A @ h_inv(r1)[0] - r2)[:, None], low)[:, 0]
        x, y = x + h_inv(r1 - A.mT @ dy)[0], y + dy
    return torch.cat((x, y)).cpu().numpy()


def _exact_model(case, seed):
    w, b = _random_weights(seed)
    x, labels = _model_rows(case, seed)
    ws, bs, ow, ob = [], [], 0, 0
    for i, o in zip(MODEL_SIZES[:-1], MODEL_SIZES[1:]):
        ws.append(_to(w[ow:ow + i * o].reshape(o, i)).requires_grad_())
        bs.append(_to(b[ob:ob + o]).requires_grad_())
        ow, ob = ow + i * o, ob + o
    h = _to(x)
    for l, (wl, bl) in enumerate(zip(ws, bs)):
        h = torch.nn.functional.linear(h, wl, bl)
        h = torch.relu(h) if l + 1 < len(ws) else h
    if case["kind"] == "forward":
        return h.detach()
    loss = torch.nn.functional.binary_cross_entropy_with_logits(
        h, _to(labels), pos_weight=torch.tensor(8.0, dtype=torch.float64, device="cuda"), reduction="sum") / len(x)
    loss.backward()
    return {"loss": np.float64(loss.item()), "weights": torch.cat([t.grad.reshape(-1) for t in ws]).cpu().numpy(),
            "biases": torch.cat([t.grad for t in bs]).cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "kkt":
        return _exact_kkt(case, seed)
    if kind in ("forward", "gradient"):
        return _exact_model(case, seed)
    if kind == "warm":
        fam = _family()
        theta = np.random.default_rng([seed, 1]).standard_normal((case["count"], MODEL_SIZES[0]))
        return _exact_mpc_shared(fam.base, theta @ fam.P.T, fam.d0[None, :] + theta @ fam.S.T)
    if kind == "single":
        qp = _single(case, seed)
        x, y, z, o = (t.cpu().numpy().reshape(-1) for t in _exact_general(qp, qp.q))
        # a pinned vertex of the mesh has its bound and its pin: the multipliers are not unique
        unique = case["family"] != "mesh"
        return {"x": x, "y": y if unique else None, "z": z if unique else None, "objective": float(o[0]), "status": None}
    qps = _batch_problems(case, seed)
    q, _, d = _batch_vectors(case, qps, seed)
    if case["family"] == "mpc":
        return _exact_mpc_shared(qps[0], q.reshape(len(qps), -1), d.reshape(len(qps), -1))
    if case["family"] == "uneven":
        return _exact_mpc_uneven(qps, q)
    at = np.cumsum([0] + [p.n for p in qps])
    return _stack_answers([_exact_general(p, q[at[i]:at[i + 1]]) for i, p in enumerate(qps)])
