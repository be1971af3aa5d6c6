"""The workloads the solvers' speed is judged on: what a user's program calls, over the range of
sizes, precisions and problem families this package is used on.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  the inputs and handles a program holds before the call
    run(state)           one pass through the public entry points, with its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the outputs in 64 bits, by plain torch / numpy

Kinds:
  kkt      primal residual and objective of a candidate point on device buffers
           (cp_al_gb300_primal_kkt_noalloc)
  lp       a solve on a device-resident session (LPSession.solve, then fetch): equilibration,
           the sigma_max estimate, the iterations and the result
  lp_host  the same from host arrays (lp.solve)
  qp       a convex QP from host arrays (qp.solve)
  batch    many uneven LPs in one launch (lp.solve_batch)
  train    one epoch of the warm-start network (MLP.set_params, train, get_params)
  grad     loss and gradient of one batch of it (MLP.loss_grad)
  predict  network inference on host rows (MLP.predict)
  warm     warm starts of a family of transportation LPs (WarmStart.predict_device)

LP and QP solves run a stated number of iterations: a pass is the same work on both sides of a
comparison, and it ends as a solve with an iteration budget does.  In the fp32_refine form those
iterations all lie in the FP32 phase, which holds x and y in 32 bits; they are returned in 32 bits.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from pdal_gb300 import _native as N
from pdal_gb300 import instances, learn, lp, qp

DEV = "cuda" if torch.cuda.is_available() else "cpu"
L2_BYTES = 126e6

# the random-LP protocol of the solver's benchmark runs (sigma mode); "default" is the library's own
PROTOCOL = learn.SIGMA_PROTOCOL
LP_PARAMS = {"eps": 1e-6, "l_inf_ruiz_iterations": 10}


# --------------------------------------------------------------------------- the cases

def listed():
    return [
        # a candidate point checked inside another program's loop: the smallest call, all latency
        {"name": "kkt_2k", "kind": "kkt", "m": 2000, "n": 5000, "per_col": 8},
        # the plain LP of the benchmark, solved again and again on one session (a parametric study):
        # launches and dependent loads bound it, in both forms
        {"name": "lp_2k_fp64", "kind": "lp", "family": "random", "m": 2000, "n": 5000, "per_col": 8, "iters": 1000,
         "precision": "fp64", "protocol": "default"},
        {"name": "lp_2k_fp32", "kind": "lp", "family": "random", "m": 2000, "n": 5000, "per_col": 8, "iters": 1000,
         "precision": "fp32_refine", "protocol": "default"},
        # the transportation family (200 x 200): columns of two entries, rows of 200
        {"name": "lp_transport_fp32", "kind": "lp", "family": "transport", "m": 200, "n": 200, "per_col": 2,
         "iters": 1000, "precision": "fp32_refine", "protocol": "sigma"},
        # an ordinary LP from host arrays: the whole call, upload and download included
        {"name": "lp_host_20k_fp64", "kind": "lp_host", "family": "random", "m": 20000, "n": 50000, "per_col": 8,
         "iters": 600, "precision": "fp64", "protocol": "default"},
        # the power-law LP at half the benchmark's size: larger than L2, long rows, badly scaled
        {"name": "lp_zipf_fp32", "kind": "lp", "family": "zipf", "m": 500000, "n": 1000000, "per_col": 10,
         "iters": 400, "precision": "fp32_refine", "protocol": "sigma"},
        {"name": "lp_zipf_fp64", "kind": "lp", "family": "zipf", "m": 500000, "n": 1000000, "per_col": 10,
         "iters": 400, "precision": "fp64", "protocol": "sigma"},
        # the convex QP at a quarter of and at the benchmark's size, from host arrays
        {"name": "qp_50k_fp64", "kind": "qp", "m": 25000, "n": 50000, "iters": 300, "precision": "fp64",
         "form": "sparse"},
        {"name": "qp_200k_fp32", "kind": "qp", "m": 100000, "n": 200000, "iters": 200, "precision": "fp32_refine",
         "form": "sparse"},
        # a batch of uneven LPs in one launch, one resident set of blocks
        {"name": "batch_300_fp32", "kind": "batch", "count": 300, "m_lo": 50, "m_hi": 5000, "iters": 400,
         "precision": "fp32_refine"},
        # an epoch of the warm-start network on the 40 x 40 family, and its use on held-out instances
        {"name": "train_40x40", "kind": "train", "supplies": 40, "demands": 40, "rows": 1024, "batch": 128},
        {"name": "warm_40x40", "kind": "warm", "supplies": 40, "demands": 40, "rows": 256, "bf16": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["kkt", "lp", "lp", "lp", "lp_host", "qp", "qp", "batch", "train", "grad", "predict", "warm"])
    if kind == "kkt":
        m = _log_int(rng, 50, 200000)
        return {"kind": kind, "m": m, "n": int(m * rng.uniform(1.5, 3)), "per_col": rng.randint(3, 20)}
    if kind in ("lp", "lp_host"):
        family = rng.choice(["random", "random", "transport", "zipf"]) if kind == "lp" else "random"
        iters = 200 * rng.randint(1, 4)
        case = {"kind": kind, "family": family, "precision": rng.choice(["fp64", "fp32_refine"]),
                "protocol": "sigma" if family == "zipf" else rng.choice(["default", "sigma"])}
        if family == "transport":
            return {**case, "m": rng.randint(12, 200), "n": rng.randint(12, 200), "per_col": 2, "iters": iters}
        if family == "zipf":
            m = _log_int(rng, 20000, 400000)
            return {**case, "m": m, "n": int(m * rng.uniform(1.5, 2.5)), "per_col": 10, "iters": min(iters, 400)}
        m = _log_int(rng, 50, 60000)
        return {**case, "m": m, "n": int(m * rng.uniform(2, 3)), "per_col": rng.randint(3, 20), "iters": iters}
    if kind == "qp":
        n = _log_int(rng, 500, 150000)
        return {"kind": kind, "m": int(n * rng.uniform(0.3, 0.6)), "n": n, "iters": 100 * rng.randint(1, 2),
                "precision": rng.choice(["fp64", "fp32_refine"]), "form": rng.choice(["sparse", "lowrank"])}
    if kind == "batch":
        hi = _log_int(rng, 200, 4000)
        return {"kind": kind, "count": _log_int(rng, 8, 300), "m_lo": 50, "m_hi": hi, "iters": 200,
                "precision": rng.choice(["fp64", "fp32_refine"])}
    s, d = rng.randint(12, 48), rng.randint(12, 48)
    if kind == "train":
        batch = rng.choice([64, 100, 128, 256])
        return {"kind": kind, "supplies": s, "demands": d, "rows": batch * rng.randint(1, 6) + rng.randint(0, 30),
                "batch": batch}
    if kind == "grad":
        return {"kind": kind, "supplies": s, "demands": d, "rows": _log_int(rng, 16, 512)}
    return {"kind": kind, "supplies": s, "demands": d, "rows": _log_int(rng, 1, 1500),
            "bf16": rng.choice([True, True, False])}


# --------------------------------------------------------------------------- inputs

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _csr_of_keys(key, m, n, values):
    """(row_ptr, col, val) on the host of the distinct keys row * n + col; values(rows, cols) on the device."""
    key = torch.unique(key)
    rows, cols = torch.div(key, n, rounding_mode="floor"), key % n
    rp = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    return rp.cpu().numpy().astype(np.int32), cols.cpu().numpy().astype(np.int32), values(rows, cols).cpu().numpy()


def _planted(rng, A, m, n, is_eq, lo, hi, free=None):
    """Objective and row bounds of a feasible and bounded LP (instances.random_lp's planting)."""
    rp, ci, v = A
    row_of = np.repeat(np.arange(m), np.diff(rp))
    base = np.where(np.isfinite(lo), lo, 0.0)
    top = np.where(np.isfinite(hi), hi, base + 5.0)
    x0 = base + rng.random(n) * np.minimum(top - base, 5.0)
    b = np.bincount(row_of, weights=v * x0[ci], minlength=m) + np.where(is_eq, 0.0, rng.random(m))
    y0 = rng.standard_normal(m)
    y0 = np.where(is_eq, y0, np.minimum(y0, 0.0))
    s = rng.random(n)
    if free is not None:
        s[free] = 0.0
    c = np.bincount(ci, weights=v * y0[row_of], minlength=n) + s
    return c, np.where(is_eq, b, -np.inf), b


def _random_blocks(ms, ns, per_col, seed):
    """One block-diagonal draw of random LPs (sizes ms, ns; per_col entries a column, a number or one
    per column): the LPs one by one."""
    g = _generator(seed)
    M, n_all = int(sum(ms)), int(sum(ns))
    ms_d = torch.tensor(ms, device=DEV)
    first_row = torch.cumsum(ms_d, 0) - ms_d
    owner = torch.repeat_interleave(torch.arange(len(ns), device=DEV), torch.tensor(ns, device=DEV))
    k = torch.as_tensor(np.broadcast_to(per_col, (n_all,)).copy(), device=DEV)
    cols = torch.repeat_interleave(torch.arange(n_all, device=DEV), k)
    own = owner[cols]
    u = torch.rand(cols.numel(), generator=g, device=DEV, dtype=torch.float64)
    rows = first_row[own] + torch.minimum((u * ms_d[own]).long(), ms_d[own] - 1)
    rp, ci, v = _csr_of_keys(rows * n_all + cols, M, n_all,
                             lambda r, c: torch.randn(r.numel(), generator=g, device=DEV, dtype=torch.float64))
    rng = np.random.default_rng(seed)
    out, r0, c0 = [], 0, 0
    for m, n in zip(ms, ns):
        k0, k1 = rp[r0], rp[r0 + m]
        A = (rp[r0:r0 + m + 1] - k0, ci[k0:k1] - c0, v[k0:k1])
        lo, hi = np.zeros(n), np.full(n, 10.0)
        c, cl, cu = _planted(rng, A, m, n, np.arange(m) < m // 2, lo, hi)
        out.append(lp.LPData(c, (*A, (m, n)), cl, cu, lo, hi))
        r0, c0 = r0 + m, c0 + n
    return out


def _zipf_lp(m, n, nnz, seed, max_row=20000):
    """instances.zipf_lp's structure (power-law rows, entries scaled by 10^U[-3,3] per row and column),
    drawn on the GPU."""
    g = _generator(seed)
    rng = np.random.default_rng(seed)
    z = rng.zipf(1.5, size=m).astype(np.float64)
    lo, hi = 1e-9, 1.0
    for _ in range(40):
        f = math.sqrt(lo * hi)
        lo, hi = (f, hi) if np.clip(np.round(z * f), 1, max_row).sum() < nnz else (lo, f)
    lens = torch.as_tensor(np.clip(np.round(z * math.sqrt(lo * hi)), 1, min(max_row, n)).astype(np.int64), device=DEV)
    rows = torch.repeat_interleave(torch.arange(m, device=DEV), lens)
    cols = torch.randint(0, n, (rows.numel(),), generator=g, device=DEV)
    rf = 10.0 ** (6 * torch.rand(m, generator=g, device=DEV, dtype=torch.float64) - 3)
    cf = 10.0 ** (6 * torch.rand(n, generator=g, device=DEV, dtype=torch.float64) - 3)
    A = _csr_of_keys(rows * n + cols, m, n, lambda r, c: rf[r] * cf[c] * torch.randn(
        r.numel(), generator=g, device=DEV, dtype=torch.float64))
    low, up = np.zeros(n), rng.uniform(1, 100, size=n)
    free = rng.random(n) < 0.05
    low[free], up[free] = -np.inf, np.inf
    c, cl, cu = _planted(rng, A, m, n, np.arange(m) < m // 2, low, up, free)
    return lp.LPData(c, (*A, (m, n)), cl, cu, low, up)


def _lp_data(case, seed):
    if case["family"] == "transport":
        return instances.transport_lp(case["m"], case["n"], seed=seed)
    if case["family"] == "zipf":
        return _zipf_lp(case["m"], case["n"], case["per_col"] * case["n"], seed)
    return _random_blocks([case["m"]], [case["n"]], case["per_col"], seed)[0]


def _batch_data(case, seed):
    rng = np.random.default_rng(case["count"])  # the sizes belong to the case, the instances to the seed
    ms = np.round(np.exp(rng.uniform(math.log(case["m_lo"]), math.log(case["m_hi"]), case["count"]))).astype(int)
    ms[0] = case["m_hi"]  # the largest instance bounds the launch
    ns = np.round(ms * rng.uniform(2, 3, case["count"])).astype(int)
    return _random_blocks(ms.tolist(), ns.tolist(), rng.integers(3, 21, size=int(ns.sum())), seed)


def _qp_data(case, seed):
    n = case["n"]
    return instances.planted_qp(n=n, m=case["m"], b_rows=n // 4, seed=seed, q_form=case["form"])[0]


def _params(case):
    return {**LP_PARAMS, "iteration_limit": case["iters"], "eps": 1e-12}


def _options(case):
    o = {"precision": case["precision"]}
    if case["precision"] == "fp32_refine":
        # the budget ends inside the FP32 phase, whatever the instance
        o.update(fp32_switch_tol=1e-12, fp32_stall_evals=0)
    return {**(PROTOCOL if case.get("protocol", "sigma") == "sigma" else {}), **o}


def _net_sizes(case):
    s, d = case["supplies"], case["demands"]
    return 2 * s * d + s + d, 256, s * d + s + d + 1


def _net_inputs(case, seed):
    """Network parameters (He-uniform weights, small biases) and standardised rows: features, and targets that
    depend on them."""
    inp, hid, out = _net_sizes(case)
    g = _generator(seed)
    u = lambda a, b, fan: (2 * torch.rand(a, b, generator=g, device=DEV) - 1) * math.sqrt(6.0 / fan)
    layers = []
    for a, b in ((inp, hid), (hid, hid), (hid, out)):
        layers += [u(a, b, a).reshape(-1), 0.01 * torch.randn(b, generator=g, device=DEV)]
    p = torch.cat(layers).cpu().numpy()
    X = torch.randn(case["rows"], inp, generator=g, device=DEV)
    Y = 0.6 * X[:, :out].contiguous() + 0.8 * torch.randn(case["rows"], out, generator=g, device=DEV)
    return p, X.cpu().numpy(), Y.cpu().numpy()


def _family(case, seed):
    """Instances of the transportation family, and the standardisation of a training set of them."""
    s, d = case["supplies"], case["demands"]
    items = instances.transport_family(s, d, [1000 * seed + k for k in range(case["rows"])])
    inp, _, out = _net_sizes(case)
    g = np.random.default_rng(seed + 7)
    f = np.stack([learn.features(i, s, d) for i in items[:64]])
    xm, xs = f.mean(0), f.std(0) + 0.05
    ym = np.concatenate([np.full(s * d, 0.03), g.normal(0.3, 0.1, s + d), [0.0]])
    ys = np.concatenate([np.full(s * d, 0.08), np.full(s + d, 0.2), [0.5]])
    return items, xm, xs, ym, ys


# --------------------------------------------------------------------------- one pass

def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": dict(case)}
    if kind == "kkt":
        d = _random_blocks([case["m"]], [case["n"]], case["per_col"], seed)[0]
        x = np.random.default_rng(seed + 1).uniform(0, 5, case["n"])
        dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV)
        rp, ci, v, _ = d.csr()
        state["in"] = [dev(a) for a in (rp, ci, v, d.con_lb, d.con_ub, d.c, x)]
        state["out"] = torch.empty(3, dtype=torch.float64, device=DEV)
        state["lib"] = N.load_lp()
    elif kind == "lp":
        state["session"] = lp.LPSession(_lp_data(case, seed), _params(case), _options(case))
    elif kind == "lp_host":
        state["data"] = _lp_data(case, seed)
    elif kind == "qp":
        state["data"] = _qp_data(case, seed)
    elif kind == "batch":
        state["data"] = _batch_data(case, seed)
    elif kind in ("train", "grad", "predict"):
        state["params"], state["X"], state["Y"] = _net_inputs(case, seed)
        state["mlp"] = learn.MLP(*_net_sizes(case), seed=1)
        if kind == "train":
            state["mlp"].set_data(state["X"], state["Y"])
        else:
            state["mlp"].set_params(state["params"])
    elif kind == "warm":
        state["items"], xm, xs, ym, ys = _family(case, seed)
        mlp = learn.MLP(*_net_sizes(case), seed=1)
        mlp.set_params(_net_inputs(dict(case, rows=1), seed)[0])
        state["start"] = learn.WarmStart(mlp, case["supplies"], case["demands"], xm, xs, ym, ys, 0.0, 0.0)
    else:
        raise ValueError(kind)
    return state


def _held(case, *vectors):
    """Vectors in the precision the phase they come from holds them in."""
    t = np.float32 if case["precision"] == "fp32_refine" else np.float64
    return [v.astype(t, copy=False) for v in vectors]


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "kkt":
        p = [C.c_void_p(t.data_ptr()) for t in (*state["in"], state["out"])]
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        if state["lib"].cp_al_gb300_primal_kkt_noalloc(case["m"], case["n"], *p, stream) != 0:
            raise RuntimeError(N.last_error(state["lib"]))
        return state["out"]
    if kind == "lp":
        r = state["session"].solve()
        x, y, rc = _held(case, *state["session"].fetch())
        return {"x": x, "y": y, "reduced_cost": rc, "iterations": r.iterations}
    if kind == "lp_host":
        r = lp.solve(state["data"], _params(case), _options(case))
        x, y, rc = _held(case, r.x, r.y, r.reduced_cost)
        return {"x": x, "y": y, "reduced_cost": rc, "iterations": r.iterations}
    if kind == "qp":
        o = _options({**case, "protocol": "default"})
        r = qp.solve(state["data"], {"eps": 1e-12, "iteration_limit": case["iters"]}, o)
        x, y = _held(case, r.x, r.y)
        return {"x": x, "y": y, "iterations": r.iterations}
    if kind == "batch":
        rs, _ = lp.solve_batch(state["data"], _params(case), {**_options(case), "spmv_nnz_per_block": 2048,
                                                              "batch_blocks_per_sm": 2})
        x, y = _held(case, np.concatenate([r.x for r in rs]), np.concatenate([r.y for r in rs]))
        return {"x": x, "y": y, "iterations": np.array([r.iterations for r in rs])}
    if kind == "train":
        state["mlp"].set_params(state["params"])
        loss = state["mlp"].train(1, case["batch"], 1e-3, 5)
        return {"params": state["mlp"].get_params(), "loss": loss}
    if kind == "grad":
        loss, grad = state["mlp"].loss_grad(state["X"], state["Y"])
        return {"loss": loss, "grad": grad}
    if kind == "predict":
        return {"y": state["mlp"].predict(state["X"], bf16=case["bf16"])}
    # the network's precision bounds what a warm start is worth: returned in 32 bits
    x, y, sigma, kp, kc = state["start"].predict_device(state["items"], bf16=case["bf16"])
    f = np.float32
    return {"x": x.astype(f), "y": y.astype(f), "sigma": sigma.astype(f), "kkt": kp.astype(f), "kkt_cold": kc}


# --------------------------------------------------------------------------- floors

def work(case):
    """Operations: two per nonzero and product, the epilogues' few per row and column.  Bytes: the inputs and
    outputs once; matrices that no cache of the chip holds are read by every iteration."""
    kind = case["kind"]
    if kind == "kkt":
        m, n, z = case["m"], case["n"], case["per_col"] * case["n"]
        return {"bytes": 12 * z + 20 * m + 16 * n, "flops": 2 * z + 4 * m + 2 * n}
    if kind in ("lp", "lp_host"):
        if case["family"] == "transport":
            m, n = case["m"] + case["n"], case["m"] * case["n"]
        else:
            m, n = case["m"], case["n"]
        z = case["per_col"] * n
        s = 4 if case["precision"] == "fp32_refine" else 8
        once = 12 * z + 8 * (5 * n + 4 * m)
        each = 2 * z * (s + 4) + 4 * (n + m) + s * (7 * n + 7 * m) + 8 * n + 16 * m
        return {"bytes": once + (case["iters"] * each if each > L2_BYTES else 0),
                "flops": case["iters"] * (4 * z + 12 * (n + m))}
    if kind == "qp":
        n, m = case["n"], case["m"]
        za, zq = 10 * n, int(7.2 * n)
        s = 4 if case["precision"] == "fp32_refine" else 8
        each = (2 * za + zq) * (s + 4) + s * (12 * n + 8 * m)
        return {"bytes": 12 * (za + zq) + 8 * (6 * n + 4 * m) + (case["iters"] * each if each > L2_BYTES else 0),
                "flops": case["iters"] * (4 * za + 2 * zq + 12 * (n + m))}
    if kind == "batch":
        # sizes are log-uniform: the mean of m, and 2.5 m columns of 11.5 entries
        lo, hi = case["m_lo"], case["m_hi"]
        m = case["count"] * (hi - lo) / math.log(hi / lo)
        n = 2.5 * m
        z = 11.5 * n
        return {"bytes": 12 * z + 8 * (5 * n + 4 * m), "flops": case["iters"] * (4 * z + 12 * (n + m))}
    inp, hid, out = _net_sizes(case)
    w = inp * hid + hid * hid + hid * out
    r = case["rows"]
    if kind == "train":
        steps = r // min(case["batch"], r)
        used = steps * min(case["batch"], r)
        return {"bytes": steps * 8 * 4 * w + 4 * used * (inp + out), "flops": used * (6 * w - 2 * inp * hid)}
    if kind == "grad":
        return {"bytes": 4 * (2 * w + r * (inp + out)), "flops": r * (6 * w - 2 * inp * hid)}
    if kind == "predict":
        return {"bytes": 4 * (w + r * (inp + out)), "flops": 2 * r * w}
    s, d = case["supplies"], case["demands"]
    return {"bytes": 4 * w + 8 * r * (3 * s * d + 2 * (s + d)), "flops": r * (2 * w + 20 * s * d)}


# --------------------------------------------------------------------------- 64-bit values

def _mt_normals(count):
    """The start vector of the sigma_max estimate: normal variates by Marsaglia's polar method over the
    32-bit words of MT19937 seeded with 1, two words a uniform (the low one first)."""
    want = int(count * 1.4) + 64
    while True:
        w = np.random.RandomState(1).randint(0, 2**32, size=4 * want, dtype=np.uint32).astype(np.float64)
        u = (w[0::2] + w[1::2] * 2.0**32) / 2.0**64
        a, b = 2 * u[0::2] - 1, 2 * u[1::2] - 1
        r2 = a * a + b * b
        ok = (r2 <= 1) & (r2 > 0)
        a, b, r2 = a[ok], b[ok], r2[ok]
        if 2 * a.size >= count:
            f = np.sqrt(-2 * np.log(r2) / r2)
            return np.stack([b * f, a * f], 1).reshape(-1)[:count]
        want *= 2


class _Csr:
    def __init__(self, rp, ci, v, shape):
        self.rp, self.ci, self.v, self.shape = rp, ci, v, shape
        self.row = torch.repeat_interleave(torch.arange(shape[0], device=DEV), rp[1:] - rp[:-1])

    def __matmul__(self, x):
        M = torch.sparse_csr_tensor(self.rp, self.ci, self.v, self.shape, check_invariants=False)
        return M @ x

    def rows(self, how, val):
        z = torch.zeros(self.shape[0], dtype=torch.float64, device=DEV)
        return z.scatter_reduce(0, self.row, val, how)

    def transposed(self):
        order = torch.sort(self.ci, stable=True).indices
        rp = torch.zeros(self.shape[1] + 1, dtype=torch.int64, device=DEV)
        rp[1:] = torch.cumsum(torch.bincount(self.ci, minlength=self.shape[1]), 0)
        return _Csr(rp, self.row[order], self.v[order], self.shape[::-1])


def _sigma_max_squared(A, At, lanczos):
    v = torch.as_tensor(_mt_normals(A.shape[0]), device=DEV)
    if not lanczos:  # power iteration on A A^T to an absolute residual of 1e-4
        s2 = 0.0
        for _ in range(5000):
            q = v / v.norm()
            v = A @ (At @ q)
            s2 = float(q @ v)
            if float((v - s2 * q).norm()) < 1e-4:
                break
        return s2
    q, last, al, be, prev = v / v.norm(), torch.zeros_like(v), [], [], -1.0
    limit = 128
    while True:
        for _ in range(16):
            w = A @ (At @ q)
            al.append(float(q @ w))
            r = w - al[-1] * q - (be[-1] if be else 0.0) * last
            be.append(float(r.norm()))
            last, q = q, (r / be[-1] if be[-1] > 0 else r)
        k = next((i + 1 for i, b in enumerate(be) if not b > 0), len(al))
        T = np.diag(al[:k]) + np.diag(be[:k - 1], 1) + np.diag(be[:k - 1], -1)
        theta = float(np.linalg.eigvalsh(T)[-1])
        if k < len(al) or be[k - 1] <= 1e-12 * theta or len(al) >= limit or len(al) >= A.shape[0] or (
                prev > 0 and abs(theta - prev) <= 1e-8 * theta):
            return theta
        prev = theta


def _lp_exact(data, case):
    """The restarted reflected Halpern iteration in 64 bits: equilibration (10 Ruiz passes,
    Pock-Chambolle, bound and objective scaling), step sizes, evaluation blocks of 200 iterations with the restart
    rule and the weight (or sigma) controller, the unscaled result."""
    lanczos = case["precision"] == "fp32_refine"
    o = {"al_lambda": 0.05, **(PROTOCOL if case["protocol"] == "sigma" else {})}
    t = lambda a, ty=torch.float64: torch.as_tensor(np.ascontiguousarray(a), device=DEV).to(ty)
    rp, ci, v, (m, n) = data.csr()
    A = _Csr(t(rp, torch.int64), t(ci, torch.int64), t(v), (m, n))
    At = A.transposed()
    c, vl, vu, cl, cu = (t(a) for a in (data.c, data.var_lb, data.var_ub, data.con_lb, data.con_ub))
    vl_raw, vu_raw = vl, vu
    obj_norm = float(c.norm())
    lo_part = torch.where(torch.isfinite(cl) & (cl != cu), cl, torch.zeros_like(cl))
    bnd_norm = math.sqrt(float((lo_part**2).sum()) + float((torch.where(torch.isfinite(cu), cu, torch.zeros_like(cu))**2).sum()))
    D, R = torch.ones_like(c), torch.ones_like(cl)
    for k in range(11):
        how = "amax" if k < 10 else "sum"
        r = A.rows(how, A.v.abs()) if how == "amax" else A.rows("sum", A.v.abs())
        d = At.rows(how, At.v.abs())
        r, d = (torch.where(z < 1e-12, torch.ones_like(z), z.sqrt()) for z in (r, d))
        A.v = A.v / (r[A.row] * d[A.ci])
        At.v = At.v / (d[At.row] * r[At.ci])
        D, R, c, vl, vu, cl, cu = D * d, R * r, c / d, vl * d, vu * d, cl / r, cu / r
    fl, fu = torch.isfinite(cl), torch.isfinite(cu)
    zero = torch.zeros_like(cl)
    bsum = torch.where(fl & (~fu | ((cl - cu).abs() > 1e-12)), cl**2, zero) + torch.where(fu, cu**2, zero)
    cbr, ovr = 1 / (math.sqrt(float(bsum.sum())) + 1), 1 / (float(c.norm()) + 1)
    c, vl, vu, cl, cu = c * ovr, vl * cbr, vu * cbr, cl * cbr, cu * cbr
    clf, cuf = (torch.where(torch.isfinite(z), z, torch.zeros_like(z)) for z in (cl, cu))
    lam = _sigma_max_squared(A, At, lanczos)

    margin, pw, sigma, lp_ = 0.998 * 0.998, 1.0, 0.0, 0.0
    sig_on = bool(o.get("sigma_mode"))
    if sig_on:
        lp_ = max(o["lambda_factor"] * lam, (2 + 1e-12) * lam)
        base = 1 / math.sqrt(lp_)
        lo_s, hi_s = o["sigma_min_factor"] * base, o["sigma_max_factor"] * base
        sigma = min(max(o["sigma_init_factor"] * base, lo_s), hi_s)

    def schedule():
        nonlocal pw
        if sig_on:
            tau = 1 / (sigma * lp_)
            pw = math.sqrt(sigma / tau)
            return math.sqrt(tau * sigma), sigma
        step = math.sqrt(margin * (1 - o["al_lambda"]) / lam)
        return step, step * pw * o["al_lambda"] / (1 - o["al_lambda"])

    step, beta = schedule()
    best = {"pw": pw, "sigma": sigma, "gap": math.inf}
    e_sum = e_last = 0.0
    x = torch.zeros_like(c)
    y = torch.zeros_like(cl)
    x0, y0, ax = x, y, A @ x
    clip = lambda z, a, b: torch.maximum(a, torch.minimum(z, b))
    inner, total, fp0, fp_last = 0, 0, 0.0, math.inf
    rp_ = {"suff": o.get("restart_sufficient", 0.2), "nec": o.get("restart_necessary", 0.5),
           "art": o.get("restart_artificial", 0.36)}
    while True:
        tau, rho = step / pw, step * pw
        for i in range(1, 201):
            w = (inner + i) / (inner + i + 1)
            u = y - beta * (ax - clip(ax - y / beta, cl, cu)) if beta > 0 else y
            tpt = x - tau * (c - At @ u)
            xh = clip(tpt, vl, vu)
            lam_x = (xh - tpt) / tau
            xb = 2 * xh - x
            p = A @ xb
            yh = y - rho * (p - clip(p - y / (rho + beta), cl, cu))
            yb = 2 * yh - y
            x, y = w * xb + (1 - w) * x0, w * yb + (1 - w) * y0
            if beta > 0:
                ax = A @ x
        inner, total = inner + 200, total + 200
        if total >= case["iters"]:
            break
        ph, dx, dy = A @ xh, xb - xh, yb - yh
        q, adx, ady = At @ yh, A @ dx, At @ dy
        nrm = lambda z: float((z * z).sum())

        def fixed_point():
            if sig_on:
                return math.sqrt(max(sigma * (lp_ * nrm(dx) - nrm(adx)) + nrm(dy) / sigma, 0.0))
            return math.sqrt(max(nrm(dx) * pw + nrm(dy) / pw + 2 * step * float(ady @ dx) - step * beta * nrm(adx), 0.0))

        fp = fixed_point()
        rel_p = math.sqrt(nrm((ph - clip(ph, cl, cu)) * R)) / cbr / (1 + bnd_norm)
        rel_d = math.sqrt(nrm((c - q - lam_x) * D)) / ovr / (1 + obj_norm)
        again = total == 200 or fp <= rp_["suff"] * fp0 or (fp <= rp_["nec"] * fp0 and fp > fp_last) or \
            inner >= rp_["art"] * total
        fp_last = fp
        if again:
            pd, dd, ratio = (xh - x0).norm().item(), (yh - y0).norm().item(), rel_d / max(rel_p, 1e-300)
            gap = abs(math.log10(max(rel_d, 1e-300) / max(rel_p, 1e-300)))
            if sig_on:
                dxm = lp_ * pd * pd - nrm(A @ (xh - x0))
                if 1e-16 < dd < 1e12 and 1e-24 < dxm < 1e24 and 1e-8 < ratio < 1e8:
                    err = math.log(dd) - 0.5 * math.log(dxm) - math.log(sigma)
                    err += o["sigma_balance_gain"] * max(-2.0, min(0.5 * math.log(ratio), 2.0))
                    e_sum = 0.3 * e_sum + err
                    sr = math.exp(o["sigma_kp"] * err + o["sigma_ki"] * e_sum + o["sigma_kd"] * (err - e_last))
                    sigma *= min(max(sr, o["sigma_update_min"]), o["sigma_update_max"])
                    e_last = err
                else:
                    sigma, e_sum, e_last = best["sigma"], 0.0, 0.0
                sigma = min(max(sigma, lo_s), hi_s)
            elif 1e-16 < pd < 1e12 and 1e-16 < dd < 1e12 and 1e-8 < ratio < 1e8:
                err = math.log(dd) - math.log(pd) - math.log(pw)
                e_sum = 0.3 * e_sum + err
                pw *= math.exp(0.99 * err + 0.01 * e_sum)
            else:
                pw, e_sum = best["pw"], 0.0
            if gap < best["gap"]:
                best = {"pw": pw, "sigma": sigma, "gap": gap}
            step, beta = schedule()
            inner, fp_last, fp0 = 0, math.inf, fixed_point()
            x, y, x0, y0, ax = xh, yh, xh, yh, ph
    rc = (c - At @ yh) * D / ovr
    rc = torch.where(torch.isfinite(vl_raw), rc, rc.clamp(max=0.0))
    rc = torch.where(torch.isfinite(vu_raw), rc, rc.clamp(min=0.0))
    return {"x": xh / D / cbr, "y": yh / R / ovr, "reduced_cost": rc, "iterations": None}


def _net_exact(p, X, case):
    inp, hid, out = _net_sizes(case)
    p = torch.as_tensor(p, device=DEV).double()
    X = torch.as_tensor(X, device=DEV).double()
    parts = torch.split(p, [inp * hid, hid, hid * hid, hid, hid * out, out])
    parts = [q.clone().requires_grad_(True) for q in parts]
    h = torch.relu(X @ parts[0].view(inp, hid) + parts[1])
    h = torch.relu(h @ parts[2].view(hid, hid) + parts[3])
    return h @ parts[4].view(hid, out) + parts[5], parts


def exact(case, seed):
    kind = case["kind"]
    if kind == "kkt":
        s = prepare(case, seed)
        rp, ci, v, lo, hi, c, x = (a.cpu().numpy() for a in s["in"])
        ax = np.bincount(np.repeat(np.arange(case["m"]), np.diff(rp)), weights=v * x[ci], minlength=case["m"])
        r = ax - np.clip(ax, lo, hi)
        return np.array([np.linalg.norm(r), np.abs(r).max(), c @ x])
    if kind in ("lp", "lp_host"):
        return _lp_exact(_lp_data(case, seed), case)
    if kind == "grad":
        p, X, Y = _net_inputs(case, seed)
        P, parts = _net_exact(p, X, case)
        loss = ((P - torch.as_tensor(Y, device=DEV).double())**2).mean()
        grad = torch.cat(torch.autograd.grad(loss, parts))
        return {"loss": loss.item(), "grad": grad}
    if kind == "predict":
        p, X, _ = _net_inputs(case, seed)
        return {"y": _net_exact(p, X, case)[0].detach()}
    if kind == "warm":
        s, d = case["supplies"], case["demands"]
        items, xm, xs, ym, ys = _family(case, seed)
        X = (np.stack([learn.features(i, s, d) for i in items]) - xm) / xs
        P = _net_exact(_net_inputs(dict(case, rows=1), seed)[0], X, case)[0].detach().cpu().numpy() * ys + ym
        cap = np.stack([i.var_ub for i in items])
        cost = np.stack([i.c for i in items])
        b = np.stack([i.con_ub for i in items])
        x = np.clip(P[:, :s * d], 0, 1) * cap
        y = P[:, s * d:-1] * 100

        def kkt(x, y):
            g = x.reshape(-1, s, d)
            res = np.linalg.norm(np.concatenate([g.sum(2), g.sum(1)], 1) - b, axis=1) / (1 + np.linalg.norm(b, axis=1))
            rc = cost - (y[:, :s, None] + y[:, None, s:]).reshape(len(y), -1)
            po, do = (cost * x).sum(1), (b * y).sum(1) + (np.minimum(rc, 0) * cap).sum(1)
            return np.maximum(res, np.abs(po - do) / (1 + np.abs(po) + np.abs(do)))

        return {"x": x, "y": y, "sigma": np.exp(P[:, -1]), "kkt": kkt(x, y), "kkt_cold": kkt(0 * x, 0 * y)}
    # QP: the inner projected Barzilai-Borwein loop stops by its own residuals.  Batch: hundreds of power
    # iterations and solves one after the other take far over 20 seconds.  Train: the mini-batches are the
    # library's own shuffle.
    return None
