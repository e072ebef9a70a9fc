"""Performance cases of the device interior-point engine.

One case is one call (or the short fixed sequence of calls) that a program makes through the
public binding: the Newton system of one IPM iteration (factorise A diag(theta) A^T, solve for
the predictor and the corrector), the products A x and A^T y, the learned-start network's
prediction and gradient, and whole LP solves, alone and as a batch. Sizes are those of the
repository's own workloads: LPs with m ~ logUniform[200, 5000] rows, n = m U[2, 3] columns and
0.5-2 % density, the 500 x 1000 LP, and block-angular LPs of 500 x 1200 blocks with linking rows.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs and the handle that a program keeps (plan, solver, weights)
    run(state)           one pass, with its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    what run() computes, in 64-bit torch / numpy
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "soverign-gpu-accelerator-_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

WEIGHTS = os.path.join(PKG, "weights", "learned_start_family3.npy")
PRECISIONS = ("fp64", "tensor", "mixed")
SOLVE_TOL = 1e-11      # relative residual asked of a Newton solve
THETA_LOG = 4.0        # theta = x / s between exp(-4) and exp(4): the middle of an IPM run
LP_ITERS = 14          # iterations of an IPM run on these families, for work()


def _sk():
    import sankhya_gb300
    return sankhya_gb300


# ------------------------------------------------------------------------- the cases

def listed():
    return [
        # The Newton system of a small LP, called with host arrays: the latency of one step.
        {"name": "newton_small_host", "kind": "newton", "m": 300, "n": 700, "density": 0.02, "precision": "fp64",
         "host": True},
        # A mid-sized dense normal matrix in plain FP64, a ragged size, device arrays.
        {"name": "newton_fp64", "kind": "newton", "m": 1447, "n": 3613, "density": 0.012, "precision": "fp64",
         "host": False},
        # The largest family member in plain FP64: the reference's arithmetic at full size.
        {"name": "newton_fp64_large", "kind": "newton", "m": 4001, "n": 10002, "density": 0.01, "precision": "fp64",
         "host": False},
        # The FP64 factorisation of a mixed-precision solve's last iterations (tensor-core updates).
        {"name": "newton_tensor", "kind": "newton", "m": 4740, "n": 12011, "density": 0.01, "precision": "tensor",
         "host": False},
        # The early iterations of a mixed-precision solve: FP32 factor, FP64 refinement.
        {"name": "newton_mixed", "kind": "newton", "m": 2999, "n": 7411, "density": 0.015, "precision": "mixed",
         "host": False},
        # A block-angular LP: the sparse multifrontal path with a dense root front.
        {"name": "newton_blocks", "kind": "blocks", "blocks": 12, "rows": 500, "cols": 1200, "links": 600,
         "precision": "mixed"},
        # A x and A^T y of the 500 x 1000 LP: launch latency.
        {"name": "spmv_small", "kind": "spmv", "lps": 1, "m": 500, "n": 1000, "density": 0.01},
        # A x and A^T y of a batch of large LPs as one matrix, more than the L2 holds.
        {"name": "spmv_batch", "kind": "spmv", "lps": 24, "m": 4973, "n": 12431, "density": 0.02},
        # The learned start of one mid-sized LP.
        {"name": "gnn_predict", "kind": "gnn", "lps": 1, "m": 2011, "n": 5003, "density": 0.012, "train": False},
        # One training batch of 16 LPs: loss and gradients.
        {"name": "gnn_train", "kind": "gnn", "lps": 16, "m": 1201, "n": 3001, "density": 0.012, "train": True},
        # One 500 x 1000 LP to 1e-8 in plain FP64: the smallest whole solve.
        {"name": "lp_single", "kind": "lp", "lps": 1, "m_lo": 500, "m_hi": 500, "ratio": 2.0, "density": 0.01,
         "precision": "fp64"},
        # An uneven batch solved at once in mixed precision from the learned start.
        {"name": "lp_batch", "kind": "lp", "lps": 40, "m_lo": 200, "m_hi": 4400, "ratio": 2.5, "density": 0.012,
         "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["newton", "newton", "newton", "blocks", "spmv", "gnn", "lp"])
    m = _log_int(rng, 200, 5000)
    n = int(math.ceil(m * rng.uniform(2.0, 3.0)))
    density = round(rng.uniform(0.005, 0.02), 4)
    if kind == "newton":
        return {"kind": kind, "m": m, "n": n, "density": density, "precision": rng.choice(PRECISIONS),
                "host": rng.random() < 0.3}
    if kind == "blocks":
        rows = rng.randint(200, 500)
        return {"kind": kind, "blocks": rng.randint(2, 12), "rows": rows, "cols": int(rows * rng.uniform(2.0, 2.6)),
                "links": rng.randint(50, 600), "precision": rng.choice(PRECISIONS)}
    if kind == "spmv":
        return {"kind": kind, "lps": _log_int(rng, 1, 24), "m": m, "n": n, "density": density}
    if kind == "gnn":
        m = _log_int(rng, 200, 2400)
        return {"kind": kind, "lps": rng.randint(1, 12), "m": m, "n": int(math.ceil(m * rng.uniform(2.0, 3.0))),
                "density": density, "train": rng.random() < 0.6}
    lps = _log_int(rng, 1, 24)
    return {"kind": kind, "lps": lps, "m_lo": 200, "m_hi": _log_int(rng, 260, 2500),
            "ratio": round(rng.uniform(2.1, 3.0), 3), "density": round(rng.uniform(0.01, 0.02), 4),
            "precision": rng.choice(("fp64", "mixed"))}


# ------------------------------------------------------------------------- inputs

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 2654435761 % (1 << 62))
    return g


def _signed(count, g):
    """Nonzeros +-U[0.1, 10]."""
    v = torch.rand(count, generator=g, device=_device(), dtype=torch.float64) * 9.9 + 0.1
    return torch.where(torch.rand(count, generator=g, device=_device()) < 0.5, -v, v)


def _entries(m, n, per_col, g):
    """(rows, cols) of a random pattern sorted by column, then row: about per_col distinct rows a
    column, and at least one entry in every row."""
    dev = _device()
    rows = torch.randint(0, m, (n, per_col), generator=g, device=dev)
    cols = torch.arange(n, device=dev).repeat_interleave(per_col)
    cover = torch.randint(0, n, (m,), generator=g, device=dev)
    key = torch.cat([cols * m + rows.reshape(-1), cover * m + torch.arange(m, device=dev)])
    key = torch.unique(key)
    return key % m, key // m


def _lp(m, n, density, seed):
    """A feasible, bounded LP min c.x, A x = b, x >= 0: CSC tensors (col_ptrs, rows, cols, vals, b, c)."""
    g = _gen(seed)
    dev = _device()
    rows, cols = _entries(m, n, min(m, max(2, int(round(density * m)))), g)
    vals = _signed(rows.numel(), g)
    return _finish(m, n, rows, cols, vals, g, dev)


def _finish(m, n, rows, cols, vals, g, dev):
    x0 = torch.rand(n, generator=g, device=dev, dtype=torch.float64) * 1.5 + 0.5
    y0 = torch.randn(m, generator=g, device=dev, dtype=torch.float64)
    s0 = torch.rand(n, generator=g, device=dev, dtype=torch.float64) * 0.9 + 0.1
    b = np.bincount(rows.cpu().numpy(), weights=(vals * x0[cols]).cpu().numpy(), minlength=m)
    c = np.bincount(cols.cpu().numpy(), weights=(vals * y0[rows]).cpu().numpy(), minlength=n) + s0.cpu().numpy()
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    ptr[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0)
    return {"m": m, "n": n, "ptr": ptr, "rows": rows, "cols": cols, "vals": vals, "b": b, "c": c}


def _blocks(case, seed):
    """A block-angular LP: dense-ish diagonal blocks with 5 entries a column, and one linking entry
    in every column."""
    g = _gen(seed)
    dev = _device()
    nb, r, c, links = case["blocks"], case["rows"], case["cols"], case["links"]
    m, n = nb * r + links, nb * c
    keys = []
    for k in range(nb):
        rows, cols = _entries(r, c, 5, g)
        keys.append((cols + k * c) * m + rows + k * r)
    link_rows = torch.randint(0, links, (n,), generator=g, device=dev)
    link_rows[torch.randperm(n, generator=g, device=dev)[:links]] = torch.arange(links, device=dev)
    keys.append(torch.arange(n, device=dev) * m + nb * r + link_rows)
    key = torch.unique(torch.cat(keys))
    rows, cols = key % m, key // m
    return _finish(m, n, rows, cols, _signed(rows.numel(), g), g, dev)


def _csr(lp):
    """(row_ptrs, col_idx, vals) of A by row, columns ascending, as device tensors."""
    order = torch.argsort(lp["rows"] * lp["n"] + lp["cols"])
    ptr = torch.zeros(lp["m"] + 1, dtype=torch.int64, device=lp["rows"].device)
    ptr[1:] = torch.cumsum(torch.bincount(lp["rows"], minlength=lp["m"]), 0)
    return ptr, lp["cols"][order], lp["vals"][order]


def _np32(t):
    return t.to(torch.int32).cpu().numpy()


def _newton_vectors(m, n, seed):
    g = _gen(seed + 7919)
    dev = _device()
    theta = torch.exp((torch.rand(n, generator=g, device=dev, dtype=torch.float64) * 2 - 1) * THETA_LOG)
    rhs = torch.randn(2, m, generator=g, device=dev, dtype=torch.float64)
    return theta, rhs


def _stack(lps):
    """Block-diagonal matrix of several LPs."""
    ro = np.cumsum([0] + [lp["m"] for lp in lps])
    co = np.cumsum([0] + [lp["n"] for lp in lps])
    rows = torch.cat([lp["rows"] + int(r) for lp, r in zip(lps, ro)])
    cols = torch.cat([lp["cols"] + int(c) for lp, c in zip(lps, co)])
    m, n = int(ro[-1]), int(co[-1])
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=rows.device)
    ptr[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0)
    return {"m": m, "n": n, "ptr": ptr, "rows": rows, "cols": cols, "vals": torch.cat([lp["vals"] for lp in lps]),
            "b": np.concatenate([lp["b"] for lp in lps]), "c": np.concatenate([lp["c"] for lp in lps])}


def _sizes(case):
    """Rows and columns of each LP of a batch: spread evenly over the logarithm of the row count."""
    k = case["lps"]
    out = []
    for i in range(k):
        t = i / (k - 1) if k > 1 else 1.0
        m = int(round(case["m_lo"] * (case["m_hi"] / case["m_lo"]) ** t))
        out.append((m, int(math.ceil(m * case["ratio"]))))
    return out


def _scaled(lp):
    """The LP after three passes of row / column equilibration: what the network is given."""
    r, c = lp["rows"].cpu().numpy(), lp["cols"].cpu().numpy()
    v, b, cc = lp["vals"].cpu().numpy().copy(), lp["b"].copy(), lp["c"].copy()
    for _ in range(3):
        rm, cm = np.zeros(lp["m"]), np.zeros(lp["n"])
        np.maximum.at(rm, r, np.abs(v))
        np.maximum.at(cm, c, np.abs(v))
        rm, cm = 1.0 / np.sqrt(rm), 1.0 / np.sqrt(np.where(cm > 0, cm, 1.0))
        v *= rm[r] * cm[c]
        b *= rm
        cc *= cm
    return dict(lp, vals=torch.from_numpy(v).to(lp["vals"].device), b=b, c=cc)


def _gnn_inputs(case, seed):
    lp = _scaled(_stack([_lp(case["m"], case["n"], case["density"], seed * 64 + k) for k in range(case["lps"])]))
    rng = np.random.default_rng(seed)
    targets = None
    if case["train"]:
        targets = (rng.normal(0.0, 2.0, lp["n"]), rng.normal(0.0, 2.0, lp["n"]), rng.normal(0.0, 1.0, lp["m"]))
    return lp, targets


def prepare(case, seed):
    sk = _sk()
    kind = case["kind"]
    if kind in ("newton", "blocks"):
        lp = _lp(case["m"], case["n"], case["density"], seed) if kind == "newton" else _blocks(case, seed)
        ptr, ci, v = _csr(lp)
        mixed = case["precision"] == "mixed"
        kkt = sk.Kkt(lp["m"], lp["n"], _np32(ptr), _np32(ci), v.cpu().numpy(),
                     precision=sk.PREC_MIXED if mixed else sk.PREC_FP64)
        if case["precision"] == "tensor":
            kkt.set_fp64_update(sk.FP64_UPDATE_TENSOR)
        theta, rhs = _newton_vectors(lp["m"], lp["n"], seed)
        host = bool(case.get("host"))
        if host:
            theta, rhs = theta.cpu().numpy(), rhs.cpu().numpy()
        return {"kind": "newton", "host": host, "kkt": kkt, "theta": theta, "rhs": rhs,
                "out": None if host else torch.empty_like(rhs)}
    if kind == "spmv":
        lp = _stack([_lp(case["m"], case["n"], case["density"], seed * 64 + k) for k in range(case["lps"])])
        ptr, ci, v = _csr(lp)
        mats, nnz = [], v.numel()
        g = _gen(seed + 104729)
        for rows, cols, p, i, w in ((lp["m"], lp["n"], ptr, ci, v),
                                    (lp["n"], lp["m"], lp["ptr"], lp["rows"], lp["vals"])):
            p, i, w = p.to(torch.int32), i.to(torch.int32), w.contiguous()
            x = torch.randn(cols, generator=g, device=w.device, dtype=torch.float64)
            y = torch.zeros(rows, device=w.device, dtype=torch.float64)
            torch.cuda.current_stream().synchronize()
            plan = sk.SpmvPlan(rows, cols, nnz, p.data_ptr(), i.data_ptr(), w.data_ptr())
            mats.append((plan, x, y, (p, i, w)))
        return {"kind": kind, "mats": mats}
    if kind == "gnn":
        lp, targets = _gnn_inputs(case, seed)
        ptr, ci, v = _csr(lp)
        net = sk.Gnn(1)
        net.load(WEIGHTS)
        batch = sk.GnnBatch.from_arrays(lp["m"], lp["n"], _np32(ptr), _np32(ci), v.cpu().numpy(), lp["b"], lp["c"],
                                        targets)
        return {"kind": kind, "train": case["train"], "net": net, "batch": batch}
    lps = [_sk_lp(sk, _lp(m, n, case["density"], seed * 64 + k)) for k, (m, n) in enumerate(_sizes(case))]
    if case["precision"] == "mixed":
        net = sk.Gnn(1)
        net.load(WEIGHTS)
        solver = sk.Solver(lps, precision=sk.PREC_MIXED, start=sk.START_LEARNED)
        solver.set_gnn(net)
    else:
        net = None
        solver = sk.Solver(lps, precision=sk.PREC_FP64, start=sk.START_MEHROTRA)
    return {"kind": "lp", "solver": solver, "net": net}


def _sk_lp(sk, lp):
    return sk.LP(lp["m"], lp["n"], _np32(lp["ptr"]), _np32(lp["rows"]), lp["vals"].cpu().numpy(), lp["b"], lp["c"])


# ------------------------------------------------------------------------- one pass

def run(state):
    kind = state["kind"]
    if kind == "newton":
        return _run_host(state) if state["host"] else _run_device(state)
    if kind == "spmv":
        for plan, x, y, _ in state["mats"]:
            plan.execute(x.data_ptr(), y.data_ptr())
        return [y for _, _, y, _ in state["mats"]]
    if kind == "gnn":
        if state["train"]:
            loss, grad = state["net"].loss_grad(state["batch"])
            return {"loss": loss, "grad": grad}
        return list(state["net"].predict(state["batch"]))
    solver = state["solver"]
    solver.run()
    got = [solver.result(k) for k in range(len(solver.lps))]
    return {"x": np.concatenate([r[1] for r in got]), "y": np.concatenate([r[2] for r in got]),
            "s": np.concatenate([r[3] for r in got]), "objective": np.array([r[0]["objective"] for r in got])}


def _run_host(state):
    sk, kkt = _sk(), state["kkt"]
    sk.check(kkt.factorize(state["theta"]), "sk_kkt_factorize")
    out = []
    for rhs in state["rhs"]:                  # predictor, corrector
        rc, dy = kkt.solve(rhs, tol=SOLVE_TOL)
        sk.check(rc, "sk_kkt_solve")
        out.append(dy)
    return out


def _run_device(state):
    sk, kkt, out = _sk(), state["kkt"], state["out"]
    lib = sk.lib()
    out.copy_(state["rhs"])                    # the engine solves in place, on a stream of its own
    torch.cuda.current_stream().synchronize()
    sk.check(lib.sk_kkt_factorize_device(kkt.h, state["theta"].data_ptr()), "sk_kkt_factorize_device")
    for k in range(2):                         # predictor, corrector
        sk.check(lib.sk_kkt_solve_device(kkt.h, out[k].data_ptr(), SOLVE_TOL), "sk_kkt_solve_device")
    return [out[0], out[1]]


# ------------------------------------------------------------------------- work and reference

def _dense_work(m, n, density):
    """(bytes, flops) of forming A diag(theta) A^T, factoring it and two solves, m x m dense."""
    per = max(2.0, density * m)
    flops = n * per * per + m ** 3 / 3.0 + 2 * (2.0 * m * m + 4.0 * n * per)
    return 12.0 * n * per + 8.0 * n + 2 * 16.0 * m, flops


def work(case):
    kind = case["kind"]
    if kind == "newton":
        b, f = _dense_work(case["m"], case["n"], case["density"])
        return {"bytes": b, "flops": f}
    if kind == "blocks":
        nb, r, links = case["blocks"], case["rows"], case["links"]
        n = nb * case["cols"]
        # each block is dense once factored, and so is the linking part it updates
        flops = nb * (r ** 3 / 3.0 + 1.0 * r * r * links + 1.0 * r * links * links) + links ** 3 / 3.0
        entries = nb * (r * r / 2.0 + r * links) + links * links / 2.0
        return {"bytes": 12.0 * 6 * n + 8.0 * n + 32.0 * (nb * r + links), "flops": flops + 2 * 4.0 * entries}
    per = max(2, int(round(case["density"] * case.get("m", 0))))
    if kind == "spmv":
        m, n = case["lps"] * case["m"], case["lps"] * case["n"]
        nnz = n * per
        return {"bytes": 2 * (12.0 * nnz + 8.0 * (m + n)) + 4.0 * (m + n), "flops": 4.0 * nnz}
    if kind == "gnn":
        m, n = case["lps"] * case["m"], case["lps"] * case["n"]
        nnz = n * per
        forward = 3 * (2 * 2.0 * nnz * 64 + 2 * (m + n) * 2 * 64 * 64)
        return {"bytes": 12.0 * nnz + 8.0 * (m + n) + 4.0 * 50243 + 8.0 * (m + 2 * n),
                "flops": forward * (3 if case["train"] else 1)}
    b = f = 0.0
    for m, n in _sizes(case):
        db, df = _dense_work(m, n, case["density"])
        b += 12.0 * n * max(2.0, case["density"] * m) + 8.0 * (2 * m + 3 * n)
        f += LP_ITERS * df
    return {"bytes": b, "flops": f}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("newton", "blocks"):
        lp = _lp(case["m"], case["n"], case["density"], seed) if kind == "newton" else _blocks(case, seed)
        theta, rhs = _newton_vectors(lp["m"], lp["n"], seed)
        a = torch.zeros(lp["m"], lp["n"], dtype=torch.float64, device=theta.device)
        a[lp["rows"], lp["cols"]] = lp["vals"]
        normal = (a * theta) @ a.T
        x = torch.linalg.solve(normal, rhs.T)
        for _ in range(2):                     # refined, so that it is better than one solve's rounding
            x = x + torch.linalg.solve(normal, rhs.T - a @ (theta[:, None] * (a.T @ x)))
        x = x.T
        return [x[0].cpu().numpy(), x[1].cpu().numpy()] if case.get("host") else [x[0], x[1]]
    if kind == "spmv":
        lp = _stack([_lp(case["m"], case["n"], case["density"], seed * 64 + k) for k in range(case["lps"])])
        g = _gen(seed + 104729)
        x = torch.randn(lp["n"], generator=g, device=lp["vals"].device, dtype=torch.float64)
        y = torch.randn(lp["m"], generator=g, device=lp["vals"].device, dtype=torch.float64)
        ax = torch.zeros(lp["m"], dtype=torch.float64, device=x.device).index_add_(0, lp["rows"],
                                                                                  lp["vals"] * x[lp["cols"]])
        aty = torch.zeros(lp["n"], dtype=torch.float64, device=x.device).index_add_(0, lp["cols"],
                                                                                   lp["vals"] * y[lp["rows"]])
        return [ax, aty]
    if kind == "gnn":
        return _gnn_exact(case, seed)
    if case["lps"] > 1 or case["m_hi"] > 600:
        return None                            # a reference optimum of every member would take minutes
    m, n = _sizes(case)[0]
    return _optimum(_lp(m, n, case["density"], seed * 64))


def _gnn_exact(case, seed):
    """The network in 64 bits: BF16 weights, two linear maps and a ReLU per layer and side."""
    lp, targets = _gnn_inputs(case, seed)
    m, n, h = lp["m"], lp["n"], 64
    w = torch.from_numpy(np.load(WEIGHTS)).to(torch.bfloat16).to(torch.float64).to(lp["vals"].device)
    w.requires_grad_(case["train"])
    at = [0]

    def take(*shape):
        count = math.prod(shape)
        at[0] += count
        return w[at[0] - count:at[0]].reshape(shape)

    ec_w, ec_b, er_w, er_b = take(h, 3), take(h), take(h, 3), take(h)
    layers = [[take(h, h), take(h, h), take(h), take(h, h), take(h, h), take(h)] for _ in range(3)]
    hc_w, hc_b, hr_w, hr_b = take(2, h), take(2), take(1, h), take(1)
    ptr, ci, v = _csr(lp)
    a = torch.sparse_csr_tensor(ptr, ci, v, (m, n))
    at_ = torch.sparse_csr_tensor(lp["ptr"], lp["rows"], lp["vals"], (n, m))
    deg_r = torch.bincount(lp["rows"], minlength=m).double()
    deg_c = torch.bincount(lp["cols"], minlength=n).double()

    def norms(idx, count):
        return torch.zeros(count, dtype=torch.float64, device=v.device).index_add_(0, idx, lp["vals"] ** 2).sqrt()

    fc = torch.stack([torch.from_numpy(lp["c"]).to(v.device), torch.log(1 + deg_c), norms(lp["cols"], n)], 1)
    fr = torch.stack([torch.from_numpy(lp["b"]).to(v.device), torch.log(1 + deg_r), norms(lp["rows"], m)], 1)
    xc, xr = torch.relu(fc @ ec_w.T + ec_b), torch.relu(fr @ er_w.T + er_b)
    inv_r, inv_c = 1 / deg_r.clamp(min=1)[:, None], 1 / deg_c.clamp(min=1)[:, None]
    for wrr, wrm, br, wcc, wcm, bc in layers:
        xr = torch.relu(xr @ wrr.T + (_Product.apply(a, at_, xc) * inv_r) @ wrm.T + br)
        xc = torch.relu(xc @ wcc.T + (_Product.apply(at_, a, xr) * inv_c) @ wcm.T + bc)
    oc, orow = xc @ hc_w.T + hc_b, xr @ hr_w.T + hr_b
    if not case["train"]:
        return [oc[:, 0].cpu().numpy(), oc[:, 1].cpu().numpy(), orow[:, 0].cpu().numpy()]
    tx, ts, ty = (torch.from_numpy(t).to(v.device) for t in targets)
    loss = ((oc[:, 0] - tx) ** 2 + (oc[:, 1] - ts) ** 2).sum() / (2 * n) + ((orow[:, 0] - ty) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "grad": w.grad.cpu().numpy()}


class _Product(torch.autograd.Function):
    """A x for a sparse A with its transpose at hand."""

    @staticmethod
    def forward(ctx, a, a_t, x):
        ctx.a_t = a_t
        return a @ x

    @staticmethod
    def backward(ctx, g):
        return None, None, ctx.a_t @ g.contiguous()


def _optimum(lp):
    """The LP's optimal vertex: a short dense primal-dual run finds the basis, two linear solves give
    x, y and s to rounding. None unless the optimum is a non-degenerate vertex."""
    m, n = lp["m"], lp["n"]
    a = np.zeros((m, n))
    a[lp["rows"].cpu().numpy(), lp["cols"].cpu().numpy()] = lp["vals"].cpu().numpy()
    b, c = lp["b"], lp["c"]
    x, s, y = np.ones(n), np.ones(n), np.zeros(m)
    for _ in range(60):
        rp, rd, mu = b - a @ x, c - a.T @ y - s, x @ s / n
        if mu < 1e-9 and max(np.abs(rp).max(), np.abs(rd).max()) < 1e-7:
            break
        normal = (a * (x / s)) @ a.T
        normal[np.diag_indices(m)] += 1e-14 * np.diag(normal)
        target, dxa, dsa = 0.0, 0.0, 0.0
        for step in range(2):
            rc = target - x * s - dxa * dsa
            dy = np.linalg.solve(normal, rp + a @ ((x * rd - rc) / s))
            ds = rd - a.T @ dy
            dx = (rc - x * ds) / s
            ap = min(1.0, 0.995 * np.min(np.where(dx < 0, -x / np.where(dx < 0, dx, -1.0), 1e30)))
            ad = min(1.0, 0.995 * np.min(np.where(ds < 0, -s / np.where(ds < 0, ds, -1.0), 1e30)))
            if step == 0:
                target = ((x + ap * dx) @ (s + ad * ds) / n / mu) ** 3 * mu
                dxa, dsa = dx, ds
        x, y, s = x + ap * dx, y + ad * dy, s + ad * ds
    basis = np.flatnonzero(x > s)
    if basis.size != m:
        return None
    ab = a[:, basis]
    xb, y = np.linalg.solve(ab, b), np.linalg.solve(ab.T, c[basis])
    s = c - a.T @ y
    s[basis] = 0.0
    if xb.min() < 0 or s.min() < 0:
        return None
    x = np.zeros(n)
    x[basis] = xb
    return {"x": x, "y": y, "s": s, "objective": np.array([c @ x])}
