"""Performance cases: what a user of rulinalg_gb300 has it do, through its public entry
points, over the real range of sizes.

listed() names the cases, draw() gives more of the same ranges, prepare() makes the
inputs (and the plan, factor or output buffers a program keeps), run() is one pass and
work() the bytes and floating-point operations the pass cannot do without. exact() is the
same result from plain torch / numpy in 64 bits.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import rulinalg_gb300 as rl
from rulinalg_gb300._lib import SolveInfo, lib
from rulinalg_gb300.workloads import log_uniform_sizes

F64, F32 = torch.float64, torch.float32


def listed():
    return [
        # Matrix::solve of one small system, host arrays: the smallest call of the crate,
        # where launches, copies and the call itself count.
        {"name": "solve_47", "op": "solve", "n": 47, "dtype": "f64"},
        # PartialPivLu::decompose + solve of one n = 1024 system, host arrays (U(-1,1) plus
        # 1 on the diagonal, one right-hand side): the plain method.
        {"name": "lu_1024", "op": "lu", "n": 1024, "dtype": "f64"},
        # HouseholderQr::decompose + unpack_thin of a tall odd-sized matrix, host arrays.
        {"name": "qr_1201x499", "op": "qr", "m": 1201, "n": 499, "dtype": "f64"},
        # Matrix product on device buffers, f32 and f64: the middle of the 1024-8192 sweep.
        {"name": "gemm_f32_4096", "op": "gemm", "m": 4096, "k": 4096, "n": 4096, "dtype": "f32"},
        {"name": "gemm_f64_2048", "op": "gemm", "m": 2048, "k": 2048, "n": 2048, "dtype": "f64"},
        # The batched uneven mix, f64-accurate through mixed precision: 20,000 SPD systems
        # and 20,000 general ones, n log-uniform in [8, 512], a plan kept between calls.
        {"name": "batch_mixed_40k", "op": "batch", "spd": 20000, "general": 20000, "lo": 8, "hi": 512,
         "precision": "mixed"},
        # The f32 SPD half of the same batch (Cholesky in FP32).
        {"name": "batch_f32_spd_20k", "op": "batch", "spd": 20000, "general": 0, "lo": 8, "hi": 512,
         "precision": "f32"},
        # Mixed-precision LU solve of one ill-conditioned system: FP32 factor, FP64
        # refinement over several steps, one right-hand side.
        {"name": "mixed_lu_4096", "op": "mixed", "n": 4096, "nrhs": 1, "kappa": 1e6},
        # The same with many right-hand sides on a large, well-conditioned system.
        {"name": "mixed_lu_8192_rhs64", "op": "mixed", "n": 8192, "nrhs": 64, "kappa": 1e2},
        # The all-FP64 solve of one system on device buffers (factor + solve).
        {"name": "fp64_lu_4096", "op": "fp64", "n": 4096, "nrhs": 1, "kind": "lu"},
        # Least squares with m = 2n, f64-accurate through an FP32 QR: the served stream's
        # regression requests, at an odd size.
        {"name": "lstsq_2999x1501", "op": "lstsq", "m": 2999, "n": 1501},
        # A new right-hand side against a factor that stays on the device: the served
        # stream's re-solves.
        {"name": "resolve_3000", "op": "resolve", "n": 3000, "nrhs": 1, "kind": "lu"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["solve", "lu", "qr", "gemm", "gemm", "batch", "mixed", "fp64", "lstsq", "resolve"])
    if op == "solve":
        return {"op": op, "n": _log_int(rng, 8, 512), "dtype": rng.choice(["f64", "f32"])}
    if op == "lu":
        return {"op": op, "n": _log_int(rng, 64, 2048), "dtype": "f64"}
    if op == "qr":
        n = _log_int(rng, 32, 700)
        return {"op": op, "m": n + rng.randrange(1, 2 * n), "n": n, "dtype": "f64"}
    if op == "gemm":
        hi = 3000 if (dt := rng.choice(["f64", "f32"])) == "f64" else 8192
        m, k, n = (_log_int(rng, 64, hi) for _ in range(3))
        return {"op": op, "m": m, "k": k, "n": n, "dtype": dt}
    if op == "batch":
        total, spd = _log_int(rng, 100, 20000), rng.choice([0.0, 0.5, 1.0])
        return {"op": op, "spd": int(total * spd), "general": total - int(total * spd), "lo": 8,
                "hi": _log_int(rng, 32, 512), "precision": rng.choice(["mixed", "mixed", "f64", "f32"])}
    if op == "mixed":
        nrhs = rng.choice([1, 1, _log_int(rng, 2, 64)])
        return {"op": op, "n": _log_int(rng, 600, 6000), "nrhs": nrhs,
                "kappa": 10.0 ** rng.choice([2, 4, 6] if nrhs == 1 else [2, 4])}
    if op == "fp64":
        return {"op": op, "n": _log_int(rng, 600, 4096), "nrhs": rng.choice([1, _log_int(rng, 2, 64)]),
                "kind": rng.choice(["lu", "cholesky"])}
    if op == "lstsq":
        n = _log_int(rng, 64, 2000)
        return {"op": op, "m": 2 * n + rng.randrange(0, 9), "n": n}
    return {"op": op, "n": _log_int(rng, 600, 4096), "nrhs": rng.choice([1, _log_int(rng, 2, 64)]),
            "kind": rng.choice(["lu", "cholesky"])}


# ------------------------------------------------------------------------- inputs --
def _device():
    return torch.device("cuda", 0)


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape, dtype=F64):
    return torch.randn(*shape, dtype=dtype, device=_device(), generator=g)


def _general(g, n, dtype=F64, shift=1.0):
    """U(-1,1) entries plus `shift` on the diagonal."""
    a = torch.rand(n, n, dtype=dtype, device=_device(), generator=g) * 2 - 1
    a.diagonal().add_(shift)
    return a


def _spd(g, n):
    """G G^T + n I with G ~ N(0,1)."""
    x = _randn(g, n, n)
    a = x @ x.T
    a.diagonal().add_(float(n))
    return a


def _conditioned(g, n, kappa):
    """U diag(sigma) V^T, sigma geometric from 1 to 1 / kappa, U and V random orthogonal."""
    def haar():
        q, r = torch.linalg.qr(_randn(g, n, n, dtype=F32))
        return (q * torch.sign(torch.diagonal(r))).to(F64)
    sigma = kappa ** (-torch.arange(n, dtype=F64, device=_device()) / max(n - 1, 1))
    return ((haar() * sigma) @ haar().T).contiguous()


def _batch_shape(case):
    """Orders and kinds of a batch (the plan's, the same for every seed)."""
    rng = np.random.default_rng(case["spd"] + 7 * case["general"] + 13 * case["hi"])
    n = log_uniform_sizes(case["spd"] + case["general"], case["lo"], case["hi"], rng)
    kind = np.concatenate([np.ones(case["spd"], np.uint8), np.zeros(case["general"], np.uint8)])
    return n, kind


def _groups(n, kind):
    """(size, kind, indices) of the systems of equal order and kind."""
    for size in np.unique(n):
        for k in (1, 0):
            idx = np.nonzero((n == size) & (kind == k))[0]
            if len(idx):
                yield int(size), k, idx


def _batch_inputs(case, seed):
    n, kind = _batch_shape(case)
    dev, g = _device(), _gen(seed)
    a_off = np.concatenate([[0], np.cumsum(n.astype(np.int64) ** 2)])
    a = torch.rand(int(a_off[-1]), dtype=F64, device=dev, generator=g).mul_(2).sub_(1)
    b = _randn(g, int(n.sum()))
    for size, k, idx in _groups(n, kind):
        off = torch.from_numpy(a_off[idx]).to(dev)
        if k:
            x = _randn(g, len(idx), size, size)
            blk = torch.bmm(x, x.transpose(1, 2))
            blk.diagonal(dim1=1, dim2=2).add_(float(size))
            a[off[:, None] + torch.arange(size * size, device=dev)] = blk.reshape(len(idx), -1)
        else:
            a[off[:, None] + torch.arange(size, device=dev) * (size + 1)] += float(size)
    if case["precision"] == "f32":
        a, b = a.float(), b.float()
    return n, kind, a, b


def _inputs(case, seed):
    op = case["op"]
    if op in ("solve", "lu"):
        g, dt = _gen(seed), F32 if case["dtype"] == "f32" else F64
        # Matrix::solve's small systems are diagonally weighted like the batched general ones
        a = _general(g, case["n"], dt, 1.0 if op == "lu" else float(case["n"]))
        return a.cpu().numpy(), _randn(g, case["n"], dtype=dt).cpu().numpy()
    if op == "qr":
        return (_randn(_gen(seed), case["m"], case["n"]).cpu().numpy(),)
    if op == "gemm":
        g, dt = _gen(seed), F32 if case["dtype"] == "f32" else F64
        return _randn(g, case["m"], case["k"], dtype=dt), _randn(g, case["k"], case["n"], dtype=dt)
    if op == "lstsq":
        g = _gen(seed)
        return _randn(g, case["m"], case["n"]), _randn(g, case["m"])
    g = _gen(seed)
    if op == "mixed":
        a = _conditioned(g, case["n"], case["kappa"])
    else:
        a = _spd(g, case["n"]) if case["kind"] == "cholesky" else _general(g, case["n"])
    return a, _randn(g, case["n"], case["nrhs"])


def prepare(case, seed):
    op = case["op"]
    state = {"op": op, "case": case}
    if op == "batch":
        n, kind, a, b = _batch_inputs(case, seed)
        prec = {"mixed": rl.PREC_MIXED, "f64": rl.PREC_FP64, "f32": rl.PREC_FP32}[case["precision"]]
        state.update(plan=rl.BatchPlan(n, kind, prec), a=a, b=b, x=torch.zeros_like(b),
                     info=torch.zeros(len(n), dtype=torch.int32, device=a.device))
        return state
    state["in"] = _inputs(case, seed)
    if op == "gemm":
        state["c"] = torch.empty(case["m"], case["n"], dtype=state["in"][0].dtype, device=_device())
    elif op == "lstsq":
        state["x"] = torch.empty(case["n"], dtype=F64, device=_device())
    elif op in ("mixed", "fp64", "resolve"):
        state["x"] = torch.empty(case["n"], case["nrhs"], dtype=F64, device=_device())
        if op == "resolve":
            state["factor"] = rl.ResidentFactor(state["in"][0], case["kind"], _stream())
    return state


# --------------------------------------------------------------------------- runs --
def _stream():
    return torch.cuda.current_stream().cuda_stream


def _ok(status):
    if status:
        raise RuntimeError(lib.rl_status_string(status).decode())


def run(state):
    op, case = state["op"], state["case"]
    if op == "solve":
        return {"x": rl.solve(*state["in"])}
    if op == "lu":
        a, b = state["in"]
        lu = rl.PartialPivLu.decompose(a)
        return {"lu": lu.lu, "perm": lu.p.perm, "x": lu.solve(b)}
    if op == "qr":
        thin = rl.HouseholderQr.decompose(state["in"][0]).unpack_thin()
        return {"q1": thin.q1, "r1": thin.r1}
    if op == "batch":
        x, info = state["x"], state["info"]
        state["plan"].solve_dev(state["a"].data_ptr(), state["b"].data_ptr(), x.data_ptr(), info.data_ptr(),
                                stream=_stream())
        return {"x": x, "info": info}
    a, b = state["in"]
    if op == "gemm":
        c, fn = state["c"], lib.rl_sgemm_dev if a.dtype == F32 else lib.rl_dgemm_dev
        m, k, n = case["m"], case["k"], case["n"]
        _ok(fn(m, k, n, a.data_ptr(), k, b.data_ptr(), n, c.data_ptr(), n, _stream() or None))
        return {"c": c}
    x = state["x"]
    if op == "lstsq":
        info = SolveInfo()
        _ok(lib.rl_dlstsq_mixed_dev(case["m"], case["n"], a.data_ptr(), case["n"], b.data_ptr(), x.data_ptr(),
                                    C.byref(info), _stream() or None))
        return {"x": x}
    n, nrhs = case["n"], case["nrhs"]
    if op == "resolve":
        state["factor"].solve(b, x, _stream())
    elif op == "mixed":
        info = SolveInfo()
        _ok(lib.rl_dsolve_mixed_dev(n, nrhs, 0, a.data_ptr(), n, b.data_ptr(), nrhs, x.data_ptr(), nrhs,
                                    C.byref(info), _stream() or None))
    else:
        _ok(lib.rl_dsolve_fp64_dev(n, nrhs, 1 if case["kind"] == "cholesky" else 0, a.data_ptr(), n, b.data_ptr(),
                                   nrhs, x.data_ptr(), nrhs, None, _stream() or None))
    return {"x": x}


def work(case):
    op = case["op"]
    size = 4 if case.get("dtype") == "f32" or case.get("precision") == "f32" else 8
    if op == "gemm":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": size * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    if op == "batch":
        n, kind = _batch_shape(case)
        n = n.astype(np.float64)
        factor = np.where(kind == 1, n ** 3 / 3, 2 * n ** 3 / 3)
        return {"bytes": float((size * (n * n + 2 * n) + 4).sum()), "flops": float((factor + 2 * n * n).sum())}
    if op in ("qr", "lstsq"):
        m, n = case["m"], case["n"]
        factor = 2 * m * n * n - 2 * n ** 3 / 3
        if op == "lstsq":
            return {"bytes": size * (m * n + m + n), "flops": factor + 4 * m * n + n * n}
        return {"bytes": size * (2 * m * n + n * n), "flops": 2 * factor}
    n, nrhs = case["n"], case.get("nrhs", 1)
    if op == "resolve":  # one residual against the matrix and one pass over the factor
        return {"bytes": 8 * n * n + 4 * n * n + 16 * n * nrhs, "flops": 4 * n * n * nrhs}
    factor = n ** 3 / 3 if case.get("kind") == "cholesky" else 2 * n ** 3 / 3
    out = n * n + n if op == "lu" else 0  # the packed factor and the permutation
    return {"bytes": size * (n * n + out + 2 * n * nrhs), "flops": factor + 2 * n * n * nrhs}


# -------------------------------------------------------------------------- exact --
def exact(case, seed):
    op = case["op"]
    if op == "batch":
        n, kind, a, b = _batch_inputs(case, seed)
        a, b = a.double(), b.double()
        a_off = np.concatenate([[0], np.cumsum(n.astype(np.int64) ** 2)])
        b_off = np.concatenate([[0], np.cumsum(n.astype(np.int64))])
        x = torch.empty_like(b)
        for size, k, idx in _groups(n, kind):
            ao = torch.from_numpy(a_off[idx]).to(a.device)
            bo = torch.from_numpy(b_off[idx]).to(a.device)
            mats = a[ao[:, None] + torch.arange(size * size, device=a.device)].reshape(len(idx), size, size)
            at = bo[:, None] + torch.arange(size, device=a.device)
            x[at] = torch.linalg.solve(mats, b[at])
        return {"x": x, "info": None}
    ins = [torch.as_tensor(v).to(_device()).double() for v in _inputs(case, seed)]
    if op == "qr":
        # the compact QR's signs: R's diagonal opposes the leading entry of each reflected column
        q, r = torch.linalg.qr(ins[0])
        return {"q1": q.cpu().numpy(), "r1": r.cpu().numpy()}
    if op == "gemm":
        return {"c": ins[0] @ ins[1]}
    if op == "lstsq":
        q, r = torch.linalg.qr(ins[0])
        return {"x": torch.linalg.solve_triangular(r, (q.T @ ins[1])[:, None], upper=True)[:, 0]}
    x = torch.linalg.solve(ins[0], ins[1])
    if op == "solve":
        return {"x": x.cpu().numpy()}
    if op == "lu":
        return {"lu": torch.linalg.lu_factor(ins[0])[0].cpu().numpy(), "perm": None, "x": x.cpu().numpy()}
    return {"x": x}
