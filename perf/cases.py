"""The work that users of this framework have it do, as cases that can be timed.

A case names one public entry point and its sizes:

  solve     ``equation.solve`` on host arrays (fast or exact mode, f64 or f32)
  factor    ``luhot_?getrf_dev`` + ``luhot_?getrs_dev`` on device buffers
  resident  ``luhot_dfactor_solve_dev``: new right-hand sides on a kept factor
  refine    ``luhot_dgesv_ir_dev``: low-precision LU with FP64 refinement
  backward  ``luhot_dgesv_backward_dev``: the adjoint on stored factors
  batch     ``BatchSolver.solve_device``: uneven small systems, one launch
  qr        ``luhot_dgeqrf_dev``

Matrices are either iid N(0,1) ("normal") or N(0,1) plus 3 sqrt(n) on the
diagonal with the rows in random order ("shuffled": well conditioned, every
step interchanges rows), so that solutions can be compared between two
roundings of the same arithmetic.
"""
import ctypes
import random

import numpy as np
import torch

from lair_gb300 import _lib, equation
from lair_gb300.batched import BatchSolver

_stream = None


def listed():
    return [
        # one small system from host arrays: launches and latency (the reference's own benchmarks are 100 x 100)
        {"name": "solve_f64_100", "kind": "solve", "n": 100, "dtype": "f64", "mode": "fast"},
        # the bit-exact mode, as a caller checks results against the CPU crate
        {"name": "solve_exact_201", "kind": "solve", "n": 201, "dtype": "f64", "mode": "exact"},
        # an ordinary system on the device, one right-hand side
        {"name": "factor_f64_1000", "kind": "factor", "n": 1000, "nrhs": 1, "dtype": "f64", "matrix": "normal"},
        # a ragged mid-size system with several right-hand sides
        {"name": "factor_f64_4097_rhs16", "kind": "factor", "n": 4097, "nrhs": 16, "dtype": "f64", "matrix": "normal"},
        # the largest benchmark size
        {"name": "factor_f64_16384_rhs16", "kind": "factor", "n": 16384, "nrhs": 16, "dtype": "f64",
         "matrix": "shuffled"},
        # single precision throughout
        {"name": "factor_f32_2500_rhs4", "kind": "factor", "n": 2500, "nrhs": 4, "dtype": "f32", "matrix": "shuffled"},
        # time stepping: one right-hand side after another on a kept factor
        {"name": "resident_f64_6000", "kind": "resident", "n": 6000, "nrhs": 1},
        # FP64 answers from tensor-core factors
        {"name": "refine_bf16x3_8192", "kind": "refine", "n": 8192, "nrhs": 1, "precision": "bf16x3"},
        # a solve as a layer of a model: its backward pass
        {"name": "backward_2048_rhs8", "kind": "backward", "n": 2048, "nrhs": 8},
        # many small systems of different sizes at once
        {"name": "batch_f64_1500", "kind": "batch", "count": 1500, "nmin": 8, "nmax": 256, "dtype": "f64"},
        {"name": "batch_f32_10000", "kind": "batch", "count": 10000, "nmin": 8, "nmax": 256, "dtype": "f32"},
        # least squares: a tall Householder factorization
        {"name": "qr_f64_2000x1500", "kind": "qr", "m": 2000, "n": 1500},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["solve", "factor", "factor", "factor", "resident", "refine", "backward", "batch", "batch", "qr"])
    if kind == "solve":
        mode = rng.choice(["fast", "fast", "exact"])
        return {"kind": kind, "n": _log(rng, 16, 700 if mode == "fast" else 300), "dtype": rng.choice(["f64", "f64", "f32"]),
                "mode": mode}
    if kind == "factor":
        dtype = rng.choice(["f64", "f64", "f32"])
        n = _log(rng, 200, 12000 if dtype == "f64" else 6000)
        matrix = "normal" if dtype == "f64" and n <= 4500 and rng.random() < 0.5 else "shuffled"
        return {"kind": kind, "n": n, "nrhs": _log(rng, 1, 16), "dtype": dtype, "matrix": matrix}
    if kind == "resident":
        return {"kind": kind, "n": _log(rng, 500, 12000), "nrhs": rng.choice([1, 1, _log(rng, 2, 16)])}
    if kind == "refine":
        return {"kind": kind, "n": _log(rng, 1000, 12000), "nrhs": rng.choice([1, 1, 2]),
                "precision": rng.choice(["bf16x3", "bf16x3", "fp32"])}
    if kind == "backward":
        return {"kind": kind, "n": _log(rng, 200, 6000), "nrhs": _log(rng, 1, 16)}
    if kind == "batch":
        nmax = _log(rng, 24, 256)
        return {"kind": kind, "count": _log(rng, 100, 6000), "nmin": rng.randint(1, nmax // 2), "nmax": nmax,
                "dtype": rng.choice(["f64", "f32"])}
    n = _log(rng, 200, 2000)
    return {"kind": "qr", "m": n + rng.choice([0, rng.randint(1, 600)]), "n": n}


def _dt(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.float64


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _matrix(n, matrix, dtype, g):
    a = torch.randn((n, n), dtype=dtype, device="cuda", generator=g)
    if matrix == "shuffled":
        a.diagonal().add_(3.0 * n ** 0.5)
        a = a[torch.randperm(n, device="cuda", generator=g)]
    return a


def _randn(shape, dtype, g):
    return torch.randn(shape, dtype=dtype, device="cuda", generator=g)


def _sizes(case):
    r = random.Random(case["count"] * 1000 + case["nmax"])
    return [r.randint(case["nmin"], case["nmax"]) for _ in range(case["count"])]


def _inputs(case, seed):
    """The inputs of a case, from the seed alone."""
    g, kind, dt = _gen(seed), case["kind"], _dt(case)
    if kind == "batch":
        # U[-1,1] entries plus n on the diagonal, every other system with its rows reversed
        sizes = np.array(_sizes(case))
        a = torch.rand(int((sizes ** 2).sum()), dtype=dt, device="cuda", generator=g).mul_(2).sub_(1)
        b = torch.rand(int(sizes.sum()), dtype=dt, device="cuda", generator=g).mul_(2).sub_(1)
        row = np.arange(sizes.sum()) - np.repeat(np.cumsum(sizes) - sizes, sizes)
        n = np.repeat(sizes, sizes)
        col = np.where(np.repeat(np.arange(len(sizes)) % 2, sizes) == 1, n - 1 - row, row)
        at = np.repeat(np.cumsum(sizes ** 2) - sizes ** 2, sizes) + row * n + col
        at = torch.from_numpy(at).cuda()
        a[at] += torch.from_numpy(n).cuda().to(dt)
        return a, b
    if kind == "qr":
        return (_randn((case["m"], case["n"]), dt, g),)
    n = case["n"]
    a = _matrix(n, case.get("matrix", "shuffled"), dt, g)
    if kind == "solve":
        return a, _randn((n,), dt, g)
    b = _randn((n, case["nrhs"]), dt, g)
    return (a, b, _randn((n, case["nrhs"]), dt, g)) if kind == "backward" else (a, b)


def _use_stream():
    """One stream for torch's copies and the library's kernels."""
    global _stream
    lib, ctx = _lib.load(), _lib.context()
    if _stream is None:
        _stream = torch.cuda.Stream()
    _lib.check(lib.luhot_set_stream(ctx, ctypes.c_void_p(_stream.cuda_stream)), ctx)
    return lib, ctx


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


class _Factor:
    """A kept factor (``luhot_dfactor_create_dev``)."""

    def __init__(self, lib, ctx, a):
        n = a.shape[0]
        self.lib, self.h = lib, ctypes.c_void_p()
        piv, sing = np.zeros(n, dtype=np.uint64), ctypes.c_int64()
        _lib.check(lib.luhot_dfactor_create_dev(ctx, n, n, _p(a), n, _lib.MODE_FAST, piv.ctypes.data,
                                                ctypes.byref(sing), ctypes.byref(self.h)), ctx)

    def __del__(self):
        if self.h:
            self.lib.luhot_factor_destroy(self.h)


def prepare(case, seed):
    lib, ctx = _use_stream()
    kind = case["kind"]
    given = _inputs(case, seed)
    torch.cuda.synchronize()
    s = {"case": case, "lib": lib, "ctx": ctx}
    if kind == "solve":
        s["a"], s["b"] = (t.cpu().numpy() for t in given)
        return s
    if kind == "batch":
        s["a0"], s["b0"] = given
        s["plan"] = BatchSolver(_sizes(case), dtype=np.float32 if case["dtype"] == "f32" else np.float64)
        s["plan"].autotune(given[0].data_ptr(), given[1].data_ptr())
        s["a"], s["b"] = torch.empty_like(given[0]), torch.empty_like(given[1])
        s["piv"] = torch.zeros(given[1].numel(), dtype=torch.int32, device="cuda")
        s["info"] = torch.zeros(case["count"], dtype=torch.int32, device="cuda")
        return s
    if kind == "qr":
        s["a0"] = given[0]
        s["a"] = torch.empty_like(given[0])
        s["tau"] = torch.zeros(min(given[0].shape), dtype=torch.float64, device="cuda")
        return s
    n = case["n"]
    if kind == "resident":
        s["factor"], s["b0"], s["b"] = _Factor(lib, ctx, given[0]), given[1], torch.empty_like(given[1])
        return s
    if kind == "refine":
        s["a"], s["b"], s["x"] = given[0], given[1], torch.empty_like(given[1])
        return s
    piv = torch.zeros(n, dtype=torch.int32, device="cuda")
    s["piv"] = piv
    if kind == "factor":
        s["a0"], s["b0"] = given
        s["a"], s["b"] = torch.empty_like(given[0]), torch.empty_like(given[1])
        return s
    lu, x, s["w"] = given
    sing = ctypes.c_int64()
    _lib.check(lib.luhot_dgetrf_dev(ctx, n, n, _p(lu), n, _p(piv), ctypes.byref(sing), _lib.MODE_FAST), ctx)
    s["lu"], s["x"] = lu, x  # a given solution: the gradient formula holds for any x
    s["db"], s["da"] = torch.empty_like(x), torch.empty_like(lu)
    return s


def run(s):
    case, lib, ctx = s["case"], s["lib"], s["ctx"]
    kind = case["kind"]
    if kind == "solve":
        return equation.solve(s["a"], s["b"], mode=case["mode"])
    with torch.cuda.stream(_stream):
        if kind == "batch":
            s["a"].copy_(s["a0"])
            s["b"].copy_(s["b0"])
            s["plan"].solve_device(s["a"].data_ptr(), s["b"].data_ptr(), s["piv"].data_ptr(), s["info"].data_ptr())
            return s["a"], s["b"], s["piv"], s["info"]
        if kind == "qr":
            s["a"].copy_(s["a0"])
            m, n = case["m"], case["n"]
            _lib.check(lib.luhot_dgeqrf_dev(ctx, m, n, _p(s["a"]), n, _p(s["tau"]), _lib.MODE_FAST), ctx)
            return s["a"], s["tau"]
        n, nrhs = case["n"], case["nrhs"]
        if kind == "resident":
            s["b"].copy_(s["b0"])
            _lib.check(lib.luhot_dfactor_solve_dev(s["factor"].h, nrhs, _p(s["b"]), nrhs, 0), ctx)
            return s["b"]
        if kind == "refine":
            info = _lib.IrInfo()
            _lib.check(lib.luhot_dgesv_ir_dev(ctx, n, nrhs, _p(s["a"]), n, _p(s["b"]), nrhs, _p(s["x"]), nrhs,
                                              _lib.PRECISIONS[case["precision"]], _lib.REFINE_IR, 0.0, 30,
                                              ctypes.byref(info)), ctx)
            return s["x"]
        if kind == "backward":
            _lib.check(lib.luhot_dgesv_backward_dev(ctx, n, nrhs, _p(s["lu"]), n, _p(s["piv"]), _p(s["x"]), nrhs,
                                                    _p(s["w"]), nrhs, _p(s["db"]), nrhs, _p(s["da"]), n,
                                                    _lib.MODE_FAST), ctx)
            return s["db"], s["da"]
        s["a"].copy_(s["a0"])
        s["b"].copy_(s["b0"])
        pre = "s" if case["dtype"] == "f32" else "d"
        sing = ctypes.c_int64()
        _lib.check(getattr(lib, f"luhot_{pre}getrf_dev")(ctx, n, n, _p(s["a"]), n, _p(s["piv"]), ctypes.byref(sing),
                                                         _lib.MODE_FAST), ctx)
        _lib.check(getattr(lib, f"luhot_{pre}getrs_dev")(ctx, n, nrhs, _p(s["a"]), n, _p(s["piv"]), _p(s["b"]), nrhs,
                                                         0, _lib.MODE_FAST), ctx)
        return s["a"], s["piv"], s["b"]


def work(case):
    kind = case["kind"]
    e = 4 if case.get("dtype") == "f32" else 8
    if kind == "batch":
        sizes = [float(n) for n in _sizes(case)]
        return {"bytes": sum(2 * e * (n * n + n) + 4 * n for n in sizes),
                "flops": sum(2 / 3 * n ** 3 + 2 * n * n for n in sizes)}
    if kind == "qr":
        m, n = float(case["m"]), float(case["n"])
        return {"bytes": 16 * m * n + 8 * n, "flops": 2 * n * n * (m - n / 3)}
    n, r = float(case["n"]), float(case.get("nrhs", 1))
    lu, sweeps = 2 / 3 * n ** 3, 2 * n * n * r
    if kind == "solve":
        return {"bytes": e * (n * n + 2 * n), "flops": lu + sweeps}
    if kind == "resident":
        return {"bytes": 8 * n * n + 16 * n * r, "flops": sweeps}
    if kind == "refine":
        return {"bytes": 8 * n * n + 16 * n * r, "flops": lu + sweeps}
    if kind == "backward":
        return {"bytes": 16 * n * n + 24 * n * r, "flops": 2 * sweeps}
    return {"bytes": 2 * e * n * n + 2 * e * n * r, "flops": lu + sweeps}


def exact(case, seed):
    kind = case["kind"]
    if kind != "batch" and case["n"] > 9000:
        return None
    given = [t.cpu().to(torch.float64) for t in _inputs(case, seed)]
    if kind == "qr":
        return torch.geqrf(given[0])
    if kind == "batch":
        a, b = given
        sizes = np.array(_sizes(case))
        a_at, b_at = np.cumsum(sizes ** 2) - sizes ** 2, np.cumsum(sizes) - sizes
        lu, x = torch.empty_like(a), torch.empty_like(b)
        for n in sorted(set(sizes.tolist())):
            which = np.nonzero(sizes == n)[0]
            ia = torch.from_numpy(a_at[which][:, None] + np.arange(n * n))
            ib = torch.from_numpy(b_at[which][:, None] + np.arange(n))
            f, p = torch.linalg.lu_factor(a[ia].reshape(-1, n, n))
            lu[ia] = f.reshape(len(which), -1)
            x[ib] = torch.linalg.lu_solve(f, p, b[ib].unsqueeze(2)).squeeze(2)
        return lu, x, None, None
    a, b = given[:2]
    f, p = torch.linalg.lu_factor(a)
    if kind == "solve":
        return torch.linalg.lu_solve(f, p, b.unsqueeze(1)).squeeze(1)
    if kind == "backward":
        lam = torch.linalg.solve(a.T, given[2])
        return lam, -lam @ b.T
    x = torch.linalg.lu_solve(f, p, b)
    return (f, None, x) if kind == "factor" else x
