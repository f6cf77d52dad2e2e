"""Performance cases of the framework: the calls its users make, at the sizes they make them.

A case is a dict of plain values; "op" names the call:

  solve      Matrix.solve on host arrays, small systems
  lu         LUDecomposition.new, det, get_piv, get_packed and solve on host arrays
  lu_device  LUDecomposition.new_device and solve_device on device arrays, FAST or EXACT arithmetic
  inverse    Matrix.inverse on a host array
  mul        Matrix * Matrix on device arrays
  chol       CholeskyDecomposition.new_device and solve_device
  qr         QRDecomposition.new_device, get_r and get_q
  mixed      lu_solve_auto_device: low-precision factors, FP64 refinement
  batch      a BatchPlan run in plain FP64 over systems of uneven size
  selector   features, class prediction, selection and a mixed BatchPlan run
  train      one Adam step of the selector network, parameters read back

Matrices have prescribed singular values, geometric from sqrt(kappa) down to 1/sqrt(kappa), between
dense orthogonal factors (Hartley transforms with random signs): entries look Gaussian, partial
pivoting moves rows at every step, and the solution is determined to about kappa * 1e-16.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "rust-la_gb300"))
import la_gpu  # noqa: E402
import selector  # noqa: E402

F64 = torch.float64
TOL = 5e-15  # backward error asked of the refined solvers, as the benchmark asks

_ctx = {}


def _context(arith=la_gpu.ARITH_FAST):
    """One context per arithmetic, kept by the program."""
    if arith not in _ctx:
        _ctx[arith] = la_gpu.Context(0, arith)
    return _ctx[arith]


# ---- the cases ---------------------------------------------------------------------------------


def listed():
    return [
        # A script that solves one small system at a time: launches and latency, no arithmetic.
        {"name": "solve_24", "op": "solve", "n": 24, "nrhs": 1, "kappa": 100.0},
        # The everyday factorization through the crate's own API, host arrays in and out.
        {"name": "lu_512", "op": "lu", "n": 512, "nrhs": 1, "kappa": 100.0},
        # An explicit inverse: as many right-hand sides as rows; a size that no tile divides.
        {"name": "inverse_1000", "op": "inverse", "n": 1000, "kappa": 100.0},
        # The large dense system of the benchmark, resident on the device.
        {"name": "lu_8192", "op": "lu_device", "n": 8192, "nrhs": 16, "kappa": 1000.0, "exact": False},
        # The bit-identical arithmetic, for users who check against the crate.
        {"name": "lu_exact_1000", "op": "lu_device", "n": 1000, "nrhs": 1, "kappa": 100.0, "exact": True},
        # The benchmark's matrix product.
        {"name": "mul_8192", "op": "mul", "m": 8192, "k": 8192, "n": 8192},
        # A covariance-type system of odd size with a few right-hand sides.
        {"name": "chol_4099", "op": "chol", "n": 4099, "nrhs": 5, "kappa": 1000.0},
        # A tall factorization of ragged shape, both factors taken to the host.
        {"name": "qr_2500x1501", "op": "qr", "m": 2500, "n": 1501, "kappa": 100.0},
        # The largest system: mixed precision to FP64 accuracy.
        {"name": "mixed_16384", "op": "mixed", "n": 16384, "nrhs": 4, "kappa": 10000.0},
        # Thousands of small systems of uneven size in plain FP64.
        {"name": "batch_4000", "op": "batch", "count": 4000, "nmin": 8, "nmax": 256},
        # The same through the learned precision selector, with larger systems among them.
        {"name": "selector_3000", "op": "selector", "count": 3000, "nmin": 16, "nmax": 512},
        # A step of the selector's training at its default minibatch.
        {"name": "train_4096", "op": "train", "count": 4096},
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi]; half of them odd, a quarter multiples of 64."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    n = max(lo, min(hi, n))
    kind = rng.randrange(4)
    if kind < 2:
        n |= 1
    elif kind == 2 and n >= 128:
        n = n // 64 * 64
    return max(lo, min(hi, n))


def draw(rng):
    op = rng.choice(["solve", "lu", "inverse", "lu_device", "lu_device", "lu_exact", "mul", "mul",
                     "chol", "qr", "mixed", "batch", "selector", "train"])
    kappa = 10.0 ** rng.uniform(1.0, 4.0)
    if op == "solve":
        return {"op": op, "n": _size(rng, 2, 200), "nrhs": rng.randint(1, 4), "kappa": kappa}
    if op == "lu":
        return {"op": op, "n": _size(rng, 100, 700), "nrhs": rng.randint(1, 8), "kappa": kappa}
    if op == "inverse":
        return {"op": op, "n": _size(rng, 50, 2500), "kappa": kappa}
    if op == "lu_device":
        return {"op": op, "n": _size(rng, 200, 8192), "nrhs": _size(rng, 1, 64), "kappa": kappa,
                "exact": False}
    if op == "lu_exact":
        return {"op": "lu_device", "n": _size(rng, 100, 1500), "nrhs": rng.randint(1, 8),
                "kappa": kappa, "exact": True}
    if op == "mul":
        return {"op": op, "m": _size(rng, 64, 8192), "k": _size(rng, 64, 8192),
                "n": _size(rng, 64, 8192)}
    if op == "chol":
        return {"op": op, "n": _size(rng, 100, 8192), "nrhs": _size(rng, 1, 32), "kappa": kappa}
    if op == "qr":
        m = _size(rng, 100, 4096)
        return {"op": op, "m": m, "n": _size(rng, max(1, m // 8), m), "kappa": min(kappa, 1000.0)}
    if op == "mixed":
        return {"op": op, "n": _size(rng, 1000, 16384), "nrhs": rng.randint(1, 16), "kappa": kappa}
    if op == "batch":
        nmax = rng.choice([64, 128, 256, 400])
        return {"op": op, "count": _size(rng, 200, 6000), "nmin": rng.randint(2, nmax // 2), "nmax": nmax}
    if op == "selector":
        nmax = rng.choice([128, 256, 512])
        return {"op": op, "count": _size(rng, 200, 3000), "nmin": 16, "nmax": nmax}
    return {"op": "train", "count": _size(rng, 256, 16384)}


# ---- inputs ------------------------------------------------------------------------------------


def _hartley(x, dim):
    f = torch.fft.fft(x, dim=dim, norm="ortho")
    return f.real - f.imag


def _signs(g, n):
    return torch.randint(0, 2, (n,), generator=g, device="cuda").to(F64) * 2 - 1


def _conditioned(g, m, n, kappa):
    """m x n, m >= n, singular values geometric from sqrt(kappa) to 1/sqrt(kappa)."""
    t = torch.linspace(0.5, -0.5, n, dtype=F64, device="cuda")
    x = torch.zeros((m, n), dtype=F64, device="cuda")
    x.diagonal().copy_(torch.pow(torch.tensor(kappa, dtype=F64, device="cuda"), t))
    x = _hartley(x, 0) * _signs(g, m)[:, None]
    x = _hartley(x, 0) * _signs(g, n)
    x = _hartley(x, 1) * _signs(g, n)
    return x.contiguous()


def _spd(g, n, kappa):
    t = torch.linspace(0.5, -0.5, n, dtype=F64, device="cuda")
    s = torch.pow(torch.tensor(kappa, dtype=F64, device="cuda"), t)
    x = torch.zeros((n, n), dtype=F64, device="cuda")
    x.diagonal().copy_(s[torch.randperm(n, generator=g, device="cuda")])
    for _ in range(2):
        d = _signs(g, n)
        x = _hartley(_hartley(x * d * d[:, None], 0), 1)
    return ((x + x.t()) * 0.5).contiguous()


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=F64)


def _inputs(case, seed):
    """The arrays of a case, from the seed alone."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + 7)
    op = case["op"]
    if op in ("solve", "lu", "lu_device", "mixed"):
        n = case["n"]
        return {"a": _conditioned(g, n, n, case["kappa"]), "b": _randn(g, n, case["nrhs"])}
    if op == "inverse":
        return {"a": _conditioned(g, case["n"], case["n"], case["kappa"])}
    if op == "mul":
        return {"a": _randn(g, case["m"], case["k"]), "b": _randn(g, case["k"], case["n"])}
    if op == "chol":
        return {"a": _spd(g, case["n"], case["kappa"]), "b": _randn(g, case["n"], case["nrhs"])}
    if op == "qr":
        return {"a": _conditioned(g, case["m"], case["n"], case["kappa"])}
    if op in ("batch", "selector"):
        # The batch's sizes belong to the case, its values to the seed.
        rng = np.random.default_rng(case["count"])
        ns = rng.integers(case["nmin"], case["nmax"] + 1, size=case["count"])
        rs = rng.integers(1, 5, size=case["count"])
        systems, na, nb = la_gpu.batch_systems(ns, rs)
        a = torch.empty(na, dtype=F64, device="cuda")
        b = torch.empty(nb, dtype=F64, device="cuda")
        torch.cuda.synchronize()
        la_gpu.generate_conditioned_batch(_context(), systems, 1.0, 4.0, int(seed) * 31 + 5,
                                          a.data_ptr(), b.data_ptr())
        return {"a": a, "b": b, "systems": systems, "ns": ns, "rs": rs}
    x = torch.randn((case["count"], 16), generator=g, device="cuda")
    y = (x[:, :3] + 0.3 * torch.randn((case["count"], 3), generator=g, device="cuda")).argmax(1)
    rng = np.random.default_rng(int(seed))
    w = [rng.standard_normal(64 * 16) / 4, rng.standard_normal(64) * 0.1,
         rng.standard_normal(64 * 64) / 8, rng.standard_normal(64) * 0.1,
         rng.standard_normal(3 * 64) / 8, rng.standard_normal(3) * 0.1,
         rng.standard_normal(16) * 0.1, 1 + 0.2 * rng.random(16)]
    return {"x": x, "y": y.to(torch.int32), "p": np.concatenate(w).astype(np.float32)}


def prepare(case, seed):
    s = _inputs(case, seed)
    op = case["op"]
    s["case"] = case
    s["ctx"] = _context(la_gpu.ARITH_EXACT if case.get("exact") else la_gpu.ARITH_FAST)
    if op in ("solve", "lu", "inverse"):
        s["a"] = s["a"].cpu().numpy()
        if "b" in s:
            s["b"] = s["b"].cpu().numpy()
    elif op in ("lu_device", "mixed", "chol", "batch", "selector"):
        s["x"] = torch.zeros_like(s["b"])
    elif op == "mul":
        s["c"] = torch.zeros((case["m"], case["n"]), dtype=F64, device="cuda")
    torch.cuda.synchronize()
    # Plan shapes: what the autotuner picks for systems of these sizes.
    if op == "batch":
        small = case["nmax"] <= 256
        s["plan"] = la_gpu.BatchPlan(s["ctx"], s["a"].data_ptr(), s["b"].data_ptr(), s["x"].data_ptr(),
                                     s["systems"], la_gpu.BATCH_FP64, ctas_per_sm=2 if small else 1,
                                     warps_per_system=4 if small else 8)
    elif op == "selector":
        small = case["nmax"] <= 256
        s["plan"] = la_gpu.BatchPlan(s["ctx"], s["a"].data_ptr(), s["b"].data_ptr(), s["x"].data_ptr(),
                                     s["systems"], la_gpu.BATCH_MIXED, ctas_per_sm=4 if small else 2,
                                     warps_per_system=4 if small else 8, tol=TOL)
        s["sel"] = selector.PrecisionSelector.from_file(
            s["ctx"], os.path.join(os.path.dirname(la_gpu.__file__), "selector_weights.npy"))
        s["f"] = torch.empty((case["count"], 16), dtype=torch.float32, device="cuda")
        s["cls"] = torch.empty(case["count"], dtype=torch.int32, device="cuda")
    elif op == "train":
        s["mlp"] = la_gpu.Mlp(s["ctx"], 1)
        s["mlp"].set_params(s["p"])
    torch.cuda.synchronize()
    return s


# ---- the calls ---------------------------------------------------------------------------------


def run(s):
    case, ctx = s["case"], s["ctx"]
    op = case["op"]
    if op == "solve":
        return la_gpu.Matrix(s["a"], ctx).solve(la_gpu.Matrix(s["b"], ctx)).data
    if op == "lu":
        lu = la_gpu.LUDecomposition.new(la_gpu.Matrix(s["a"], ctx))
        out = {"det": lu.det(), "piv": lu.get_piv().astype(np.int64),
               "x": lu.solve(la_gpu.Matrix(s["b"], ctx)).data, "lu": lu.get_packed().data}
        lu.free()
        return out
    if op == "inverse":
        return la_gpu.Matrix(s["a"], ctx).inverse().data
    if op == "lu_device":
        n, r = case["n"], case["nrhs"]
        lu = la_gpu.LUDecomposition.new_device(s["a"].data_ptr(), n, n, n, ctx)
        lu.solve_device(s["b"].data_ptr(), r, n, r, s["x"].data_ptr(), r)
        out = {"x": s["x"], "piv": lu.get_piv().astype(np.int64)}
        lu.free()
        return out
    if op == "mul":
        m, k, n = case["m"], case["k"], case["n"]
        la_gpu.matrix_mul_device(ctx, s["a"].data_ptr(), k, s["b"].data_ptr(), n, s["c"].data_ptr(), n,
                                 m, k, n)
        return s["c"]
    if op == "chol":
        n, r = case["n"], case["nrhs"]
        ch = la_gpu.CholeskyDecomposition.new_device(s["a"].data_ptr(), n, n, ctx)
        ch.solve_device(s["b"].data_ptr(), r, n, r, s["x"].data_ptr(), r)
        ch.free()
        return s["x"]
    if op == "qr":
        qr = la_gpu.QRDecomposition.new_device(s["a"].data_ptr(), case["n"], case["m"], case["n"], ctx)
        out = {"r": qr.get_r().data, "q": qr.get_q().data}
        qr.free()
        return out
    if op == "mixed":
        n, r = case["n"], case["nrhs"]
        la_gpu.lu_solve_auto_device(ctx, s["a"].data_ptr(), n, n, s["b"].data_ptr(), r, r,
                                    s["x"].data_ptr(), r, tol=TOL)
        return s["x"]
    if op == "batch":
        s["plan"].run()
        return s["x"]
    if op == "selector":
        la_gpu.batch_features_device(ctx, s["a"].data_ptr(), s["systems"], s["f"].data_ptr())
        s["sel"].predict(s["f"], out=s["cls"], sync=False)
        s["plan"].select_device(s["cls"].data_ptr())
        s["plan"].run()
        return {"x": s["x"], "features": s["f"], "classes": s["cls"]}
    loss = s["mlp"].train_step(s["x"].data_ptr(), s["y"].data_ptr(), case["count"], 3e-3, want_loss=True)
    return {"loss": loss, "params": s["mlp"].get_params()}


# ---- what a pass cannot do without -------------------------------------------------------------


def work(case):
    op = case["op"]
    if op in ("batch", "selector"):
        lo, hi, c = case["nmin"], case["nmax"], case["count"]
        n = np.arange(lo, hi + 1, dtype=np.float64)
        n2, n3 = float((n * n).mean()), float((n ** 3).mean())
        return {"bytes": c * 8 * (n2 + 5 * float(n.mean())), "flops": c * (2 / 3 * n3 + 5 * n2)}
    if op == "train":
        weights = 16 * 64 + 64 * 64 + 64 * 3
        return {"bytes": 68 * case["count"] + 12 * weights, "flops": 6 * weights * case["count"]}
    n, r = case["n"], case.get("nrhs", 0)
    if op in ("solve", "lu", "lu_device", "mixed"):
        lu = 8 * n * n if op == "lu" else 0
        return {"bytes": 8 * (n * n + 2 * n * r) + lu, "flops": 2 / 3 * n ** 3 + 2 * n * n * r}
    if op == "inverse":
        return {"bytes": 16 * n * n, "flops": 2 * n ** 3}
    if op == "chol":
        return {"bytes": 8 * (n * n / 2 + 2 * n * r), "flops": n ** 3 / 3 + 2 * n * n * r}
    m = case["m"]
    if op == "mul":
        k = case["k"]
        return {"bytes": 8 * (m * k + k * n + m * n), "flops": 2 * m * n * k}
    return {"bytes": 8 * (2 * m * n + m * m), "flops": 4 * n * n * (m - n / 3)}


# ---- the same in plain torch, 64 bits ----------------------------------------------------------


def exact(case, seed):
    s = _inputs(case, seed)
    op = case["op"]
    if op == "solve" or (op == "lu_device" and case["n"] <= 8192) or op == "mixed":
        x = torch.linalg.solve(s["a"], s["b"])
        return {"x": x, "piv": None} if op == "lu_device" else x
    if op == "lu":
        lu, piv = torch.linalg.lu_factor(s["a"])
        return {"det": float(torch.linalg.det(s["a"])), "piv": None,
                "x": torch.linalg.lu_solve(lu, piv, s["b"]), "lu": lu}
    if op == "inverse":
        return torch.linalg.inv(s["a"])
    if op == "mul":
        return s["a"] @ s["b"]
    if op == "chol":
        return torch.cholesky_solve(s["b"], torch.linalg.cholesky(s["a"]))
    if op == "qr":
        # Householder factors with LAPACK's signs, which are the crate's; its Q has the first
        # min(m, n) columns and zeros after them.
        q, r = torch.linalg.qr(s["a"], mode="reduced")
        m, n = case["m"], case["n"]
        full = torch.zeros((m, m), dtype=F64, device="cuda")
        full[:, :n] = q
        low = torch.zeros((m, n), dtype=F64, device="cuda")
        low[:n] = r
        return {"r": low, "q": full}
    if op in ("batch", "selector"):
        x = torch.zeros_like(s["b"])
        groups = {}
        for i, (n, r) in enumerate(zip(s["ns"], s["rs"])):
            groups.setdefault((int(n), int(r)), []).append(i)
        for (n, r), ids in groups.items():
            a = torch.stack([s["a"][s["systems"][i].a_offset:][:n * n].view(n, n) for i in ids])
            b = torch.stack([s["b"][s["systems"][i].b_offset:][:n * r].view(n, r) for i in ids])
            y = torch.linalg.solve(a, b)
            for j, i in enumerate(ids):
                x[s["systems"][i].b_offset:][:n * r] = y[j].reshape(-1)
        return {"x": x, "features": None, "classes": None} if op == "selector" else x
    # One Adam step from zero moments on the mean cross-entropy.
    p = torch.from_numpy(s["p"]).double().cuda()
    at, parts = 0, []
    for shape in ((64, 16), (64,), (64, 64), (64,), (3, 64), (3,)):
        k = math.prod(shape)
        parts.append(p[at:at + k].view(shape).clone().requires_grad_(True))
        at += k
    mean, std = p[at:at + 16], p[at + 16:at + 32]
    h = (s["x"].double() - mean) / std
    h = torch.relu(h @ parts[0].t() + parts[1])
    h = torch.relu(h @ parts[2].t() + parts[3])
    loss = torch.nn.functional.cross_entropy(h @ parts[4].t() + parts[5], s["y"].long())
    loss.backward()
    new = [w.detach() - 3e-3 * w.grad / (w.grad.abs() + 1e-8) for w in parts]
    return {"loss": float(loss.detach()), "params": torch.cat([w.reshape(-1) for w in new] + [mean, std])}
