"""Performance cases of the library's public entry points, on seeded synthetic fields.

A case is a dict of plain values with a "kind":

  solve         loadQcuGauge, then qcuInvert of m right-hand sides: a propagator on a new
                configuration (plain FP64 BiCGStab, or the mixed-precision solver)
  mat           loadQcuGauge, then mat_Qcu on full-lattice per-RHS fields (FP64 in and out)
  dslash        loadQcuGauge, then start_dslash on half-lattice per-RHS fields (FP64 in and
                out, the hop in another precision)
  hop, schur    qcuDslashMrhs / qcuSchurMrhs on the caller's gathered fields (a caller with a
                solver of its own)
  blas          the multi-RHS vector operations of one such solver step
  batch         qcuInvertBatch of independent uneven systems with kept contexts (serving loop)
  precond       the learned preconditioner applied to gathered fields
  precond_grad  its training loss and weight gradient (forward, adjoint, weight gradient)

The qcu.h interface holds one process-wide context, so the cases that go through it load
their gauge field in every pass; the context itself is made once per shape.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

import qcu_mrhs_b200 as q
from qcu_mrhs_b200.precond import LearnedPreconditioner

PREC = {"double": q.DOUBLE, "single": q.SINGLE, "half": q.HALF, "bf16": q.BF16}
DTYPE = {"double": torch.float64, "single": torch.float32, "half": torch.float16, "bf16": torch.bfloat16}
BYTES = {"double": 8, "single": 4, "half": 2, "bf16": 2}   # of one real number
MAX_ITER = 5000


# ---------------------------------------------------------------- cases

def listed():
    return [
        # smallest call: one right-hand side on a tiny lattice, where launch latency is everything
        {"name": "hop_f64_4x4x4x4_m1", "kind": "hop", "L": "4x4x4x4", "n": 3, "m": 1, "prec": "double"},
        # the plain solve of the first benchmark configuration: small lattice, Haar links
        {"name": "solve_f64_8x8x8x8_m4", "kind": "solve", "L": "8x8x8x8", "n": 3, "m": 4, "kappa": 0.10, "eps": 0.0,
         "solver": "fused", "sloppy": "bf16", "delta": 0.1, "quorum": 0.0, "true_stop": False, "tol": 1e-10},
        # an ordinary plain solve with an odd number of right-hand sides, the reference's stopping rule
        {"name": "solve_f64_16x16x16x32_m5", "kind": "solve", "L": "16x16x16x32", "n": 3, "m": 5, "kappa": 0.115,
         "eps": 0.3, "solver": "fused", "sloppy": "bf16", "delta": 0.1, "quorum": 0.0, "true_stop": False,
         "tol": 1e-8},
        # the headline benchmark: a whole propagator (12 sources) in mixed precision, near-critical kappa
        {"name": "solve_f16_24x24x24x48_m12", "kind": "solve", "L": "24x24x24x48", "n": 3, "m": 12, "kappa": 0.124,
         "eps": 0.3, "solver": "mixed", "sloppy": "half", "delta": 0.003, "quorum": 1.0, "true_stop": True,
         "tol": 1e-10},
        # mixed precision at the library's default rule (BF16, delta 0.1), a ragged lattice and odd m
        {"name": "solve_bf16_12x10x14x16_m7", "kind": "solve", "L": "12x10x14x16", "n": 3, "m": 7, "kappa": 0.12,
         "eps": 0.4, "solver": "mixed", "sloppy": "bf16", "delta": 0.1, "quorum": 0.0, "true_stop": True,
         "tol": 1e-10},
        # the full operator on the largest lattice through qcu.h: residual checks of a propagator
        {"name": "mat_f64_24x24x24x48_m12", "kind": "mat", "L": "24x24x24x48", "n": 3, "m": 12, "kappa": 0.124,
         "eps": 0.3},
        # the FP64 hop on gathered fields at an ordinary size
        {"name": "hop_f64_16x16x16x32_m12", "kind": "hop", "L": "16x16x16x32", "n": 3, "m": 12, "prec": "double"},
        # 16-bit operator of a caller's own solver, SU(3), from the SU(N) sweep
        {"name": "schur_bf16_16x16x16x16_m16", "kind": "schur", "L": "16x16x16x16", "n": 3, "m": 16, "prec": "bf16"},
        # the wide end of the SU(N) sweep in FP32
        {"name": "hop_f32_16x16x16x16_n6_m8", "kind": "hop", "L": "16x16x16x16", "n": 6, "m": 8, "prec": "single"},
        # uneven systems solved together, as a serving loop calls it
        {"name": "batch_f16_12_systems", "kind": "batch", "systems": 12, "draw": 4, "solver": "mixed",
         "sloppy": "half", "delta": 0.003, "tol": 1e-10},
        # the learned preconditioner at its benchmark size: inference and training
        {"name": "precond_16x16x16x16_m8", "kind": "precond", "L": "16x16x16x16", "n": 3, "m": 8, "layers": 4,
         "channels": 8, "prec": "double"},
        {"name": "precond_grad_8x8x8x16_m8", "kind": "precond_grad", "L": "8x8x8x16", "n": 3, "m": 8, "layers": 4,
         "channels": 8, "prec": "double", "kappa": 0.1245},
    ]


def _lattice(rng, lo, hi):
    """Even extents with a volume between lo and hi, spread over its logarithm."""
    target = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    best = None
    for _ in range(200):
        L = [rng.choice((4, 6, 8, 10, 12, 14, 16, 20, 24)) for _ in range(3)]
        L.append(rng.choice((4, 6, 8, 12, 16, 24, 32, 48)))
        off = abs(math.log(math.prod(L) / target))
        if best is None or off < best[0]:
            best = (off, L)
    return "x".join(str(v) for v in best[1])


def draw(rng):
    kind = rng.choice(("solve", "solve", "mat", "dslash", "hop", "hop", "schur", "blas", "batch", "precond",
                       "precond_grad"))
    if kind == "solve":
        mixed = rng.random() < 0.6
        haar = not mixed and rng.random() < 0.3
        sloppy = rng.choice(("half", "bf16", "single"))
        delta, quorum = rng.choice(((0.1, 0.0), (0.01, 1.0), (0.003, 1.0)))
        return {"kind": kind, "L": _lattice(rng, 256, 140000), "n": 3, "m": rng.randint(1, 12),
                "kappa": round(rng.uniform(0.09, 0.10 if haar else 0.124), 4),
                "eps": 0.0 if haar else round(rng.uniform(0.2, 0.4), 3), "solver": "mixed" if mixed else "fused",
                "sloppy": sloppy, "delta": delta, "quorum": quorum, "true_stop": mixed or rng.random() < 0.5,
                "tol": 1e-10 if mixed else rng.choice((1e-8, 1e-10))}
    if kind in ("mat", "dslash"):
        c = {"kind": kind, "L": _lattice(rng, 256, 300000), "n": rng.choice((2, 3, 3, 3, 4)), "m": rng.randint(1, 16),
             "kappa": round(rng.uniform(0.10, 0.125), 4), "eps": round(rng.uniform(0.2, 0.5), 3)}
        if kind == "dslash":
            c["prec"] = rng.choice(("double", "single", "half", "bf16"))
        return c
    if kind in ("hop", "schur"):
        n = rng.choice((2, 3, 3, 3, 4, 5, 6, 7, 8))
        m = rng.choice((1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 12, 13, 16, 20, 24, 32))
        return {"kind": kind, "L": _lattice(rng, 256, min(600000, 2.0e7 / (n * m))), "n": n, "m": m,
                "prec": rng.choice(("double", "single", "half", "bf16"))}
    if kind == "blas":
        return {"kind": kind, "L": _lattice(rng, 256, 300000), "n": rng.choice((2, 3, 3, 4, 6, 8)),
                "m": rng.randint(1, 16), "prec": rng.choice(("double", "single", "half", "bf16"))}
    if kind == "batch":
        mixed = rng.random() < 0.7
        return {"kind": kind, "systems": rng.randint(2, 12), "draw": rng.randint(1, 10**6),
                "solver": "mixed" if mixed else "fused", "sloppy": rng.choice(("half", "bf16")),
                "delta": rng.choice((0.1, 0.01, 0.003)), "tol": 1e-10}
    channels = rng.choice((2, 3, 4, 6, 8, 8))
    c = {"kind": kind, "L": _lattice(rng, 256, 32768 if kind == "precond" else 6000), "n": rng.choice((2, 3, 3, 3, 4)),
         "m": rng.randint(1, 12), "layers": rng.randint(2, 4), "channels": channels,
         "prec": rng.choice(("double", "single"))}
    if kind == "precond_grad":
        c["kappa"] = round(rng.uniform(0.11, 0.1245), 4)
    return c


# ---------------------------------------------------------------- fields

def _L(case):
    return tuple(int(v) for v in case["L"].split("x"))


def _vh(L):
    return math.prod(L) // 2


def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(seed * 1000003 + salt)


def _gaussian(shape, gen):
    """Complex Gaussian entries of unit variance."""
    z = torch.randn(tuple(shape) + (2,), dtype=torch.float64, device="cuda", generator=gen)
    return torch.view_as_complex(z.mul_(1 / math.sqrt(2)))


def _links(L, n, seed, eps, salt=1):
    """Even/odd gauge field [4][2][Vh][n][n] complex128: exp(i eps H) with H a traceless
    Hermitian Gaussian matrix, or Haar-random SU(n) for eps = 0."""
    gen = _gen(seed, salt)
    count = 8 * _vh(L)
    out = torch.empty((count, n, n), dtype=torch.complex128, device="cuda")
    eye = torch.eye(n, dtype=torch.complex128, device="cuda")
    for s in range(0, count, 1 << 20):
        a = _gaussian((min(count - s, 1 << 20), n, n), gen)
        if eps > 0:
            h = 0.5 * (a + a.mH)
            h -= (torch.diagonal(h, dim1=-2, dim2=-1).sum(-1).real / n)[:, None, None] * eye
            h = h * (1j * eps / 16)
            u = eye + h / 9   # Taylor series of order 9 of exp(h), squared four times
            for k in range(8, 0, -1):
                u = eye + torch.matmul(h, u) / k
            for _ in range(4):
                u = torch.matmul(u, u)
        else:
            cols = []   # Gram-Schmidt on the columns, twice, then the phase of the determinant
            for c in range(n):
                v = a[:, :, c]
                for _ in range(2):
                    for p in cols:
                        v = v - p * (p.conj() * v).sum(-1, keepdim=True)
                cols.append(v / torch.linalg.vector_norm(v, dim=-1, keepdim=True))
            u = torch.stack(cols, -1)
            u = u * torch.polar(torch.ones(len(u), dtype=torch.float64, device="cuda"),
                                -torch.linalg.det(u).angle() / n)[:, None, None]
        out[s:s + len(u)] = u
    return out.reshape(4, 2, _vh(L), n, n)


def _store(z, prec):
    """Complex tensor -> storage tensor [..., 2] of a precision."""
    return torch.view_as_real(z).to(DTYPE[prec]).contiguous()


def _load(t):
    """Storage tensor -> complex128."""
    return torch.view_as_complex(t.to(torch.float64).contiguous())


def _specs(case):
    """The systems of a batch: lattices, RHS counts, kappa and link smoothing."""
    rng = random.Random(case["draw"])
    out = []
    for _ in range(case["systems"]):
        out.append({"L": rng.choice(("8x8x8x8", "12x12x12x12", "16x16x16x32")), "n": 3, "m": rng.randint(1, 16),
                    "kappa": round(rng.uniform(0.10, 0.124), 5), "eps": round(rng.uniform(0.2, 0.5), 3)})
    return out


def _weights(case, seed):
    """Layer weights near the identity network with every path in use (as after training)."""
    gen = _gen(seed, 7)
    ws = []
    for l in range(case["layers"]):
        cin = 1 if l == 0 else case["channels"]
        cout = 1 if l == case["layers"] - 1 else case["channels"]
        w = 0.05 * _gaussian((cout, cin, 9, 4, 4), gen)
        w[0, 0, 0] += torch.eye(4, dtype=torch.complex128, device="cuda")
        ws.append(w.to(torch.complex64).cpu().numpy())
    return ws


def _inputs(case, seed):
    """The fields of a case in the precisions its entry point takes."""
    kind = case["kind"]
    if kind == "batch":
        return [_inputs(dict(s, kind="solve"), seed + 7919 * (i + 1)) for i, s in enumerate(_specs(case))]
    L, n, m = _L(case), case["n"], case["m"]
    vh = _vh(L)
    gen = _gen(seed, 2)
    if kind in ("solve", "mat"):
        return {"gauge": _store(_links(L, n, seed, case["eps"]), "double"),
                "src": _store(_gaussian((m, 2, vh, 4, n), gen), "double")}
    if kind == "dslash":
        return {"gauge": _store(_links(L, n, seed, case["eps"]), "double"),
                "src": _store(_gaussian((m, vh, 4, n), gen), "double")}
    if kind in ("hop", "schur"):
        return {"gauge": _store(_links(L, n, seed, 0.0), case["prec"]),
                "src": _store(_gaussian((vh, 4, n, m), gen), case["prec"])}
    if kind == "blas":
        x = _gaussian((vh, 4, n, m), gen)
        y = 0.5 * x + _gaussian((vh, 4, n, m), gen)
        return {"x": _store(x, case["prec"]), "y": _store(y, case["prec"]),
                "a": _store(_gaussian((3, m), gen), "double")}
    return {"gauge": _store(_links(L, n, seed, 0.3), "double"),
            "src": _store(_gaussian((2, vh, 4, n, m), gen), case["prec"]), "w": _weights(case, seed)}


# ---------------------------------------------------------------- passes

_context_key = None


def _context(case):
    """The process-wide qcu.h context of a case's shape (made when another one is current)."""
    global _context_key
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key == _context_key:
        return
    lib = q.lib()
    grid = q.QcuGrid((ctypes.c_int * 4)(1, 1, 1, 1))
    param = q.QcuParam((ctypes.c_int * 4)(*_L(case)))
    hop = PREC[case["prec"]] if case["kind"] == "dslash" else q.DOUBLE
    lib.initGridSize(ctypes.byref(grid), ctypes.byref(param), case["n"], case["m"], q.DOUBLE, hop)
    q.check()
    o = q.default_options()
    o.t_boundary = -1.0
    if case["kind"] == "solve":
        o.solver = q.SOLVER_MIXED if case["solver"] == "mixed" else q.SOLVER_FUSED
        o.sloppy_precision = PREC[case["sloppy"]]
        o.reliable_delta, o.reliable_quorum = case["delta"], case["quorum"]
        o.stop_true_residual = int(case["true_stop"])
        o.check_interval = 16
    q.check(lib.qcuSetSolverOptions(ctypes.byref(o)))
    lib.getDslash(0, 1.0 / (2 * case["kappa"]) - 4.0)
    q.check()
    _context_key = key


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "in": _inputs(case, seed)}
    d = s["in"]
    if kind == "batch":
        s["out"] = [torch.empty_like(e["src"]) for e in d]
        arr = (q.QcuBatchSystem * len(d))()
        s["keep"] = []
        for a, spec, e, x in zip(arr, _specs(case), d, s["out"]):
            bp = q.ptr_array([t.data_ptr() for t in e["src"]])
            xp = q.ptr_array([t.data_ptr() for t in x])
            s["keep"] += [bp, xp]
            a.lattice_size[:] = list(_L(spec))
            a.n_color, a.m_rhs, a.kappa, a.tol = spec["n"], spec["m"], spec["kappa"], case["tol"]
            a.max_iteration = MAX_ITER
            a.gauge = e["gauge"].data_ptr()
            a.b = ctypes.cast(bp, ctypes.POINTER(ctypes.c_void_p))
            a.x = ctypes.cast(xp, ctypes.POINTER(ctypes.c_void_p))
        o = q.default_options()
        o.solver = q.SOLVER_MIXED if case["solver"] == "mixed" else q.SOLVER_FUSED
        o.sloppy_precision = PREC[case["sloppy"]]
        o.stop_true_residual = 1
        o.t_boundary = -1.0
        o.reliable_delta = case["delta"]
        o.check_interval = 16
        s["systems"], s["opts"] = arr, o
    elif kind in ("solve", "mat", "dslash"):
        s["out"] = torch.empty_like(d["src"])
        _context(case)
    elif kind in ("hop", "schur"):
        s["out"], s["tmp"] = torch.empty_like(d["src"]), torch.empty_like(d["src"])
        s["L"] = q.lattice(_L(case))
    elif kind == "blas":
        m = case["m"]
        s["dot"] = torch.empty((m, 2), dtype=torch.float64, device="cuda")
        s["norm"] = torch.empty(m, dtype=torch.float64, device="cuda")
        s["out"] = [torch.empty_like(d["x"]) for _ in range(3)]
    else:
        P = LearnedPreconditioner(_L(case), case["n"], case["m"], case["layers"], case["channels"], t_boundary=-1.0)
        P.set_weights(d.pop("w"))
        P.set_gauge(d["gauge"])
        s["P"], s["out"] = P, torch.empty_like(d["src"])
    return s


def run(s):
    case, d = s["case"], s["in"]
    kind = case["kind"]
    lib = q.lib()
    if kind == "batch":
        q.check(lib.qcuInvertBatch(s["systems"], len(s["systems"]), ctypes.byref(s["opts"]), q.BATCH_KEEP_CONTEXTS))
        return s["out"]
    if kind in ("solve", "mat", "dslash"):
        _context(case)
        lib.loadQcuGauge(d["gauge"].data_ptr(), q.DOUBLE)
        for j in range(case["m"]):
            lib.pushBackFermions(s["out"][j].data_ptr(), d["src"][j].data_ptr())
        if kind == "solve":
            lib.qcuInvert(MAX_ITER, case["tol"])
        elif kind == "mat":
            lib.mat_Qcu(0)
        else:
            lib.start_dslash(0, 0)
        q.check()
        return s["out"]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if kind == "hop":
        q.check(lib.qcuDslashMrhs(s["out"].data_ptr(), d["src"].data_ptr(), d["gauge"].data_ptr(), s["L"], case["n"],
                                  case["m"], 0, 0, -1.0, PREC[case["prec"]], stream))
        return s["out"]
    if kind == "schur":
        q.check(lib.qcuSchurMrhs(s["out"].data_ptr(), d["src"].data_ptr(), s["tmp"].data_ptr(),
                                 d["gauge"].data_ptr(), 0.08, s["L"], case["n"], case["m"], -1.0, PREC[case["prec"]],
                                 stream))
        return s["out"]
    if kind == "blas":
        x, y, a = d["x"].data_ptr(), d["y"].data_ptr(), [t.data_ptr() for t in d["a"]]
        o = [t.data_ptr() for t in s["out"]]
        n, m, p = _vh(_L(case)) * 4 * case["n"], case["m"], PREC[case["prec"]]
        q.check(lib.qcuMrhsDotc(s["dot"].data_ptr(), x, y, n, m, p, stream))
        q.check(lib.qcuMrhsNorm(s["norm"].data_ptr(), y, n, m, p, stream))
        q.check(lib.qcuMrhsXsay(o[0], x, a[0], y, n, m, p, stream))
        q.check(lib.qcuMrhsAxpby(o[1], a[0], x, a[1], y, n, m, p, stream))
        q.check(lib.qcuMrhsAxpbypcz(o[2], a[0], x, a[1], y, a[2], o[0], n, m, p, stream))
        return [s["dot"], s["norm"]] + s["out"]
    if kind == "precond":
        s["P"].apply(s["out"], d["src"], PREC[case["prec"]], stream)
        return s["out"]
    loss, grad = s["P"].loss_grad(d["src"], case["kappa"], PREC[case["prec"]])
    return {"loss": loss, "grad": grad}


# ---------------------------------------------------------------- work and tolerance

def _hop_work(vh, n, m, b):
    return {"bytes": vh * (16 * n * n * b + 16 * n * m * b), "flops": vh * m * (128 * n * n + 56 * n)}


def _solve_work(c, sloppy, tol):
    """Inputs and outputs once, and for each iteration (about two per e-fold of the residual)
    the operator twice: four hops that each read and write a field in the iteration's precision."""
    L = _L(c)
    it = 2 * math.log(1 / tol)
    h = _hop_work(_vh(L), c["n"], c["m"], BYTES[sloppy])
    io = 16 * _vh(L) * (8 * c["n"] ** 2 + 16 * c["n"] * c["m"])
    return {"bytes": io + 4 * it * h["bytes"], "flops": 4 * it * h["flops"]}


def work(case):
    kind = case["kind"]
    mixed = case.get("solver") == "mixed"
    if kind == "batch":
        ws = [_solve_work(s, case["sloppy"] if mixed else "double", case["tol"]) for s in _specs(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if kind == "solve":
        return _solve_work(case, case["sloppy"] if mixed else "double", case["tol"])
    L, n, m = _L(case), case["n"], case["m"]
    vh = _vh(L)
    if kind == "mat":    # the gauge field, the input and the output once, both parities
        return {"bytes": 16 * vh * (8 * n * n + 16 * n * m), "flops": 2 * vh * m * (128 * n * n + 60 * n)}
    if kind == "dslash":
        return {"bytes": 16 * vh * (8 * n * n + 8 * n * m), "flops": vh * m * (128 * n * n + 56 * n)}
    b = BYTES.get(case.get("prec"), 8)
    if kind == "hop":
        return _hop_work(vh, n, m, b)
    if kind == "schur":  # D_oe D_eo: the links and the input once, the output once, and the vector between
        w = _hop_work(vh, n, m, b)
        return {"bytes": 2 * w["bytes"], "flops": 2 * w["flops"]}
    if kind == "blas":   # each operation reads its vectors and writes its result
        return {"bytes": 12 * 2 * b * vh * 4 * n * m, "flops": vh * 4 * n * m * (8 + 4 + 8 + 14 + 22)}
    layers, ch = case["layers"], case["channels"]
    flops = 0.0
    for l in range(layers):
        cin, cout = (1 if l == 0 else ch), (1 if l == layers - 1 else ch)
        flops += 2 * vh * m * 8 * (9 * cin * cout * 16 * n + 8 * min(cin, cout) * 4 * n * n)
    field = 2 * vh * 4 * n * m * 2
    if kind == "precond":
        return {"bytes": 2 * field * b + 64 * vh * n * n, "flops": flops}
    return {"bytes": field * b + 64 * vh * n * n + 2 * 4 * field * (1 + ch * (layers - 1)), "flops": 3 * flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("solve", "batch"):
        return {"rel": 30 * case["tol"]}   # two solutions, each with a residual below tol
    if kind == "mat":
        return {"rel": 2e-15, "max": 2e-13}
    if kind == "precond":
        return {"rel": 5e-6}
    if kind == "precond_grad":
        return {"rel": 4e-6}
    return {"double": {"rel": 2e-15, "max": 2e-13}, "single": {"rel": 5e-7}, "half": {"rel": 2e-3, "max": 3e-2},
            "bf16": {"rel": 1.5e-2, "max": 0.25}}[case["prec"]]


# ---------------------------------------------------------------- plain torch in 64 bits

# lower half of (1 + s g_mu) in the chiral basis: half spinors h0 = p0 + s c0 p_a, h1 = p1 + s c1 p_b;
# spins 2 and 3 of the result take s d2 w_e and s d3 w_f
_PROJ = {0: (3, 1j, 2, 1j, 1, -1j, 0, -1j), 1: (3, -1, 2, 1, 1, 1, 0, -1), 2: (2, 1j, 3, -1j, 0, -1j, 1, 1j),
         3: (2, 1, 3, 1, 0, 1, 1, 1)}


def _neighbours(L, parity):
    """{(mu, forward): (half index of the neighbour, crosses the t boundary)} of one parity's sites."""
    X, Y, Z, T = L
    i = torch.arange(_vh(L), device="cuda")
    xh, r = i % (X // 2), i // (X // 2)
    y, r = r % Y, r // Y
    z, t = r % Z, r // Z
    x = 2 * xh + ((parity + y + z + t) & 1)
    out = {}
    for mu in range(4):
        for fwd in (True, False):
            c = [x, y, z, t]
            c[mu] = (c[mu] + (1 if fwd else -1)) % L[mu]
            wrap = (t == (T - 1 if fwd else 0)) if mu == 3 else torch.zeros_like(t, dtype=torch.bool)
            out[mu, fwd] = (((c[3] * Z + c[2]) * Y + c[1]) * (X // 2) + torch.div(c[0], 2, rounding_mode="floor"),
                            wrap)
    return out


def _transport(u, psi, nbr, parity, mu, fwd, t_sign):
    """U_mu(x) psi(x + mu) or U_mu(x - mu)^dag psi(x - mu) on [Vh][s][N][m] (psi of the other parity)."""
    idx, wrap = nbr[mu, fwd]
    link = u[mu, parity] if fwd else u[mu, 1 - parity][idx].mH
    w = torch.einsum("xab,xsbm->xsam", link, psi[idx])
    return torch.where(wrap[:, None, None, None], t_sign * w, w)


def _hop(u, psi, L, parity, t_sign=-1.0, dagger=False):
    nbr = _neighbours(L, parity)
    out = torch.zeros_like(psi)
    for mu in range(4):
        a, c0, b, c1, e, d2, f, d3 = _PROJ[mu]
        for fwd in (True, False):
            s = -1 if fwd != dagger else 1
            h = torch.stack((psi[:, 0] + s * c0 * psi[:, a], psi[:, 1] + s * c1 * psi[:, b]), 1)
            w = _transport(u, h, nbr, parity, mu, fwd, t_sign)
            out[:, :2] += w
            out[:, 2] += s * d2 * w[:, e]
            out[:, 3] += s * d3 * w[:, f]
    return out


def _full(u, v, kappa, L, dagger=False):
    """(1 - kappa D) v on [2][Vh][4][N][m]."""
    return torch.stack([v[p] - kappa * _hop(u, v[1 - p], L, p, dagger=dagger) for p in (0, 1)])


def _solve_exact(c, d):
    """M x = b in 64 bits: BiCGStab on the odd Schur system until the residual stops at rounding."""
    L, kappa = _L(c), c["kappa"]
    u = _load(d["gauge"])
    be, bo = (t.contiguous() for t in _load(d["src"]).permute(1, 2, 3, 4, 0))

    def schur(v):
        return v - kappa * kappa * _hop(u, _hop(u, v, L, 0), L, 1)

    def dot(a, b):
        return (a.conj() * b).sum((0, 1, 2))

    bp = bo + kappa * _hop(u, be, L, 1)
    x, r, r0, p = torch.zeros_like(bp), bp.clone(), bp.clone(), bp.clone()
    rho, ref = dot(r0, r), dot(bp, bp).real
    for _ in range(400):
        v = schur(p)
        alpha = rho / dot(r0, v)
        sv = r - alpha * v
        t = schur(sv)
        omega = dot(t, sv) / dot(t, t).real
        x += alpha * p + omega * sv
        r = sv - omega * t
        if bool((dot(r, r).real <= 1e-27 * ref).all()):
            break
        new = dot(r0, r)
        p = r + (new / rho * alpha / omega) * (p - omega * v)
        rho = new
    xe = be + kappa * _hop(u, x, L, 0)
    return torch.view_as_real(torch.stack((xe, x)).permute(4, 0, 1, 2, 3).contiguous())


def _net(u, v, ws, L):
    """The parallel-transport network on [2][Vh][4][N][m]."""
    nbr = [_neighbours(L, p) for p in (0, 1)]
    f = v[None]
    for w in ws:
        out = 0
        for k in range(9):
            if k == 0:
                t = f
            else:
                mu, fwd = (k - 1) // 2, (k - 1) % 2 == 0
                t = torch.stack([torch.stack([_transport(u, c[1 - p], nbr[p], p, mu, fwd, -1.0) for p in (0, 1)])
                                 for c in f])
            out = out + torch.einsum("oiab,ipxbcm->opxacm", w[:, :, k], t)
        f = out
    return f[0]


def exact(case, seed):
    kind = case["kind"]
    cost = work(case)
    if kind in ("solve", "batch") and cost["bytes"] > 1.2e11 * (2 if case.get("solver") == "fused" else 1):
        return None
    d = _inputs(case, seed)
    if kind == "batch":
        return [_solve_exact(s, e) for s, e in zip(_specs(case), d)]
    if kind == "solve":
        return _solve_exact(case, d)
    L = _L(case)
    if kind == "blas":
        x, y, a = _load(d["x"]), _load(d["y"]), _load(d["a"])
        o0 = x - a[0] * y
        o0s = _load(_store(o0, case["prec"]))   # the step reads this vector back as it was stored
        outs = [o0, a[0] * x + a[1] * y, a[0] * x + a[1] * y + a[2] * o0s]
        return [torch.view_as_real((x.conj() * y).sum((0, 1, 2))), torch.linalg.vector_norm(y, dim=(0, 1, 2))] + \
            [torch.view_as_real(t) for t in outs]
    u = _load(d["gauge"])
    if kind == "mat":
        v = _load(d["src"]).permute(1, 2, 3, 4, 0).contiguous()
        return torch.view_as_real(_full(u, v, case["kappa"], L).permute(4, 0, 1, 2, 3).contiguous())
    if kind == "dslash":
        v = _load(d["src"]).permute(1, 2, 3, 0).contiguous()
        return torch.view_as_real(_hop(u, v, L, 0).permute(3, 0, 1, 2).contiguous())
    v = _load(d["src"])
    if kind == "hop":
        return torch.view_as_real(_hop(u, v, L, 0))
    if kind == "schur":
        return torch.view_as_real(v - 0.08 ** 2 * _hop(u, _hop(u, v, L, 0), L, 1))
    ws = [torch.from_numpy(w.astype(np.complex128)).cuda() for w in d["w"]]
    if kind == "precond":
        return torch.view_as_real(_net(u, v, ws, L))
    for w in ws:
        w.requires_grad_(True)
    r = _full(u, _net(u, v, ws, L), case["kappa"], L) - v
    loss = ((r.abs() ** 2).sum((0, 1, 2, 3)) / (v.abs() ** 2).sum((0, 1, 2, 3))).sum()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": [w.grad.cpu().numpy() for w in ws]}
