"""Performance cases of the framework: the calls its users make, with the sizes they make them at.

Each case goes through a public entry point: solves through the XAMG C API (XAMG_solver_solve2,
XAMG_b200_solver_solve_batch), the kernel-level calls on device arrays (XAMG_b200_spmv,
XAMG_b200_dot, XAMG_b200_gemm_bf16) and the learned guess's MLP (XAMG_b200_mlp_*).

  listed()              the fixed cases
  draw(rng)             one more case of the same ranges
  prepare(case, seed)   what a program holds before the call, on the GPU
  run(state)            one pass, and its outputs
  work(case)            bytes and operations one pass cannot do without
  tolerance(case)       how far another correct implementation may be off
  exact(case, seed)     the outputs in 64 bits, in plain torch

A solve's matrix belongs to the case (a program assembles it once and solves with many right-hand
sides); the right-hand sides come from the seed. Everything else comes from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "softx-d-21-00014_b200"))
import xamg_b200 as X  # noqa: E402

# Nonzeros a row of the generated matrices, rows of the whole AMG hierarchy's operators included,
# per row of the finest level (operator complexity, as the setup builds it).
PER_ROW = {7: 6.9, 27: 26.4}
COMPLEXITY = {7: 2.6, 27: 1.4}


def listed():
    return [
        # the reference's own example problem: 7-point Poisson, one right-hand side, Jacobi;
        # the smallest solve a user runs, bound by latency
        {"name": "solve_poisson32_jacobi", "kind": "solve", "stencil": 0, "nx": 32, "ny": 32,
         "nz": 32, "sigma": 0.0, "aniso": 1.0, "nv": 1, "form": "fp64", "precond": "Jacobi",
         "order": 0, "sweeps": 1},
        # the benchmark's method (27-point finite elements, eight right-hand sides, V(1,1) with
        # Chebyshev-2) in its chosen form: FP32 cycle, BF16 values on the two finest levels
        {"name": "solve_fe27_96_nv8_chosen", "kind": "solve", "stencil": 27, "nx": 96, "ny": 96,
         "nz": 96, "sigma": 1.0, "aniso": 1.0, "nv": 8, "form": "bf16", "precond": "Chebyshev",
         "order": 2, "sweeps": 1},
        # the same method in plain FP64, as a user of the reference runs it, on an uneven grid
        {"name": "solve_fe27_64_nv8_fp64", "kind": "solve", "stencil": 27, "nx": 67, "ny": 64,
         "nz": 61, "sigma": 1.0, "aniso": 1.0, "nv": 8, "form": "fp64", "precond": "Chebyshev",
         "order": 2, "sweeps": 1},
        # many right-hand sides on an anisotropic, high-contrast matrix: V(2,2), Chebyshev-3, FP32
        {"name": "solve_aniso27_48_nv32_f32", "kind": "solve", "stencil": 27, "nx": 48, "ny": 48,
         "nz": 48, "sigma": 2.0, "aniso": 4.0, "nv": 32, "form": "f32", "precond": "Chebyshev",
         "order": 3, "sweeps": 2},
        # a 7-point matrix, one right-hand side, Gauss-Seidel smoothers: a single small AMG solve
        {"name": "solve_fv7_40_nv1_hsgs", "kind": "solve", "stencil": 7, "nx": 43, "ny": 40,
         "nz": 37, "sigma": 1.5, "aniso": 1.0, "nv": 1, "form": "f32", "precond": "HSGS",
         "order": 0, "sweeps": 1},
        # uneven independent systems solved in one call, Gauss-Seidel smoothers in FP32
        {"name": "batch12_fv7_hsgs", "kind": "batch", "systems": 12, "lo": 16, "hi": 48,
         "pick": 3, "sigma": 1.5},
        # y = A x on a caller's matrix: the finest level of the benchmark, FP64, 32-bit columns
        {"name": "spmv_fe27_128_nv8_f64", "kind": "spmv", "pattern": "box27", "nx": 128,
         "ny": 128, "nz": 128, "nv": 8, "dtype": "f64", "col_bytes": 4, "mode": 0},
        # y += A x, one right-hand side, FP32, odd sizes
        {"name": "spmv_fv7_odd_nv1_f32", "kind": "spmv", "pattern": "star7", "nx": 211, "ny": 173,
         "nz": 97, "nv": 1, "dtype": "f32", "col_bytes": 4, "mode": 1},
        # a dot product of short vectors: the smallest call there is
        {"name": "dot_30k_nv1", "kind": "dot", "n": 30011, "nv": 1},
        # the learned guess applied to one block of right-hand sides (5,242 coarse unknowns)
        {"name": "mlp_predict_b128", "kind": "mlp_predict", "width": 5248, "hidden": 1024,
         "batch": 128},
        # a refresh of a trained guess: Adam steps on mini-batches (forward, backward, update)
        {"name": "mlp_train_b512", "kind": "mlp_train", "width": 5248, "hidden": 1024,
         "batch": 512, "steps": 24},
        # the first dense layer over a whole training set
        {"name": "gemm_4096x1024x5248_relu", "kind": "gemm", "m": 4096, "n": 1024, "k": 5248,
         "mode": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "spmv", "spmv", "dot", "mlp_predict",
                       "mlp_train", "gemm"])
    if kind == "solve":
        precond = rng.choice(["Jacobi", "Chebyshev", "Chebyshev", "HSGS"])
        stencil = rng.choice([7, 27])
        nv = rng.choice([1, 2, 4, 8, 16, 32])
        # rows x nv at most 40^3 x 32, rows at most 64^3
        cap = min(64.0, (40.0 ** 3 * 32 / nv) ** (1 / 3))
        e = [_log(rng, 14, cap) for _ in range(3)]
        return {"kind": kind, "stencil": stencil, "nx": e[0], "ny": e[1], "nz": e[2],
                "sigma": rng.choice([0.5, 1.0, 1.5]), "aniso": rng.choice([1.0, 1.0, 4.0]),
                "nv": nv, "form": rng.choice(["fp64", "f32", "bf16"]) if precond != "Jacobi"
                else "fp64", "precond": precond, "order": rng.choice([2, 3]),
                "sweeps": rng.choice([1, 1, 2])}
    if kind == "batch":
        return {"kind": kind, "systems": rng.randint(4, 12), "lo": 16,
                "hi": rng.choice([24, 32, 40, 48]), "pick": rng.randrange(1 << 16),
                "sigma": rng.choice([0.5, 1.0, 1.5])}
    if kind == "spmv":
        pattern = rng.choice(["box27", "star7", "ragged"])
        nv = rng.choice([1, 2, 4, 8, 16, 32])
        col_bytes = rng.choice([4, 4, 2])
        top = min(2097152.0 * 8 / nv, 1500000.0)
        n = _log(rng, 900, min(top, 60000.0) if col_bytes == 2 else top)
        e = max(3, int(round(n ** (1 / 3))))
        nx, ny = max(3, e + rng.randint(-e // 4, e // 4)), max(3, e + rng.randint(-e // 4, e // 4))
        return {"kind": kind, "pattern": pattern, "nx": nx, "ny": ny,
                "nz": max(1, n // (nx * ny)), "nv": nv, "dtype": rng.choice(["f64", "f32"]),
                "col_bytes": col_bytes, "mode": rng.choice([0, 1])}
    if kind == "dot":
        nv = rng.choice([1, 2, 4, 8, 16, 32])
        return {"kind": kind, "n": _log(rng, 1000, 16000000 // nv), "nv": nv}
    if kind == "gemm":
        return {"kind": kind, "m": 128 * _log(rng, 1, 32), "n": 128 * _log(rng, 2, 41),
                "k": 64 * _log(rng, 4, 82), "mode": rng.choice([0, 1, 2])}
    c = {"kind": kind, "width": 128 * _log(rng, 4, 41), "hidden": 128 * _log(rng, 2, 8),
         "batch": 128 * _log(rng, 1, 8)}
    return dict(c, steps=rng.randint(8, 24)) if kind == "mlp_train" else c


# ------------------------------------------------------------------------------ inputs
class Handle:
    """Library objects freed with the state that holds them."""

    def __init__(self, **kw):
        self.__dict__.update(kw)
        self.owned = []

    def own(self, destroy, obj):
        self.owned.append((destroy, obj.h))
        return obj

    def __del__(self):
        try:
            for destroy, h in reversed(self.owned):
                X.call(destroy, h)
        except Exception:
            pass


class DeviceVector(X.Vector):
    """A library vector that torch can view; a view keeps the vector alive."""

    def __init__(self, n, nv):
        super().__init__(n, nv)
        self.__cuda_array_interface__ = {"shape": (n, nv), "typestr": "<f8",
                                         "data": (self.device_ptr(), False), "version": 2}

    def __del__(self):
        try:
            X.call("XAMG_vector_destroy", self.h)
        except Exception:
            pass


_matrices = {}


def _host_matrix(stencil, nx, ny, nz, sigma, aniso, mseed):
    if stencil == 0:
        return X.generate_cube(nx, ny, nz)
    return X.generate_diffusion(stencil, nx, ny, nz, sigma, aniso, mseed)


def _matrix(*key):
    """The assembled matrix of a solve; the last few are kept, as a program keeps its matrix
    (its multigrid hierarchy is built by the first solver on it)."""
    if key not in _matrices:
        while len(_matrices) >= 16:
            _matrices.pop(next(iter(_matrices)))
        h = Handle()
        h.m = X.Matrix(*_host_matrix(*key))
        h.owned.append(("XAMG_matrix_destroy", h.m.h))
        _matrices[key] = h
    return _matrices[key]


def _params(form, precond, order, sweeps):
    solver = {"method": "MergedPBiCGStab", "max_iters": 1000, "rel_tolerance": 1e-8,
              "abs_tolerance": 0}
    if precond == "Jacobi":
        return {"solver": solver, "preconditioner": {"method": "Jacobi"}}
    sm = {"method": precond}
    if precond == "Chebyshev":
        sm["polynomial_order"] = order
    if sweeps != 1:
        sm["max_iters"] = sweeps
    prec = {"method": "MultiGrid", "max_iters": 1, "mg_agg_num_levels": 0,
            "mg_strength_threshold": 0.25, "mg_coarsening_type": 8, "mg_interpolation_type": 6,
            "mg_coarse_matrix_size": 500, "mg_reduced_precision": 0}
    if form != "fp64":
        prec["gpu_precond_f32"] = 1
        prec["gpu_index_compress"] = solver["gpu_index_compress"] = 2
    if form == "bf16":
        prec["gpu_level_bf16"] = 2
    return {"solver": solver, "preconditioner": prec, "pre_smoother": sm,
            "post_smoother": dict(sm), "coarse_grid_solver": {"method": "Direct"}}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _rhs(n, nv, seed):
    return torch.empty(n, nv, dtype=torch.float64, device="cuda").uniform_(-1, 1,
                                                                           generator=_gen(seed))


def _systems(case):
    """(matrix key, nv) of every system a solve or a batch has."""
    if case["kind"] == "solve":
        return [((case["stencil"], case["nx"], case["ny"], case["nz"], case["sigma"],
                  case["aniso"], 0), case["nv"])]
    r = np.random.default_rng(case["pick"])
    edges = [e for e in (16, 24, 32, 40, 48) if case["lo"] <= e <= case["hi"]]
    out = []
    for i in range(case["systems"]):
        e = int(edges[r.integers(len(edges))])
        out.append(((7, e, e, e, case["sigma"], 1.0, i), int((1, 4, 16)[r.integers(3)])))
    return out


def _system_of(case, state, key, nv, seed):
    prm = (case.get("form", "f32"), case.get("precond", "HSGS"), case.get("order", 0),
           case.get("sweeps", 1))
    mh = _matrix(*key)
    n = mh.m.n
    b, x = DeviceVector(n, nv), DeviceVector(n, nv)
    rhs = _rhs(n, nv, seed)
    torch.cuda.synchronize()
    X.call("XAMG_vector_upload_d", rhs.data_ptr(), n, 0, nv, b.h)
    x.set(0.0)
    p = state.own("XAMG_param_destroy", X.Params(_params(*prm)))
    s = state.own("XAMG_solver_destroy", X.Solver(mh.m, p, x, b))
    state.keep.append(mh)
    return s, x, b


def _csr(case, seed):
    """Random CSR on the GPU: (row u32, columns as int64, values f64, ncols)."""
    g = _gen(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    i = torch.arange(n, device="cuda")
    if case["pattern"] == "ragged":
        # uneven rows as coarse multigrid levels have them: 1 to 120 entries, some empty
        deg = torch.randint(0, 121, (n,), device="cuda", generator=g)
        deg = deg * (torch.rand(n, device="cuda", generator=g) < 0.6) + deg // 8
        row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        row[1:] = deg.cumsum(0)
        nnz = int(row[-1])
        r = torch.repeat_interleave(i, deg)
        band = max(64, n // 16)
        off = torch.randint(-band, band + 1, (nnz,), device="cuda", generator=g)
        key, _ = torch.sort(r * (n + 1) + (r + off).clamp_(0, n - 1))
        col = key % (n + 1)
    else:
        ix, iy, iz = i % nx, (i // nx) % ny, i // (nx * ny)
        offs = [(dz, dy, dx) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)
                if case["pattern"] == "box27" or abs(dz) + abs(dy) + abs(dx) <= 1]
        ok = torch.stack([((ix + dx >= 0) & (ix + dx < nx) & (iy + dy >= 0) & (iy + dy < ny) &
                           (iz + dz >= 0) & (iz + dz < nz)) for dz, dy, dx in offs], 1)
        row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        row[1:] = ok.sum(1).cumsum(0)
        d = torch.tensor([(dz * ny + dy) * nx + dx for dz, dy, dx in offs], device="cuda")
        col = (i[:, None] + d[None, :])[ok]
        del ok
    val = torch.empty(col.numel(), dtype=torch.float64, device="cuda").uniform_(-1, 1, generator=g)
    if case["dtype"] == "f32":
        val = val.float()
    x = torch.empty(n, case["nv"], dtype=val.dtype, device="cuda").uniform_(-1, 1, generator=g)
    y = torch.empty(n, case["nv"], dtype=val.dtype, device="cuda").uniform_(-1, 1, generator=g)
    return row, col, val, x, y


def _mlp_inputs(case, seed):
    """Parameters (uniform in +-1/sqrt(fan in)), inputs scaled to norm 1 a row and targets."""
    g = _gen(seed)
    w, h, b = case["width"], case["hidden"], case["batch"]
    parts = []
    for fan_in, fan_out in ((w, h), (h, h), (h, w)):
        a = 1 / math.sqrt(fan_in)
        parts.append(torch.empty(fan_out * fan_in, device="cuda").uniform_(-a, a, generator=g))
        parts.append(torch.empty(fan_out, device="cuda").uniform_(-a, a, generator=g))
    sets = 4 if case["kind"] == "mlp_train" else 1
    F = [torch.randn(b, w, device="cuda", generator=g) / math.sqrt(w) for _ in range(sets)]
    T = [torch.randn(b, w, device="cuda", generator=g) for _ in range(sets)]
    return parts, F, T


def _gemm_inputs(case, seed):
    g = _gen(seed)
    m, n, k = case["m"], case["n"], case["k"]
    A = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    B = (torch.randn(n, k, device="cuda", generator=g) / math.sqrt(k)).bfloat16()
    return A, B, torch.randn(n, device="cuda", generator=g)


# ------------------------------------------------------------------------------ passes
def prepare(case, seed):
    X.init()
    kind = case["kind"]
    st = Handle(case=case, kind=kind, keep=[], stream=X.stream())
    if kind in ("solve", "batch"):
        st.sys = [_system_of(case, st, key, nv, seed + 7919 * i)
                  for i, (key, nv) in enumerate(_systems(case))]
        st.out = [torch.as_tensor(x, device="cuda") for _, x, _ in st.sys]
    elif kind == "spmv":
        row, col, val, st.x, st.y = _csr(case, seed)
        st.keep = [row.to(torch.int32),
                   col.to(torch.int16 if case["col_bytes"] == 2 else torch.int32), val]
        n = row.numel() - 1
        st.csr = X.Csr(n, n, col.numel(), st.keep[0].data_ptr(), st.keep[1].data_ptr(),
                       st.keep[2].data_ptr(), case["col_bytes"], int(case["dtype"] == "f32"))
        st.y0 = st.y.clone()
        st.ext = torch.cuda.ExternalStream(st.stream)
    elif kind == "dot":
        st.x, st.y = _rhs(case["n"], case["nv"], seed), _rhs(case["n"], case["nv"], seed + 1)
        st.o = np.zeros(case["nv"])
    elif kind == "gemm":
        st.A, st.B, st.bias = _gemm_inputs(case, seed)
        st.C = torch.empty(case["m"], case["n"], device="cuda",
                           dtype=torch.float32 if case["mode"] == 0 else torch.bfloat16)
    else:
        parts, st.F, st.T = _mlp_inputs(case, seed)
        st.mlp = X.Mlp(case["width"], case["hidden"], case["width"], 0)
        st.mlp.set_params(torch.cat(parts).cpu().numpy())
        st.Y = torch.empty(case["batch"], case["width"], device="cuda")
    torch.cuda.synchronize()
    return st


def run(st):
    case, kind = st.case, st.kind
    if kind == "solve":
        s, x, _ = st.sys[0]
        x.set(0.0)
        s.solve()
        return st.out[0]
    if kind == "batch":
        for _, x, _ in st.sys:
            x.set(0.0)
        X.solve_batch([s for s, _, _ in st.sys], [x for _, x, _ in st.sys],
                      [b for _, _, b in st.sys])
        return st.out
    if kind == "spmv":
        if case["mode"] == 1:  # y += A x starts from the same y in every pass
            with torch.cuda.stream(st.ext):
                st.y.copy_(st.y0)
        X.call("XAMG_b200_spmv", st.csr, st.x.data_ptr(), st.y.data_ptr(), case["nv"],
               case["mode"], st.stream)
        return st.y
    if kind == "dot":
        X.call("XAMG_b200_dot", case["n"], case["nv"], st.x.data_ptr(), st.y.data_ptr(),
               st.o.ctypes.data, st.stream)
        return st.o.copy()
    if kind == "gemm":
        X.call("XAMG_b200_gemm_bf16", case["m"], case["n"], case["k"], st.A.data_ptr(),
               st.B.data_ptr(), st.C.data_ptr(), case["n"], case["mode"], st.bias.data_ptr(),
               None, 0, st.stream)
        return st.C
    if kind == "mlp_predict":
        st.mlp.predict(st.F[0].data_ptr(), st.Y.data_ptr(), case["batch"])
        return st.Y
    losses = [st.mlp.train_step(st.F[i % 4].data_ptr(), st.T[i % 4].data_ptr(), case["batch"],
                                LEARNING_RATE) for i in range(case["steps"])]
    return {"losses": losses, "params": st.mlp.params()}


# a trained guess refreshed for a changed problem: a tenth of the rate it was trained with
LEARNING_RATE = 1e-4


# ------------------------------------------------------------------------------ work
def _solve_work(key, nv, form, precond, order, sweeps):
    """Bytes of a solve of a nominal number of iterations: per iteration two Krylov products with
    their vectors, and with multigrid two V-cycles of smoother, residual and transfer products
    over the hierarchy (values and columns once a product, vectors once)."""
    n, st = key[1] * key[2] * key[3], key[0] or 7
    nnz = n * PER_ROW[st]
    krylov = 2 * (12 * nnz + 16 * n * nv) + 17 * 8 * n * nv
    if precond == "Jacobi":
        return {"bytes": 40 * krylov, "flops": 40 * 2 * (2 * nnz * nv + 9 * n * nv)}
    entry = {"fp64": 12, "f32": 6, "bf16": 4}[form]
    vec = 8 if form == "fp64" else 4
    products = 2 * sweeps * (order if precond == "Chebyshev" else 1) + 1
    cyc = products * COMPLEXITY[st] * (entry * nnz + 3 * vec * n * nv)
    it = 7
    return {"bytes": it * (krylov + 2 * cyc),
            "flops": it * 2 * (2 * nnz * nv * (1 + products * COMPLEXITY[st]) + 9 * n * nv)}


def work(case):
    kind = case["kind"]
    if kind in ("solve", "batch"):
        ws = [_solve_work(key, nv, case.get("form", "f32"), case.get("precond", "HSGS"),
                          case.get("order", 0), case.get("sweeps", 1))
              for key, nv in _systems(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if kind == "spmv":
        n = case["nx"] * case["ny"] * case["nz"]
        nnz = n * {"box27": 26.4, "star7": 6.9, "ragged": 43.0}[case["pattern"]]
        e = 8 if case["dtype"] == "f64" else 4
        vecs = (2 if case["mode"] == 0 else 5) * n * case["nv"] * e
        return {"bytes": nnz * (e + case["col_bytes"]) + 4 * (n + 1) + vecs,
                "flops": 2 * nnz * case["nv"]}
    if kind == "dot":
        return {"bytes": 16 * case["n"] * case["nv"], "flops": 2 * case["n"] * case["nv"]}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k) + m * n * (4 if case["mode"] == 0 else 2) + 4 * n,
                "flops": 2 * m * n * k}
    w, h, b = case["width"], case["hidden"], case["batch"]
    weights = 2 * w * h + h * h
    if kind == "mlp_predict":
        return {"bytes": 2 * weights + 8 * b * w, "flops": 2 * b * weights}
    # weights read in BF16 by the three products of a layer; parameter, gradient and the two Adam
    # moments in FP32, and the BF16 weights written back
    step = {"bytes": weights * (6 + 4 + 28 + 2) + 8 * b * w, "flops": 6 * b * weights}
    return {k: case["steps"] * v for k, v in step.items()}


def tolerance(case):
    kind = case["kind"]
    if kind in ("solve", "batch"):
        # two solves that both end below a relative residual of 1e-8
        return {"rel": 1e-6}
    if kind == "spmv":
        return {"rel": 1e-14} if case["dtype"] == "f64" else {"rel": 2e-6}
    if kind == "dot":
        return {"rel": 1e-11}
    if kind == "gemm":
        return {"rel": 1e-5} if case["mode"] == 0 else {"rel": 4e-3}
    if kind == "mlp_predict":
        return {"rel": 4e-3}
    # Adam divides small gradients by their own size: the same path with its sums in another order
    # moved the weights by 8e-4 of their norm, single ones by 0.03 of their root mean square
    return {"rel": 3.5e-3, "max": 0.13}


# ------------------------------------------------------------------------------ in 64 bits
def _cg(A, dinv, b):
    """Jacobi-preconditioned conjugate gradients in FP64 to 1e-13, column by column at once."""
    x = torch.zeros_like(b)
    r = b.clone()
    z = r * dinv
    p = z.clone()
    rz = (r * z).sum(0)
    bn = b.norm(dim=0)
    for it in range(20000):
        q = A @ p
        a = rz / (p * q).sum(0).clamp_min(1e-300)
        x += a * p
        r -= a * q
        if it % 20 == 19 and bool((r.norm(dim=0) <= 1e-13 * bn).all()):
            break
        z = r * dinv
        rz2 = (r * z).sum(0)
        p = z + (rz2 / rz.clamp_min(1e-300)) * p
        rz = rz2
    return x


def _exact_solve(key, nv, seed):
    row, col, val = _host_matrix(*key)
    n = len(row) - 1
    row = torch.from_numpy(row.astype(np.int64)).cuda()
    col = torch.from_numpy(col.astype(np.int64)).cuda()
    val = torch.from_numpy(val).cuda()
    r = torch.repeat_interleave(torch.arange(n, device="cuda"), row[1:] - row[:-1])
    diag = torch.zeros(n, dtype=torch.float64, device="cuda")
    on = r == col
    diag[r[on]] = val[on]
    A = torch.sparse_csr_tensor(row, col, val, (n, n))
    return _cg(A, (1 / diag)[:, None], _rhs(n, nv, seed))


def _mlp_forward(P, F):
    z1 = F @ P[0].T + P[1]
    h1 = z1.clamp_min(0)
    z2 = h1 @ P[2].T + P[3]
    h2 = z2.clamp_min(0)
    return h1, h2, h2 @ P[4].T + P[5]


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return _exact_solve(*_systems(case)[0], seed)
    if kind == "batch":
        return [_exact_solve(key, nv, seed + 7919 * i)
                for i, (key, nv) in enumerate(_systems(case))]
    if kind == "spmv":
        row, col, val, x, y = _csr(case, seed)
        A = torch.sparse_csr_tensor(row, col, val.double(), (row.numel() - 1, x.shape[0]))
        p = A @ x.double()
        return p + y.double() if case["mode"] == 1 else p
    if kind == "dot":
        x, y = _rhs(case["n"], case["nv"], seed), _rhs(case["n"], case["nv"], seed + 1)
        return (x * y).sum(0).cpu().numpy()
    if kind == "gemm":
        A, B, bias = _gemm_inputs(case, seed)
        C = A.double() @ B.double().T + bias.double()
        return C.clamp_min(0) if case["mode"] == 2 else C
    parts, F, T = _mlp_inputs(case, seed)
    w, h = case["width"], case["hidden"]
    shapes = [(h, w), (h,), (h, h), (h,), (w, h), (w,)]
    P = [p.double().reshape(s) for p, s in zip(parts, shapes)]
    F, T = [f.double() for f in F], [t.double() for t in T]
    if kind == "mlp_predict":
        return _mlp_forward(P, F[0])[2]
    m, v = [torch.zeros_like(p) for p in P], [torch.zeros_like(p) for p in P]
    losses = []
    for i in range(case["steps"]):
        f, t = F[i % 4], T[i % 4]
        h1, h2, y = _mlp_forward(P, f)
        losses.append(float(((y - t) ** 2).mean()))
        dy = 2 * (y - t) / y.numel()
        d2 = (dy @ P[4]) * (h2 > 0)
        d1 = (d2 @ P[2]) * (h1 > 0)
        grads = [d1.T @ f, d1.sum(0), d2.T @ h1, d2.sum(0), dy.T @ h2, dy.sum(0)]
        for p, a, b, g in zip(P, m, v, grads):
            a.mul_(0.9).add_(g, alpha=0.1)
            b.mul_(0.999).add_(g * g, alpha=0.001)
            c1, c2 = 1 - 0.9 ** (i + 1), 1 - 0.999 ** (i + 1)
            p.sub_(LEARNING_RATE * (a / c1) / ((b / c2).sqrt() + 1e-8))
    return {"losses": losses, "params": torch.cat([p.reshape(-1) for p in P])}
