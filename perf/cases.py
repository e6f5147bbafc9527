"""The calls whose time counts: what a program that uses this package has it do.

Each case is one call (or one short run of calls) through the public Python
entry points, on operators whose dimension, form, kernel, size and tolerances
come from the reference drivers' settings, the tests and bench.py, or lie
between them. `listed()` names twelve of them; `draw()` gives more of the same
kinds over the whole ranges. Nothing here checks a result.

Kinds of call ("call"):
  product   y = A x for one or several columns, device vectors, one precision
  gmres     FP64 GMRES of one right-hand side, host vectors (the reference's use)
  gmres_ir  mixed-precision solve of one right-hand side, host vectors
  columns   FP64 GMRES of several right-hand sides at once, device vectors
  columns_ir  the mixed-precision form of the same
  many_ir   mixed-precision solves of many independent problems in one batch
  driver    the reference's main(): tree and assembly, dense right-hand side,
            one product, one solve; host vectors

Products asked for in FP32 are kept by the caller as float32: a program that
asks for single precision goes on in it.
"""
import math

import numpy as np
import torch

import h2weak_gb300 as hw

FORMS = {"nested": hw.FORM_NESTED, "semi": hw.FORM_SEMINESTED, "plain": hw.FORM_NONNESTED}
KERNELS = {"ie": hw.KERNEL_IE, "rbf": hw.KERNEL_RBF, "helmholtz": hw.KERNEL_HELMHOLTZ}
PRECISIONS = {"fp64": hw.PREC_FP64, "fp32": hw.PREC_FP32, "df64": hw.PREC_DF64}


def _case(call, dim, form, kernel, points, n, leaf, tol, **more):
    """n: grid points per axis, or the number of random points; leaf: points per leaf box at most, on average."""
    return dict({"call": call, "dim": dim, "form": form, "kernel": kernel, "points": points, "n": n, "leaf": leaf,
                 "tol": tol}, **more)


def listed():
    c = [
        # the smallest call: one product of a short 1D problem, launches and dependent passes only
        dict(_case("product", 1, "nested", "rbf", "grid", 4096, 64, 12, precision="fp64", cols=1), name="1d_product_fp64"),
        # the ordinary product that an outer iteration of the caller's own drives
        dict(_case("product", 2, "nested", "ie", "grid", 256, 64, 10, precision="fp64", cols=1), name="2d_product_fp64"),
        # random points, odd size, the larger semi-nested operator, single precision: memory traffic
        dict(_case("product", 3, "semi", "rbf", "random", 20011, 128, 8, precision="fp32", cols=1), name="3d_product_fp32"),
        # a full block of right-hand sides in single precision (the inner products of a block solve)
        dict(_case("product", 2, "nested", "ie", "grid", 256, 64, 10, precision="fp32", cols=64), name="2d_product_fp32_64"),
        # an odd number of columns at refinement accuracy
        dict(_case("product", 3, "nested", "ie", "grid", 24, 512, 8, precision="df64", cols=37), name="3d_product_df64_37"),
        # the reference's solve, as its 1D driver runs it
        dict(_case("gmres", 1, "nested", "rbf", "grid", 32768, 64, 12, gmres_tol=10), name="1d_gmres"),
        # complex kernel, random points: complex products and the complex solve
        dict(_case("gmres", 3, "nested", "helmholtz", "random", 4001, 128, 8, gmres_tol=10), name="3d_helmholtz_gmres"),
        # a 3D problem whose far field is formed during each product; single-precision inner products,
        # FP64-accurate residuals: the family of the default benchmark, the largest case here
        dict(_case("gmres_ir", 3, "nested", "rbf", "random", 65536, 128, 10, fly=True, residual="df64", gmres_tol=10),
             name="3d_fly_gmres_ir"),
        # several right-hand sides in FP64 throughout
        dict(_case("columns", 2, "nested", "rbf", "random", 9973, 64, 8, cols=19, gmres_tol=10), name="2d_columns_gmres_19"),
        # 64 right-hand sides, mixed precision: the 2D benchmark's step
        dict(_case("columns_ir", 2, "nested", "ie", "grid", 256, 64, 10, cols=64, residual="df64", gmres_tol=10),
             name="2d_columns_ir_64"),
        # many independent problems of different sizes and kernels in one batch
        dict(_case("many_ir", 2, "nested", "mixed", "random", 12000, 64, 8, problems=24, gmres_tol=10), name="2d_many_ir_24"),
        # a whole run of the reference's main() on new points
        dict(_case("driver", 2, "nested", "rbf", "random", 9973, 64, 8, gmres_tol=10), name="2d_driver"),
    ]
    return c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _real_problem(rng, call, most, **more):
    """A problem with a real kernel in 1D, 2D or 3D; most: largest N by dimension."""
    dim = rng.choice([d for d in (1, 2, 3) if d in most])
    form = rng.choice(["nested", "nested", "semi"] if dim == 1 else ["nested", "nested", "semi", "plain"])
    points = rng.choice(["grid", "random"])
    N = _log_int(rng, {1: 1024, 2: 1000, 3: 2000}[dim], most[dim])
    n = N if points == "random" or dim == 1 else max(8, int(round(N ** (1.0 / dim))))
    leaf = {1: rng.choice([32, 64, 100]), 2: rng.choice([49, 64, 100]), 3: rng.choice([128, 216, 512])}[dim]
    tol = {1: rng.choice([8, 10, 12]), 2: rng.choice([8, 10]), 3: rng.choice([7, 8])}[dim]
    return _case(call, dim, form, rng.choice(["ie", "rbf"]), points, n, leaf, tol, **more)


def draw(rng):
    call = rng.choice(["product", "product", "product", "gmres", "gmres_ir", "columns", "columns_ir", "many_ir", "driver",
                       "helmholtz", "fly"])
    if call == "product":
        if rng.random() < 0.5:
            return _real_problem(rng, call, {1: 65536, 2: 65536, 3: 24000}, precision=rng.choice(["fp64", "fp32"]), cols=1)
        return _real_problem(rng, call, {1: 65536, 2: 65536, 3: 13824}, precision=rng.choice(["fp64", "fp32", "df64"]),
                             cols=rng.randint(2, 64))
    if call == "gmres":
        return _real_problem(rng, call, {1: 65536, 2: 40000, 3: 8000}, gmres_tol=10)
    if call == "gmres_ir":
        return _real_problem(rng, call, {1: 65536, 2: 65536, 3: 13824}, gmres_tol=10)
    if call == "columns":
        return _real_problem(rng, call, {1: 16384, 2: 12000}, cols=rng.randint(2, 24), gmres_tol=10)
    if call == "columns_ir":
        return _real_problem(rng, call, {1: 65536, 2: 65536, 3: 6000}, cols=rng.randint(2, 64), residual="df64", gmres_tol=10)
    if call == "many_ir":
        return _case(call, 2, "nested", "mixed", "random", _log_int(rng, 3000, 14000), 64, 8, problems=rng.randint(6, 30),
                     gmres_tol=10)
    if call == "driver":
        return _case(call, 2, "nested", rng.choice(["ie", "rbf"]), "random", _log_int(rng, 1500, 10000), 64, 8, gmres_tol=10)
    if call == "helmholtz":
        return _case("gmres", 3, rng.choice(["nested", "semi"]), "helmholtz", "random", _log_int(rng, 1500, 5000), 128, 8,
                     gmres_tol=10)
    return _case("gmres_ir", 3, "nested", "rbf", "random", _log_int(rng, 12000, 60000), 128, 10, fly=True, residual="df64",
                 gmres_tol=10)


# ------------------------------------------------------------------ inputs ---
def _levels(dim, N, leaf):
    return max(2, int(math.ceil(math.log(float(N) / leaf) / math.log(2 ** dim))))


def _size(case):
    return case["n"] ** case["dim"] if case["points"] == "grid" else case["n"]


def _points(dim, n, seed, grid):
    """The drivers' uniform grid, or n seeded uniform points of [-1, 1)^dim."""
    if grid:
        return None
    return np.random.default_rng(seed).uniform(-1.0, 1.0, size=(n, dim))


def _many(case, seed):
    """Sizes, kernels and points of a batch's problems: sizes over a factor of 16 up to n, as a mesh hierarchy's parts."""
    rng = np.random.default_rng(seed + 1)
    out = []
    for p in range(case["problems"]):
        # the sizes are the case's, the points the seed's
        n = int(round(case["n"] * 16.0 ** (-((p * 7) % case["problems"]) / float(case["problems"]))))
        out.append((n, ["ie", "rbf"][p % 2], rng.uniform(-1.0, 1.0, size=(n, 2))))
    return out


def _operator(dim, form, kernel, leaf, tol, N, points, grid, fly=False):
    op = hw.H2Operator(dim, FORMS[form], KERNELS[kernel], tol, _levels(dim, N, leaf), 0, kernel_n=N,
                       diag_n=2 * N if dim == 1 else N)
    if fly:
        op.set_option(hw.OPT_FAR_ON_THE_FLY, 1)
    if points is None:
        op.gen_grid(grid)
    else:
        op.set_points(points)
    op.build_tree()
    op.assemble()
    return op


def _operator_of(case, seed):
    pts = _points(case["dim"], case["n"], seed, case["points"] == "grid")
    return _operator(case["dim"], case["form"], case["kernel"], case["leaf"], case["tol"], _size(case), pts, case["n"],
                     case.get("fly", False))


def _solution(case, seed, N):
    """The vector (or block of columns, one to a row) that products take and solves look for: N(0, 1)."""
    g = np.random.default_rng(seed + 2)
    if case["call"] == "many_ir":
        return g.standard_normal(N)
    if case["kernel"] == "helmholtz":
        return g.standard_normal(N) + 1j * g.standard_normal(N)
    cols = case.get("cols", 1)
    return g.standard_normal((cols, N)) if cols > 1 or case["call"] in ("product", "columns", "columns_ir") else \
        g.standard_normal(N)


def prepare(case, seed):
    call = case["call"]
    s = {"case": case}
    if call == "driver":  # new points and a vector; everything else is the pass
        s["points"] = _points(case["dim"], case["n"], seed, False)
        s["x"] = _solution(case, seed, case["n"])
        return s
    if call == "many_ir":
        ops = [_operator(2, case["form"], k, case["leaf"], case["tol"], n, pts, None) for n, k, pts in _many(case, seed)]
        s["op"] = hw.Batch(ops)
        s["x_true"] = _solution(case, seed, s["op"].N)
        s["b"] = s["op"].matvec(s["x_true"])
        return s
    op = s["op"] = _operator_of(case, seed)
    if case.get("residual") == "df64":
        op.set_option(hw.OPT_IR_RESIDUAL, hw.PREC_DF64)
    x = _solution(case, seed, op.N)
    if call in ("gmres", "gmres_ir"):
        s["b"] = op.matvec(x)
        return s
    s["stream"] = torch.cuda.Stream()
    xd = torch.from_numpy(x).cuda()
    y = torch.empty_like(xd)
    if call == "product":
        s["x"], s["y"] = xd, y
        s["y32"] = torch.empty(y.shape, dtype=torch.float32, device="cuda") if case["precision"] == "fp32" else None
    else:
        torch.cuda.synchronize()
        op.matvec_device(xd.data_ptr(), y.data_ptr(), case["cols"])
        s["b"], s["x"] = y, torch.empty_like(xd)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    call = case["call"]
    if call == "product":
        op, st = s["op"], s["stream"]
        op.matvec_device(s["x"].data_ptr(), s["y"].data_ptr(), case["cols"], PRECISIONS[case["precision"]], st.cuda_stream)
        if s["y32"] is None:
            return s["y"]
        with torch.cuda.stream(st):
            s["y32"].copy_(s["y"])
        return s["y32"]
    if call == "gmres":
        x, it, _ = s["op"].gmres(s["b"], tol_pow=case["gmres_tol"])
        return {"x": x, "iterations": it}
    if call == "gmres_ir":
        return s["op"].gmres_ir(s["b"], tol_pow=case["gmres_tol"])[0]
    if call in ("columns", "columns_ir"):
        s["x"].fill_(1.0)  # the start the reference's drivers use
        torch.cuda.current_stream().synchronize()  # the solver runs on the handle's own stream
        f = s["op"].gmres_batch_device if call == "columns" else s["op"].gmres_ir_batch_device
        f(s["b"].data_ptr(), s["x"].data_ptr(), case["cols"], tol_pow=case["gmres_tol"])
        return s["x"]
    if call == "many_ir":
        return s["op"].gmres_ir(s["b"], tol_pow=case["gmres_tol"])[0]
    A = hw.initialisation(case["n"], _levels(case["dim"], case["n"], case["leaf"]), case["leaf"], 1, case["tol"],
                          KERNELS[case["kernel"]], dim=case["dim"], form=FORMS[case["form"]], points=s["points"])
    A.tree_initialisation()
    b = A.K.getTruePoten(s["x"])
    y = A.mat_vec_prod(s["x"])
    x = np.ones(case["n"])
    hw.iterative_solver(500, case["gmres_tol"]).GMRES(A, x, b)
    A.op.close()
    return {"b": b, "y": y, "x": x}


# -------------------------------------------------------------------- work ---
def _product_work(op, width, cols=1):
    """One product: the operator's stored entries once (as many as the reference stores) at the precision's width, the
    vectors in and out; two operations an entry and column. With the far field on the fly its entries are formed, about
    twelve operations each, and the rest read."""
    e, n = op.storage_entries(), op.N
    cplx = 2 if op.complex else 1
    if op.get_option(hw.OPT_FAR_ON_THE_FLY):
        stored = op.operator_bytes(hw.PREC_FP64) / 8.0
        return stored * width + 16.0 * n, 2.0 * stored + 12.0 * max(0.0, e - stored)
    return e * width * cplx + 16.0 * n * cols * cplx, 2.0 * e * cols * cplx * cplx


def _krylov(n, its, width):
    """Vector traffic of `its` steps: each basis vector read twice by the orthogonalisation, the new one written."""
    return width * n * sum(2 * (i + 1) + 3 for i in range(its)), 8.0 * n * sum(i + 1 for i in range(its))


def work(case):
    s = prepare(case, 1)
    call = case["call"]
    try:
        if call == "driver":
            op = _operator(case["dim"], case["form"], case["kernel"], case["leaf"], case["tol"], case["n"], s["points"], None)
            n = op.N
            x, it, _ = op.gmres(op.dense_matvec(s["x"]), tol_pow=case["gmres_tol"])
            pb, pf = _product_work(op, 8)
            kb, kf = _krylov(n, it, 8)
            e = op.storage_entries()
            op.close()
            # entries written once by the assembly, then read by it + 2 products; n^2 entries of the dense product
            return {"bytes": 8.0 * e + (it + 2) * pb + kb, "flops": (it + 2) * pf + kf + 12.0 * (n * float(n) + e)}
        op = s["op"]
        if call == "product":
            b, f = _product_work(op, 4 if case["precision"] == "fp32" else 8, case["cols"])
            return {"bytes": b, "flops": f}
        if call == "gmres":
            it = op.gmres(s["b"], tol_pow=case["gmres_tol"])[1]
            b, f = _product_work(op, 8)
            kb, kf = _krylov(op.N * (2 if op.complex else 1), it, 8)
            return {"bytes": (it + 1) * b + kb, "flops": (it + 1) * f + kf}
        if call == "gmres_ir":
            _, outer, inner, _ = op.gmres_ir(s["b"], tol_pow=case["gmres_tol"])
            b4, f4 = _product_work(op, 4)
            b8, f8 = _product_work(op, 8)
            kb, kf = _krylov(op.N, inner // outer, 8)
            return {"bytes": (inner + 1) * b4 + b8 + outer * kb, "flops": (inner + 1) * f4 + f8 + outer * kf}
        if call == "columns":
            x = torch.ones_like(s["b"])
            torch.cuda.synchronize()
            it = int(op.gmres_batch_device(s["b"].data_ptr(), x.data_ptr(), case["cols"], tol_pow=case["gmres_tol"])[0].max())
            b, f = _product_work(op, 8, case["cols"])
            kb, kf = _krylov(op.N * case["cols"], it, 8)
            return {"bytes": (it + 1) * b + kb, "flops": (it + 1) * f + kf}
        if call == "columns_ir":
            x = torch.ones_like(s["b"])
            torch.cuda.synchronize()
            outer, inner, _ = op.gmres_ir_batch_device(s["b"].data_ptr(), x.data_ptr(), case["cols"],
                                                       tol_pow=case["gmres_tol"])
            b4, f4 = _product_work(op, 4, case["cols"])
            b8, f8 = _product_work(op, 8, case["cols"])
            kb, kf = _krylov(op.N * case["cols"], inner // outer, 4)
            return {"bytes": (inner + 1) * b4 + b8 + outer * kb, "flops": (inner + 1) * f4 + f8 + outer * kf}
        _, outer, inner, _ = op.gmres_ir(s["b"], tol_pow=case["gmres_tol"])
        each = [(_product_work(o, 4), _product_work(o, 8)) for o in op.ops]
        kb, kf = _krylov(op.N, inner // outer, 8)
        return {"bytes": sum((inner + 1) * p[0] + outer * q[0] for p, q in each) + outer * kb,
                "flops": sum((inner + 1) * p[1] + outer * q[1] for p, q in each) + outer * kf}
    finally:
        if "op" in s:
            s["op"].close()


# ------------------------------------------------------------------- exact ---
def _self_term(dim, h):
    """The drivers' integral of the kernel over the box around a point: 16-point Gauss-Legendre over [0, h/2]^dim, times 2^dim."""
    z, w = np.polynomial.legendre.leggauss(16)
    x, w = 0.25 * h * (z + 1.0), 0.25 * h * w
    if dim == 1:
        return 2.0 * float(np.sum(w * np.log(x)))
    if dim == 2:
        r2 = x[:, None] ** 2 + x[None, :] ** 2
        return 4.0 * float(np.einsum("i,j,ij", w, w, -np.log(r2) / (4.0 * math.pi)))
    r = np.sqrt(x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2)
    return 8.0 * float(np.einsum("i,j,k,ijk", w, w, w, 1.0 / (4.0 * math.pi * r)))


def _grid(dim, n):
    a = -1.0 + 2.0 * (np.arange(n) + 1.0) / (n + 1.0)
    if dim == 1:
        return a[:, None]
    # the drivers' numbering: loops over (y, x) in 2D and (y, x, z) in 3D, the last one fastest
    g = np.meshgrid(*([a] * dim), indexing="ij")
    return np.stack([g[d].reshape(-1) for d in ([1, 0] if dim == 2 else [1, 0, 2])], axis=1)


def _dense(dim, kernel, pts, X):
    """K X for columns X (N x k), 64 bits, on the GPU in blocks of rows."""
    N = pts.shape[0]
    P = torch.from_numpy(np.ascontiguousarray(pts)).cuda()
    X = torch.from_numpy(np.ascontiguousarray(X)).cuda()
    a = 1e-4
    if kernel == "ie":
        h = 1.0 / N ** (1.0 / dim)
        diag = (1.0 + _self_term(dim, h)) / h ** dim
    else:
        diag = {1: math.sqrt(2.0 * N), 2: 1.0, 3: math.sqrt(N)}[dim]
    out = torch.empty_like(X)
    step = max(1, 30_000_000 // N)
    for r0 in range(0, N, step):
        Q = P[r0:r0 + step]
        R2 = sum((Q[:, d:d + 1] - P[:, d][None, :]) ** 2 for d in range(dim))
        if kernel == "ie":
            K = {1: lambda: 0.5 * torch.log(R2), 2: lambda: -torch.log(R2) / (4.0 * math.pi),
                 3: lambda: 1.0 / (4.0 * math.pi * torch.sqrt(R2))}[dim]()
        else:
            R = torch.sqrt(R2)
            if dim < 3:
                K = torch.where(R < a, R / a, a / R)
            else:
                K = torch.where(R < a, (R * torch.log(R) - 1.0) / (a * math.log(a) - 1.0), torch.log(R) / math.log(a))
        i = torch.arange(Q.shape[0], device="cuda")
        K[i, i + r0] = diag
        out[r0:r0 + step] = K @ X
    return out


def exact(case, seed):
    call = case["call"]
    if call == "product":
        pts = _grid(case["dim"], case["n"]) if case["points"] == "grid" else _points(case["dim"], case["n"], seed, False)
        return _dense(case["dim"], case["kernel"], pts, _solution(case, seed, _size(case)).T).T.contiguous()
    if call == "driver":
        x = _solution(case, seed, case["n"])
        b = _dense(case["dim"], case["kernel"], _points(case["dim"], case["n"], seed, False), x[:, None])[:, 0]
        return {"b": b, "y": b, "x": x}
    # solves: the right-hand side was made from this vector
    if call == "many_ir":
        return _solution(case, seed, sum(n for n, _, _ in _many(case, seed)))
    x = _solution(case, seed, _size(case))
    if call == "gmres":
        return {"x": x, "iterations": None}
    return torch.from_numpy(x) if call in ("columns", "columns_ir") else x
