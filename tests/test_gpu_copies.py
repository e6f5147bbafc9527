"""Products without the operator's copies (no room, or H2W_OPT_COPIES 0): FP64 on the packed operator's dataflow
launch, several vectors on the FP64 and FP32 pipes, batches by phases; and operators that share a memory budget.

Bound: both forms sum the same products in another order, as in test_gpu_single.py: 1e-13 of a result's norm; a
double-FP32 term is off by about 2^-44, in the quadratic mean far less: 1e-12."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from h2weak_gb300 import synth

# dim, form, kernel, tol, levels, points (grid side or -random count)
SHAPES = [(1, 0, 1, 10, 6, 3000), (1, 1, 1, 8, 7, 20001), (2, 0, 0, 10, 4, 64), (2, 1, 1, 8, 3, -1501), (3, 0, 1, 7, 2, -5003),
          (3, 0, 2, 7, 2, -1203)]


def make(hw, dim, form, kern, tol, nlev, n, copies=1):
    N = n ** dim if n > 0 else -n
    op = hw.H2Operator(dim, form, kern, tol, nlev, kernel_n=N, diag_n=2 * N if dim == 1 else N)
    op.set_option(hw.OPT_COPIES, copies)
    if n > 0:
        op.gen_grid(n)
    else:
        op.set_points(synth.uniform_points(synth.config_seed(75, N), N, dim))
    op.build_tree()
    op.assemble()
    return op


def off(y, r):
    return np.linalg.norm(y - r) / np.linalg.norm(r)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
def test_products_without_copies(gpu, shape):
    hw = gpu
    op = make(hw, *shape)
    assert op.get_option(hw.OPT_COPIES_MADE) == 1
    x = np.stack([synth.normal(synth.config_seed(76, c), op.N) for c in range(6)])
    if op.complex:
        x = x[:3] + 1j * x[3:]
    r = op.matvec(x[0])
    m = None if op.complex else op.matvec(x.T)
    sol = op.gmres(r, max_iter=60, tol_pow=8)
    op.set_option(hw.OPT_COPIES, 0)
    assert op.get_option(hw.OPT_COPIES_MADE) == 0
    for again in range(2):
        assert off(op.matvec(x[0]), r) <= 1e-13
    got = op.gmres(r, max_iter=60, tol_pow=8)  # the captured step takes the other form
    assert abs(got[1] - sol[1]) <= 1 and off(got[0], sol[0]) <= 1e-6
    if m is not None:
        assert off(op.matvec(x.T), m) <= 1e-13
        assert off(op.matvec(x.T, precision=hw.PREC_DF64), m) <= 1e-12
    assert op.get_option(hw.OPT_COPIES_MADE) == 0
    op.set_option(hw.OPT_COPIES, 1)
    assert np.array_equal(op.matvec(x[0]), r)


@pytest.mark.gpu
def test_first_product_under_capture_without_copies(gpu):
    """A caller's stream capture takes no allocation: the product captured first on an operator without
    copies is right, and so are later ones."""
    import torch
    hw = gpu
    op = make(hw, 2, 0, 0, 10, 3, 41, copies=0)
    x = torch.from_numpy(synth.normal(synth.config_seed(77, 1), op.N)).cuda()
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    g, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        op.matvec_device(x.data_ptr(), y.data_ptr(), 1, hw.PREC_FP64, st.cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    first = y.cpu().numpy()
    r = op.matvec(x.cpu().numpy())
    assert off(first, r) <= 1e-13


@pytest.mark.gpu
def test_captured_copies_stay(gpu):
    """A product in a caller's graph keeps reading the copy it was captured with."""
    import torch
    hw = gpu
    op = make(hw, 2, 0, 0, 10, 3, 41)
    x = torch.from_numpy(synth.normal(synth.config_seed(78, 1), op.N)).cuda()
    y = torch.zeros_like(x)
    r = op.matvec(x.cpu().numpy())
    torch.cuda.synchronize()
    g, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        op.matvec_device(x.data_ptr(), y.data_ptr(), 1, hw.PREC_FP64, st.cuda_stream)
    op.set_option(hw.OPT_COPIES, 0)
    assert op.get_option(hw.OPT_COPIES_MADE) & 1
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), r)


@pytest.mark.gpu
def test_batch_without_copies(gpu):
    hw = gpu
    shapes = [(2, 0, 0, 10, 4, 64), (2, 0, 1, 8, 3, -901), (2, 1, 1, 8, 3, -1501)]
    ops = [make(hw, *s) for s in shapes]
    b = hw.Batch(ops)
    x = synth.normal(synth.config_seed(79, 0), b.N)
    r = b.matvec(x)
    sol = b.gmres(r, tol_pow=8)
    for o in ops:
        o.set_option(hw.OPT_COPIES, 0)
    b2 = hw.Batch(ops)
    assert off(b2.matvec(x), r) <= 1e-13
    got = b2.gmres(r, tol_pow=8)
    assert np.abs(np.asarray(got[1]) - np.asarray(sol[1])).max() <= 1 and off(got[0], sol[0]) <= 1e-6
    assert off(b2.matvec(x, precision=hw.PREC_FP32), r) <= 1e-4


@pytest.mark.gpu
def test_copies_are_given_back(gpu, tmp_path):
    from h2weak_gb300 import buildlib
    lib = buildlib.build()
    exe = str(tmp_path / "memory_budget")
    r = subprocess.run([buildlib.nvcc(), "-std=c++17", "--cudart", "shared", "-I", os.path.join(ROOT, "include"),
                        os.path.join(ROOT, "tests", "memory_budget.cpp"), lib, "-o", exe, "-ldl",
                        "-Xlinker", "--export-dynamic", "-Xlinker", "-rpath=" + os.path.dirname(lib)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=200)
    assert r.returncode == 0, r.stdout + r.stderr
