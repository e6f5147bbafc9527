"""FP64 products of several vectors (mo.cu) row by row: every row keeps FP64's precision in its
own terms, whatever else is in its block row and column.

Multiply-adds round a row of W terms within W 2^-53 sum |a x| of it in any order; with the few
roundings of parts and parts' sums, (W + 8) 2^-53 sum |a x| for either form. The matrix is that of the
launches by phases for unit vectors. Points that all lie in one leaf box make an operator of stored
entries alone: a unit vector's row is then an entry itself, exactly."""
import numpy as np
import pytest

from h2weak_gb300 import synth

# name: dim, form, kernel, tol, points (grid side or -random count); one level
ONE_LEVEL = {
    "1d_rbf": (1, 0, 1, 12, 900),
    "2d_ie": (2, 0, 0, 10, 30),
    "2d_ie_random": (2, 0, 0, 10, -1500),
    "3d_ie": (3, 0, 0, 8, 10),
    "3d_semi_rbf": (3, 1, 1, 8, -700),
}


ONE_BOX = {  # the same, all points in one of the boxes
    "1d_rbf_box": (1, 0, 1, 12, -901),
    "2d_ie_box": (2, 0, 0, 10, -1500),
    "2d_rbf_box": (2, 1, 1, 10, -70),
    "3d_ie_box": (3, 0, 0, 8, -1003),
    "3d_semi_rbf_box": (3, 1, 1, 8, -700),
}


def make(hw, dim, form, kern, tol, n, nlev=1, box=False):
    N = n ** dim if n > 0 else -n
    op = hw.H2Operator(dim, form, kern, tol, nlev, kernel_n=N, diag_n=2 * N if dim == 1 else N)
    if n > 0:
        op.gen_grid(n)
    else:
        p = synth.uniform_points(synth.config_seed(71, N), N, dim)
        op.set_points(0.5 * (p - 1.0) if box else p)
    op.build_tree()
    op.assemble()
    return op


def product(hw, op, X, flow=1, prec=None):
    import torch
    op.set_option(hw.OPT_DATAFLOW, flow)
    x = torch.from_numpy(np.ascontiguousarray(X)).cuda()
    y = torch.full_like(x, 7.0)
    torch.cuda.synchronize()
    op.matvec_device(x.data_ptr(), y.data_ptr(), X.shape[0], hw.PREC_FP64 if prec is None else prec)
    torch.cuda.synchronize()
    op.set_option(hw.OPT_DATAFLOW, 1)
    return y.cpu().numpy()


def columns(N):
    """Dense, locally supported, widely spread and sparse columns; an odd number of them."""
    n = [synth.normal(synth.config_seed(72, c), N) for c in range(6)]
    u = [synth.uniform01(synth.config_seed(73, c), N) for c in range(4)]
    t = np.linspace(-1.0, 1.0, N)
    two = np.zeros(N)
    two[[N // 3, N // 3 + 1, N - 1]] = 1.0, 1e-9, -1e-13
    few = np.zeros(N)
    few[5::97] = n[4][5::97]
    return np.stack([n[0], np.exp(-200.0 * t * t), np.exp(-3000.0 * t * t) * n[1], n[2] * 10.0 ** (12.0 * u[0] - 6.0),
                     n[3] * 10.0 ** (60.0 * u[1] - 30.0), two, few, np.where(t < 0.0, 1e12, 1.0) * n[5], np.full(N, 3.5)])


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(ONE_LEVEL) + sorted(ONE_BOX))
def test_fp64_columns_rows_keep_their_own_precision(gpu, case):
    hw = gpu
    box = case in ONE_BOX
    op = make(hw, *(ONE_BOX if box else ONE_LEVEL)[case], box=box)
    N = op.N
    E = np.eye(N)
    A = np.concatenate([product(hw, op, E[i:i + 64], flow=0) for i in range(0, N, 64)]).T
    if box:
        for i in (0, N // 2, N - 40):
            assert np.array_equal(product(hw, op, E[i:i + 37]), A[:, i:i + 37].T), i
    X = columns(N)
    ref = (A.astype(np.longdouble) @ X.T.astype(np.longdouble)).T
    terms = (np.abs(A) @ np.abs(X).T).T
    for prec in (hw.PREC_FP64, hw.PREC_DF64):
        err = np.abs(product(hw, op, X, prec=prec).astype(np.longdouble) - ref).astype(np.float64)
        worst = (err / (terms + 1e-290)).max(axis=1)
        assert (worst <= (N + 8) * 2.0 ** -53).all(), worst


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 0, 0, 10, 41, 3), (3, 1, 1, 7, -4001, 2)])
def test_fp64_columns_non_finite_rows(gpu, shape):
    """An infinity or a NaN reaches the rows that use it, as itself, and no others."""
    hw = gpu
    op = make(hw, *shape)
    X = np.stack([synth.normal(synth.config_seed(74, c), op.N) for c in range(19)])
    X[2, 7] = np.inf
    X[5, op.N // 2] = -np.inf
    X[18, 0] = np.nan
    X[11, 3], X[11, op.N - 2] = np.inf, -np.inf
    y, r = product(hw, op, X), product(hw, op, X, flow=0)
    assert np.array_equal(np.isfinite(y), np.isfinite(r))
    assert np.array_equal(np.isnan(y), np.isnan(r))
    assert np.array_equal(np.sign(y[np.isinf(y)]), np.sign(r[np.isinf(r)]))
    fin = [c for c in range(19) if c not in (2, 5, 11, 18)]
    assert np.linalg.norm(y[fin] - r[fin]) <= 5e-14 * np.linalg.norm(r[fin])
