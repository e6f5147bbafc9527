"""FP64 products of many vectors on the tensor cores (mo.cu) against the same products
on the FP64 pipe, one launch per phase: rows that are no multiple of 8 or 64, one
chunk of 32 columns and block rows wider than one target, each width of the vector
groups and its neighbours, column scales far apart, zero and non-finite columns.

Bound: a pass on the FP64 pipe rounds each of its W <= 8192 partial sums at 2^-53, in the
quadratic mean sqrt(W) 2^-53 = 1e-14 of its result, and there are at most 2 L + 3 <= 15 passes:
4e-14 of the result's norm; the splitting adds 2^-59 sqrt(W) of a row's largest product."""
import numpy as np
import pytest

from h2weak_gb300 import synth

BOUND = 5e-14
# name: dim, form, kernel, tol, levels, points (grid side or -random count)
CASES = {
    "1d_tiny": (1, 0, 1, 10, 2, 37),
    "1d_semi": (1, 1, 0, 10, 5, 1111),
    "2d_few_points": (2, 0, 1, 8, 3, -90),
    "2d_odd": (2, 0, 0, 10, 3, 41),
    "2d_plain": (2, 2, 1, 8, 3, -1501),
    "3d_wide": (3, 0, 0, 7, 2, -5003),
    "3d_semi_wide": (3, 1, 1, 7, 2, -4001),
    "3d_one_level_down": (3, 0, 0, 7, 3, 13),
    "2d_three_boxes": (2, 0, 1, 8, 3, -271),
}


def make(hw, case):
    dim, form, kern, tol, nlev, n = CASES[case]
    N = n ** dim if n > 0 else -n
    op = hw.H2Operator(dim, form, kern, tol, nlev, kernel_n=N, diag_n=2 * N if dim == 1 else N)
    if n > 0:
        op.gen_grid(n)
    else:
        p = synth.uniform_points(synth.config_seed(63, N), N, dim)
        if case == "2d_three_boxes":  # all points in a row of three leaf boxes: the middle one has no far field
            p = np.ascontiguousarray((p + 1.0) * [0.375, 0.125] - 1.0)
        op.set_points(p)
    op.build_tree()
    op.assemble()
    return op


def columns(op, m):
    return np.stack([synth.normal(synth.config_seed(64, c), op.N) for c in range(m)])


def product(hw, op, X, flow=1, prec=None):
    import torch
    op.set_option(hw.OPT_DATAFLOW, flow)
    x = torch.from_numpy(X).cuda()
    y = torch.full_like(x, 7.0)
    torch.cuda.synchronize()
    op.matvec_device(x.data_ptr(), y.data_ptr(), X.shape[0], hw.PREC_FP64 if prec is None else prec)
    torch.cuda.synchronize()
    op.set_option(hw.OPT_DATAFLOW, 1)
    return y.cpu().numpy()


def off(y, r):
    return (np.linalg.norm(y - r, axis=1) / np.maximum(np.linalg.norm(r, axis=1), 1e-300)).max()


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(CASES))
def test_tensor_core_fp64_product(gpu, case):
    hw = gpu
    op = make(hw, case)
    for m in (2, 16, 17, 33, 64, 70):
        X = columns(op, m)
        y = product(hw, op, X)
        assert np.array_equal(y, product(hw, op, X)), m  # no atomics on results: the same on every run
        r = product(hw, op, X, flow=0)
        assert off(y, r) <= BOUND, (m, off(y, r))
        y = product(hw, op, X, prec=hw.PREC_DF64)
        assert off(y, r) <= BOUND, (m, off(y, r))


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["2d_odd", "3d_semi_wide"])
def test_tensor_core_fp64_product_column_scales(gpu, case):
    """Columns keep scales of their own: powers of two change nothing but the exponent, a zero
    column stays zero, a column with an infinity or a NaN leaves its neighbours alone."""
    hw = gpu
    op = make(hw, case)
    X = columns(op, 19)
    y = product(hw, op, X)
    e = np.ldexp(1.0, 40 * (np.arange(19) - 9))
    assert np.array_equal(product(hw, op, X * e[:, None]), y * e[:, None])
    Z = X.copy()
    Z[3] = 0.0
    Z[5, op.N // 2] = np.inf
    Z[18, 0] = np.nan
    z = product(hw, op, Z)
    r = product(hw, op, Z, flow=0)
    keep = [c for c in range(19) if c not in (3, 5, 18)]
    assert np.array_equal(z[keep], y[keep])
    assert not z[3].any()
    for c in (5, 18):  # no row is finite that the multiply-adds leave non-finite
        assert not np.isfinite(z[c][~np.isfinite(r[c])]).any()
    W = X * 10.0 ** (12.0 * np.stack([synth.uniform01(synth.config_seed(65, c), op.N) for c in range(19)]) - 6.0)
    r = product(hw, op, W, flow=0)
    assert off(product(hw, op, W), r) <= BOUND
