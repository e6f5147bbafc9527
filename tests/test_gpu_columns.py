"""Columns into leaf-order rows and back: each column's product does not depend on where it stands
in the block, on its neighbours, or on the side its memory lies on. Points that are no
multiple of the 32 rows of a tile, blocks that fill a row of vectors and blocks that do not,
more columns than one block takes; bit for bit, as the same sums are formed."""
import numpy as np
import pytest

from h2weak_gb300 import synth

CASES = {"1d": (1, 0, 1, 10, 2, 37), "2d": (2, 0, 1, 8, 3, 41), "2d_grid": (2, 0, 0, 8, 2, 16)}


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("m", [2, 16, 31, 64, 70])
def test_columns_keep_their_places(gpu, case, m):
    import torch
    hw = gpu
    dim, form, kern, tol, nlev, n = CASES[case]
    N = n ** dim
    op = hw.H2Operator(dim, form, kern, tol, nlev, kernel_n=N, diag_n=2 * N if dim == 1 else N)
    op.gen_grid(n)
    op.build_tree()
    op.assemble()
    X = np.stack([synth.normal(synth.config_seed(70, c), N) for c in range(m)])
    # blocks of one width: a column moves within its own block of 64 only
    order = np.concatenate([c0 + np.arange(min(64, m - c0))[::-1] for c0 in range(0, m, 64)])
    for prec in (hw.PREC_FP32, hw.PREC_FP64):
        def device(Z):
            x = torch.from_numpy(np.ascontiguousarray(Z)).cuda()
            y = torch.full_like(x, 7.0)
            torch.cuda.synchronize()
            op.matvec_device(x.data_ptr(), y.data_ptr(), m, prec)
            torch.cuda.synchronize()
            return y.cpu().numpy()
        y = device(X)
        r = np.stack([op.matvec(v, precision=hw.PREC_FP64) for v in X])
        bound = 5e-5 if prec == hw.PREC_FP32 else 1e-13
        assert (np.linalg.norm(y - r, axis=1) <= bound * np.linalg.norm(r, axis=1)).all()
        assert np.array_equal(device(X[order]), y[order])
        assert np.array_equal(op.matvec(X.T, precision=prec), y.T)  # host vectors
