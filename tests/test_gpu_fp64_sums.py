"""Rounding of single-vector FP64 products: no more of it than in the launch by phases, which adds a row's terms in the
former order (neighbouring columns together). Both are compared with the products of 64 vectors at once, whose
digit sums round a row once for 256 columns.

The quadratic mean over 64 vectors of two sums of the same number of roundings varies by some 10 %, and both differences
hold the rounding of the 64-vector products: 1.2. A thread's terms taken from every CG-th column gave 2.0, 1.4 and
1.2 on these operators."""
import numpy as np
import pytest

from h2weak_gb300 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 0, 0, 12, 9, 32768), (2, 0, 1, 8, 4, -9973), (1, 0, 1, 12, 8, 16384), (2, 0, 0, 10, 4, 128),
                                   (3, 0, 1, 8, 2, -9001)])
def test_fp64_rounding_no_larger_than_by_phases(gpu, shape):
    import torch
    hw = gpu
    dim, form, kern, tol, nlev, n = shape
    N = n ** dim if n > 0 else -n
    op = hw.H2Operator(dim, form, kern, tol, nlev, kernel_n=N, diag_n=2 * N if dim == 1 else N)
    if n > 0:
        op.gen_grid(n)
    else:
        op.set_points(synth.uniform_points(synth.config_seed(83, N), N, dim))
    op.build_tree()
    op.assemble()
    x = torch.from_numpy(np.stack([synth.normal(synth.config_seed(84, c), N) for c in range(64)])).cuda()
    many, one, phases = (torch.empty_like(x) for _ in range(3))
    torch.cuda.synchronize()
    op.matvec_device(x.data_ptr(), many.data_ptr(), 64)
    assert op.get_option(hw.OPT_COPIES_MADE) & 2  # in digits
    for c in range(64):
        op.matvec_device(x[c].data_ptr(), one[c].data_ptr())
    torch.cuda.synchronize()
    op.set_option(hw.OPT_COOP, 0)
    for c in range(64):
        op.matvec_device(x[c].data_ptr(), phases[c].data_ptr())
    torch.cuda.synchronize()

    def off(y):
        return float((((y - many).norm(dim=1) / many.norm(dim=1)) ** 2).mean()) ** 0.5

    assert off(one) <= 1.2 * off(phases), (off(one), off(phases))
