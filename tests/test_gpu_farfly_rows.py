"""The far field formed during the product, at the edges of its work items: boxes of one to four,
up to eight, sixteen, thirty-two and more skeleton rows (threads to a row change there), tables of
few and of many exponents (deep trees of few points), each kernel; single and pair precision
against FP64 entries of the same points.

Bounds: an FP32 entry and its product round at 2^-24 a few times, a pair at 2^-46; the sums of an
operator cancel by less than a hundred: 1e-4 and 2e-12 of the result's norm."""
import numpy as np
import pytest

from h2weak_gb300 import synth

# dim, kernel, tolerance, levels, points
CASES = [(3, 1, 1, 2, 901), (3, 1, 3, 2, 2003), (3, 1, 5, 3, 4001), (3, 1, 9, 2, 3001), (2, 0, 2, 3, 700), (2, 0, 4, 8, 1501),
         (2, 0, 11, 4, 3001), (3, 0, 4, 2, 1201), (2, 1, 3, 3, 801)]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_far_field_work_items(gpu, case):
    hw = gpu
    dim, kern, tol, nlev, N = case
    op = hw.H2Operator(dim, 0, kern, tol, nlev, kernel_n=N, diag_n=N)
    op.set_option(hw.OPT_FAR_ON_THE_FLY, 1)
    op.set_points(synth.uniform_points(synth.config_seed(71, N), N, dim))
    op.build_tree()
    op.assemble()
    for k in range(2):
        x = synth.normal(synth.config_seed(72, k), N)
        r = op.matvec(x, precision=hw.PREC_FP64)
        for prec, bound in ((hw.PREC_FP32, 1e-4), (hw.PREC_DF64, 2e-12)):
            y = op.matvec(x, precision=prec)
            assert np.linalg.norm(y - r) <= bound * np.linalg.norm(r), (prec, np.linalg.norm(y - r) / np.linalg.norm(r))
