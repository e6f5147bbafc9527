"""Single-vector FP32 products: how a row's terms are added. One box of N points is a dense row of N stored
entries, cut into column parts of 4096; x is made so that row 0's terms are 1 in the first 128 columns of a
part and 3e-7 in the others, which a running FP32 sum of a thread's eight ones no longer takes up.

Bound: a thread sums at most 16 terms, then 4096 / 16 / 16 such sums at most, then a row's partial sums
over at most 16 threads in sequence, three parts and the roundings of entry and source:
(16 + 16 + 16 + 5) 2^-24 = 3.2e-6 of the sum (all terms are positive). A single sum a thread loses 3e-7 * 248 / 8
= 9e-6."""
import numpy as np
import pytest

from h2weak_gb300 import synth


@pytest.mark.gpu
def test_fp32_rows_take_up_small_terms(gpu):
    hw = gpu
    N = 11500  # 1.3e8 entries: targets of 32 rows
    op = hw.H2Operator(2, 0, 1, 8, 1, kernel_n=N, diag_n=N)
    op.set_points(0.5 * (synth.uniform_points(synth.config_seed(80, N), N, 2) - 1.0))
    op.build_tree()
    op.assemble()
    e = np.zeros(N)
    e[0] = 1.0
    a = op.matvec(e)  # row 0 too, by symmetry
    s = np.where(np.arange(N) % 4096 < 128, 1.0, 3e-7)
    y = op.matvec(s / a, precision=hw.PREC_FP32)[0]
    assert abs(op.matvec(s / a)[0] - s.sum()) <= 1e-12 * s.sum()
    assert abs(y - s.sum()) <= 53 * 2.0 ** -24 * s.sum(), abs(y - s.sum()) / s.sum()


@pytest.mark.gpu
def test_fp32_rows_with_infinities(gpu):
    """The roundings that a row's sum keeps apart do not turn an infinity into a NaN."""
    hw = gpu
    op = hw.H2Operator(2, 0, 0, 10, 3)
    op.gen_grid(41)
    op.build_tree()
    op.assemble()
    x = synth.normal(synth.config_seed(81, 0), op.N)
    x[7] = 1e39  # infinite in FP32
    y = op.matvec(x, precision=hw.PREC_FP32)
    op.set_option(hw.OPT_COOP, 0)
    r = op.matvec(x, precision=hw.PREC_FP32)
    assert np.array_equal(np.isinf(y), np.isinf(r)) and np.isinf(y).any()
    assert np.array_equal(np.isnan(y), np.isnan(r))
