"""The single-vector product's dataflow launch (sv.cu) against the same products
with one launch per phase, on operators whose targets lie at the edges of the
kernel's tiles: fewer targets than CTAs, rows that are no multiple of a vector,
block rows wider than one target (column parts, one after another), leaf boxes
without far field (the explicit scatter), complex operators, caller streams.

FP64 bound: both forms sum the same products in another order. A row of W terms
is then off by at most about W * 2^-53 * sum |a x| (W <= 8192 here), 1e-12 of that
sum in the worst case and its square root in practice: 1e-13 of the result's
norm. FP32: 2^-24 in place of 2^-53, 5e-5."""
import numpy as np
import pytest

from h2weak_gb300 import synth

# name: dim, form, kernel, tol, levels, points (grid side or -random count)
CASES = {
    "1d_tiny": (1, 0, 1, 10, 2, 37),
    "1d_semi": (1, 1, 0, 10, 5, 1111),
    "1d_semi_parts": (1, 1, 1, 8, 7, 20001),  # block rows of three column parts, from the input alone
    "2d_few_points": (2, 0, 1, 8, 3, -90),
    "2d_odd": (2, 0, 0, 10, 3, 41),
    "2d_plain": (2, 2, 1, 8, 3, -1501),
    "3d_wide": (3, 0, 0, 7, 2, -5003),
    "3d_semi_wide": (3, 1, 1, 7, 2, -4001),
    "3d_one_level_down": (3, 0, 0, 7, 3, 13),
    "3d_complex": (3, 0, 2, 7, 2, -1203),
}


def make(hw, case):
    dim, form, kern, tol, nlev, n = CASES[case]
    N = n ** dim if n > 0 else -n
    op = hw.H2Operator(dim, form, kern, tol, nlev, kernel_n=N, diag_n=2 * N if dim == 1 else N)
    if n > 0:
        op.gen_grid(n)
    else:
        op.set_points(synth.uniform_points(synth.config_seed(60, N), N, dim))
    op.build_tree()
    op.assemble()
    return op


def vec(op, seed):
    x = synth.normal(synth.config_seed(61, seed), op.N)
    return x + 1j * synth.normal(synth.config_seed(62, seed), op.N) if op.complex else x


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(CASES))
def test_single_vector_dataflow_product(gpu, case):
    hw = gpu
    op = make(hw, case)
    for prec, bound in ((hw.PREC_FP64, 1e-13), (hw.PREC_FP32, 5e-5)):
        if op.complex and prec == hw.PREC_FP32:
            continue
        x = vec(op, 1)
        y = op.matvec(x, precision=prec)
        assert np.array_equal(y, op.matvec(x, precision=prec))  # no atomics: the same on every run
        op.set_option(hw.OPT_COOP, 0)
        r = op.matvec(x, precision=prec)
        op.set_option(hw.OPT_COOP, 1)
        assert np.linalg.norm(y - r) <= bound * np.linalg.norm(r), (prec, np.linalg.norm(y - r) / np.linalg.norm(r))


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["1d_semi", "3d_wide"])
def test_single_vector_product_after_recut(gpu, case):
    """Every row split gives the same product, and one on a caller's stream too."""
    import torch
    hw = gpu
    op = make(hw, case)
    x = vec(op, 2)
    r = op.matvec(x)
    for rs in (256, 4096, 65536):
        op.set_option(hw.OPT_ROW_SPLIT, rs)
        y = op.matvec(x)
        assert np.linalg.norm(y - r) <= 1e-13 * np.linalg.norm(r), rs
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        xd = torch.from_numpy(x).cuda()
        yd = torch.empty_like(xd)
        op.matvec_device(xd.data_ptr(), yd.data_ptr(), stream=st.cuda_stream)
        got = yd.cpu().numpy()
    assert np.array_equal(got, y)


@pytest.mark.gpu
def test_single_vector_product_keeps_non_finite_rows_apart(gpu):
    """An infinity in one entry of x reaches the rows that use it and no others: rows whose
    exact product is finite in the launch by phases are finite here, and the same."""
    hw = gpu
    op = make(hw, "2d_odd")
    x = vec(op, 3)
    x[7] = np.inf
    y = op.matvec(x)
    op.set_option(hw.OPT_COOP, 0)
    r = op.matvec(x)
    assert np.array_equal(np.isfinite(y), np.isfinite(r))
    assert np.array_equal(np.isnan(y), np.isnan(r))
