"""The complex GMRES step (one cooperative launch, rotations on the device) against the same
iteration in numpy on the same products: fewer points than a CTA has threads, the sizes around
whole CTAs, the step cap, the Hermitian option, a start that is the solution already.

Bound: the coefficients are sums in another order, sqrt(N) 2^-53 <= 1e-14 of their vectors'
norms, over at most 9 steps of systems whose condition is below 1e4: 1e-9 of the solution."""
import numpy as np
import pytest

from h2weak_gb300 import synth


def problem(hw, N, nlev):
    op = hw.H2Operator(3, 0, 2, 7, nlev, kernel_n=N, diag_n=N)
    op.set_points(synth.uniform_points(synth.config_seed(67, N), N, 3))
    op.build_tree()
    op.assemble()
    x = synth.normal(synth.config_seed(68, N), N) + 1j * synth.normal(synth.config_seed(69, N), N)
    return op, x


def gmres(A, b, x, m, tol, herm):
    r = b - A(x)
    nb, beta = np.linalg.norm(b), np.linalg.norm(r)
    if beta / nb <= tol:
        return x, 0, beta / nb
    V, H, s = [r / beta], np.zeros((m + 1, m), complex), np.zeros(m + 1, complex)
    s[0], rot = beta, []

    def turn(p, q, c, d):
        return c * p + d * q, (-np.conj(d) if herm else -d) * p + c * q

    for i in range(m):
        w = A(V[i])
        for k in range(i + 1):
            H[k, i] = np.vdot(V[k], w) if herm else np.vdot(w, V[k])
            w = w - H[k, i] * V[k]
        H[i + 1, i] = np.linalg.norm(w)
        V.append(w / H[i + 1, i])
        for k, (c, d) in enumerate(rot):
            H[k, i], H[k + 1, i] = turn(H[k, i], H[k + 1, i], c, d)
        p, q = H[i, i], H[i + 1, i]
        n = np.hypot(abs(p), abs(q))
        rot.append((abs(p) / n, p / abs(p) * np.conj(q) / n))
        H[i, i], H[i + 1, i] = turn(p, q, *rot[i])
        s[i], s[i + 1] = turn(s[i], s[i + 1], *rot[i])
        res = abs(s[i + 1]) / nb
        if res < tol:
            break
    y = np.linalg.solve(np.triu(H[:i + 1, :i + 1]), s[:i + 1])
    x = x + sum(v * c for v, c in zip(V, y))
    if res < tol:
        return x, i + 1, res
    res = np.linalg.norm(b - A(x)) / nb
    return x, m + 1 if res < tol else m, res


@pytest.mark.gpu
@pytest.mark.parametrize("N,nlev", [(61, 2), (255, 2), (257, 2), (1025, 2), (2600, 2)])
@pytest.mark.parametrize("herm", [0, 1])
def test_complex_gmres_steps(gpu, N, nlev, herm):
    hw = gpu
    op, x = problem(hw, N, nlev)
    op.set_option(hw.OPT_COMPLEX_ARNOLDI, herm)
    b = op.matvec(x)
    for m, tol in ((9, 6), (2, 9), (1, 9)):
        got, it, res = op.gmres(b, max_iter=m, tol_pow=tol)
        want, wit, wres = gmres(op.matvec, b, np.ones(N, complex), m, 10.0 ** -tol, bool(herm))
        assert it == wit, (m, it, wit)
        assert np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want), m
        assert abs(res - wres) <= 1e-9
    again, it2, _ = op.gmres(b, max_iter=1, tol_pow=9)  # the captured step once more
    assert it2 == it and np.array_equal(again, got)
    got, it, _ = op.gmres(b, x0=x, tol_pow=9)
    assert it == 0 and np.array_equal(got, x)
