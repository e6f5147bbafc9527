"""The real GMRES step (one cooperative launch) and the batch's lockstep steps at the sizes where they can go wrong:
rows around whole CTAs of 512, step caps, basis vectors beyond those that fit shared memory and rows that do
not fit it at all (both by a large step cap), the loop as a graph and by the host, starts that are
solutions already.

Bound: against modified Gram-Schmidt in numpy on the same products; the coefficients are sums in another order, sqrt(N)
2^-53 <= 1e-14 of their vectors' norms, over at most 9 steps of systems whose condition is below 1e4: 1e-9 of the
solution."""
import numpy as np
import pytest

from h2weak_gb300 import synth


def problem(hw, N, kern=1):
    op = hw.H2Operator(1, 0, kern, 10, 3, kernel_n=N, diag_n=2 * N)
    op.gen_grid(N)
    op.build_tree()
    op.assemble()
    x = synth.normal(synth.config_seed(82, N), N)
    return op, x, op.matvec(x)


def gmres(A, b, x, m, tol):
    r = b - A(x)
    nb, beta = np.linalg.norm(b), np.linalg.norm(r)
    if beta / nb <= tol:
        return x, 0, beta / nb
    V, H = [r / beta], np.zeros((min(m, 60) + 1, min(m, 60)))
    for i in range(min(m, 60)):
        w = A(V[i])
        for k in range(i + 1):
            H[k, i] = V[k] @ w
            w = w - H[k, i] * V[k]
        H[i + 1, i] = np.linalg.norm(w)
        V.append(w / H[i + 1, i])
        e = np.zeros(i + 2)
        e[0] = beta
        y = np.linalg.lstsq(H[:i + 2, :i + 1], e, rcond=None)[0]
        res = np.linalg.norm(e - H[:i + 2, :i + 1] @ y) / nb
        if res < tol:
            break
    return x + sum(v * c for v, c in zip(V, y)), i + 1, res


@pytest.mark.gpu
@pytest.mark.parametrize("N", [37, 511, 512, 513, 1025, 2600])
def test_gmres_steps(gpu, N):
    hw = gpu
    op, x, b = problem(hw, N)
    for m, tol in ((9, 6), (2, 9), (1, 9)):
        want, wit, wres = gmres(op.matvec, b, np.ones(N), m, 10.0 ** -tol)
        for graph in (1, 0, 1):
            op.set_option(hw.OPT_GRAPH, graph)
            got, it, res = op.gmres(b, max_iter=m, tol_pow=tol)
            assert it == wit, (m, graph, it, wit)
            assert np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want), (m, graph)
            assert abs(res - wres) <= 1e-9, (m, graph)
    got, it, _ = op.gmres(b, x0=x, tol_pow=9)
    assert it == 0 and np.array_equal(got, x)


@pytest.mark.gpu
@pytest.mark.parametrize("N,m", [(513, 8150), (1024, 8400), (1500, 8100)])
def test_gmres_steps_beyond_shared_memory(gpu, N, m):
    """Step caps whose column leaves room for three basis vectors, for no rows of w, and for one vector."""
    hw = gpu
    op, x, b = problem(hw, N)
    small = op.gmres(b, max_iter=30, tol_pow=12)
    got = op.gmres(b, max_iter=m, tol_pow=12)
    assert got[1] == small[1] and got[1] > 3
    assert np.linalg.norm(got[0] - small[0]) <= 1e-9 * np.linalg.norm(small[0])


@pytest.mark.gpu
def test_batch_steps_with_converged_problems(gpu):
    """Problems that start at their solution take no step and stay as they are; the others go on as alone,
    on the first call and on the captured loop."""
    hw = gpu
    sizes = (37, 511, 513, 1025, 64)
    probs = [problem(hw, N, kern=i % 2) for i, N in enumerate(sizes)]
    batch = hw.Batch([p[0] for p in probs])
    off = np.concatenate([[0], np.cumsum(sizes)])
    b = np.concatenate([p[2] for p in probs])
    alone = [op.gmres(rhs, tol_pow=9) for op, _, rhs in probs]
    for done in ((), (0, 3), (1, 2, 4), ()):
        x0 = np.ones(off[-1])
        for p in done:
            x0[off[p]:off[p + 1]] = probs[p][1]
        xs, its, _ = batch.gmres(b, x0=x0, tol_pow=9)
        for p in range(len(sizes)):
            got = xs[off[p]:off[p + 1]]
            if p in done:
                assert its[p] == 0 and np.array_equal(got, probs[p][1]), (done, p)
            else:
                assert its[p] == alone[p][1], (done, p, its[p], alone[p][1])
                assert np.linalg.norm(got - alone[p][0]) <= 1e-9 * np.linalg.norm(got), (done, p)
