"""The refinement's norms (k_norms): a cluster of CTAs per right-hand side adds
its sums up in the first CTA's shared memory.  Small systems leave most of the
cluster without entries, so those CTAs store at once, before the first may have
started: every one of many solves reports the same residual."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIAGONAL = [0, 5, 8, 9, 12, 14]   # of the 15 values of a diagonal block


@pytest.mark.parametrize("n,k", [(1, 1), (2, 4), (85, 8), (86, 8), (700, 3)])
def test_every_solve_reports_the_same_residual(oracle, engine, n, k):
    """The reported residual is that of the returned x to the rounding of the FP64
    products (at most 60 of them a row, each sum within that many units of
    2^-53), and 200 solves repeat it bit for bit."""
    import _golden as G
    rng = np.random.default_rng([n, k])
    r, c = np.arange(1, n, dtype=np.int32), np.arange(0, n - 1, dtype=np.int32)
    d15, o18 = rng.uniform(-1, 1, (n, 15)), rng.uniform(-1, 1, (n - 1, 18))
    d15[:, DIAGONAL] = 30.0
    R = G.dense_from_blocks(oracle, d15, r, c, o18, n)
    b = rng.standard_normal((k, 6 * n))
    s = engine.Solver(n, engine.PREC_FP32_REFINE, refine_max_iter=1, refine_tol=1.0)
    s.set_blocks(d15, r, c, o18, True)
    s.factorize()
    x = s.solve(b)
    first = s.last.refine_residual
    nb = np.linalg.norm(b, axis=1)
    res = np.linalg.norm(b - x @ R, axis=1) / nb
    bound = 60 * 2.0 ** -53 * (np.linalg.norm(np.abs(b) + np.abs(x) @ np.abs(R), axis=1) / nb).max()
    assert abs(first - res.max()) <= 2 * bound
    for _ in range(200):
        s.solve(b)
        assert s.last.refine_residual == first
