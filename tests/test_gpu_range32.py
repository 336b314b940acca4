"""FP32 factorisation of matrices near the ends of the exponent range: pivots whose
reciprocal is below the normal numbers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIAGONAL = [0, 5, 8, 9, 12, 14]   # of the 15 values of a diagonal block


@pytest.mark.parametrize("power", [-110, 0, 100, 120, 121])
@pytest.mark.parametrize("n,leaf", [(1, 16), (9, 16), (40, 64), (130, 8)])
def test_scaled_systems(oracle, engine, n, leaf, power):
    """Diagonal entries up to 100 x 2^121 (FP32 ends at 2^128): the residual of Cholesky solves
    is within 3 (6n + 1) u |L| |L^T| |x| (Higham, Accuracy and Stability, theorem
    10.4), whatever the power of two; |L| |L^T| exceeds |R| by at most a factor of two
    here (the diagonal dominates).  A reciprocal below the normal numbers keeps 21
    bits: 8 u instead of u."""
    import _golden as G
    rng = np.random.default_rng([n, leaf])
    r = np.array([i for i in range(n) for j in range(max(0, i - 3), i)], np.int32)
    c = np.array([j for i in range(n) for j in range(max(0, i - 3), i)], np.int32)
    d15, o18 = rng.uniform(-1, 1, (n, 15)), rng.uniform(-1, 1, (len(r), 18))
    d15[:, DIAGONAL] = 100.0
    R = G.dense_from_blocks(oracle, d15, r, c, o18, n)
    b = rng.standard_normal((2, 6 * n))
    f = 2.0 ** power
    s = engine.Solver(n, engine.PREC_FP32_REFINE, leaf_size=leaf, refine_max_iter=1, refine_tol=1.0)
    s.set_blocks(f * d15, r, c, f * o18, True)
    s.factorize()
    x = s.solve(b) * f
    assert (np.abs(b - x @ R) <= 3 * (6 * n + 8) * 2.0 ** -24 * 2 * (np.abs(x) @ np.abs(R))).all()
