"""Solves and products with the factor (lfg_solve.cu) where their forms change:
fronts of up to and above 256 columns or update rows (and 1024 rows, where several
CTAs assemble a column), one and several column
chunks, one to five right-hand sides, both precisions.  A leaf size above the
particle count makes the whole system one dense front."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIAGONAL = [0, 5, 8, 9, 12, 14]   # of the 15 values of a diagonal block


def system(engine, oracle, n, leaf, precision, **opts):
    """A banded random system: particles coupled to the next 3 and, every 7th, to
    one further away."""
    import _golden as G
    rng = np.random.default_rng([n, leaf])
    pairs = [(i, j) for i in range(n) for j in range(max(0, i - 3), i)]
    pairs += [(i, i - 5 - i % 11) for i in range(20, n, 7)]
    r, c = (np.array(v, np.int32) for v in zip(*sorted(pairs)))
    d15, o18 = rng.uniform(-1, 1, (n, 15)), rng.uniform(-1, 1, (len(r), 18))
    d15[:, DIAGONAL] = 100.0
    s = engine.Solver(n, precision, leaf_size=leaf, **opts)
    s.set_blocks(d15, r, c, o18, True)
    s.factorize()
    return s, G.dense_from_blocks(oracle, d15, r, c, o18, n), rng


SIZES = [(42, 1000), (43, 1000), (85, 1000), (86, 1000), (130, 1000), (130, 8), (300, 50), (300, 1000), (700, 16)]


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n,leaf", SIZES)
def test_solve(oracle, engine, n, leaf, k):
    """The residual of Cholesky solves is within 3 (6n + 1) u |L| |L^T| |x| (Higham,
    Accuracy and Stability, theorem 10.4).  |L| |L^T| exceeds |R| by at most a
    factor of two here: the diagonal dominates, fill is second order."""
    for precision, u in ((engine.PREC_FP64, 2.0 ** -53), (engine.PREC_FP32_REFINE, 2.0 ** -24)):
        opts = {} if precision == engine.PREC_FP64 else {"refine_max_iter": 1, "refine_tol": 1.0}
        s, R, rng = system(engine, oracle, n, leaf, precision, **opts)
        b = rng.standard_normal((k, 6 * n))
        x = s.solve(b)
        bound = 3 * (6 * n + 1) * u * 2 * (np.abs(x) @ np.abs(R))
        assert (np.abs(b - x @ R) <= bound).all()
        assert np.array_equal(s.solve(b), x)


@pytest.mark.parametrize("n,leaf", [(42, 1000), (43, 1000), (130, 1000), (130, 8)])
def test_product(oracle, engine, n, leaf):
    """The products with the unit vectors are P^T L P: its square is R to the same
    bound, plus that of the products."""
    for precision, u in ((engine.PREC_FP64, 2.0 ** -53), (engine.PREC_FP32_REFINE, 2.0 ** -24)):
        s, R, _ = system(engine, oracle, n, leaf, precision)
        M = s.multiply_L(np.eye(6 * n)).T
        assert np.abs(M @ M.T - R).max() <= 3 * (6 * n + 1) * u * 2 * np.abs(R).max()
