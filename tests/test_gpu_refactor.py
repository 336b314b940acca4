"""New values in a known pattern: factor and solve again with the same solver.
One-front systems are the ones whose first solve phase reads what the
factorisation's last kernel wrote."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIAGONAL = [0, 5, 8, 9, 12, 14]   # of the 15 values of a diagonal block


@pytest.mark.parametrize("n,leaf", [(1, 16), (10, 16), (11, 16), (43, 64), (90, 128), (90, 8)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_new_values_give_what_a_new_solver_gives(engine, n, leaf, precision):
    prec = engine.PREC_FP64 if precision == "fp64" else engine.PREC_FP32_REFINE
    opts = {} if precision == "fp64" else {"refine_max_iter": 1, "refine_tol": 1.0}
    rng = np.random.default_rng([n, leaf])
    r = np.array([i for i in range(n) for j in range(max(0, i - 2), i)], np.int32)
    c = np.array([j for i in range(n) for j in range(max(0, i - 2), i)], np.int32)
    b = rng.standard_normal((2, 6 * n))
    s = engine.Solver(n, prec, leaf_size=leaf, **opts)
    for turn in range(6):   # the third and later solves replay captured graphs
        d15, o18 = rng.uniform(-1, 1, (n, 15)), rng.uniform(-1, 1, (len(r), 18))
        d15[:, DIAGONAL] = 60.0 + turn
        s.set_blocks(d15, r, c, o18, turn == 0)
        s.factorize()
        x, y = s.solve(b), s.multiply_L(b)
        t = engine.Solver(n, prec, leaf_size=leaf, **opts)
        t.set_blocks(d15, r, c, o18, True)
        t.factorize()
        assert np.array_equal(x, t.solve(b)) and np.array_equal(y, t.multiply_L(b))
