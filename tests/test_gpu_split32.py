"""FP32 factorisation of large fronts, two-level with exact digit products
(lfg_factor32.cu).  A leaf size above the particle count makes the whole
system one dense front, large enough to take that path; its pivot columns
leave remainders of the panel, K block and tile widths."""
import numpy as np
import pytest

from _systems import RATE_PARAMS, make_packing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [400, 427, 448, 469])
def test_dense_front(oracle, engine, n):
    """The residual after one solve is at most 6n 2^-24 cond(R) |b| (Cholesky in
    FP32), refinement reaches 1e-12, and a second factorisation repeats the
    first bit for bit."""
    import _golden as G
    p = make_packing(n, 0.45, 41)
    o = oracle.OracleSim(RATE_PARAMS, p.position, p.radius, p.lx, p.ly, p.lz)
    o.first_time()
    d15, r, c, o18 = o.assemble()
    R = G.dense_from_blocks(oracle, d15, r, c, o18, n)
    b = np.random.default_rng(n).standard_normal((2, 6 * n))
    s = engine.Solver(n, engine.PREC_FP32_REFINE, leaf_size=1000, refine_max_iter=1, refine_tol=1.0)
    s.set_blocks(d15, r, c, o18, True, positions=p.position)
    assert s.stats()["max_front"] == 6 * n
    s.factorize()
    x = s.solve(b)
    res = np.abs(b - x @ R).max() / np.abs(b).max()
    assert res <= 6 * n * 2.0 ** -24 * np.linalg.cond(R)
    s.factorize()
    assert np.array_equal(s.solve(b), x)
    t = engine.Solver(n, engine.PREC_FP32_REFINE, leaf_size=1000, refine_tol=1e-12)
    t.set_blocks(d15, r, c, o18, True, positions=p.position)
    t.factorize()
    t.solve(b)
    assert t.last.refine_residual <= 1e-12
