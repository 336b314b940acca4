"""FP64 factorisation of matrices near the ends of the exponent range: the tile
products (lfg_factor64.cu) round results below the normal numbers as FP64 does."""
import numpy as np
import pytest

from _systems import RATE_PARAMS, make_packing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [-1000, -980, 0, 980])
@pytest.mark.parametrize("leaf", [16, 200])
def test_backward_error_of_scaled_systems(oracle, engine, power, leaf):
    """R times 2^power: |b - R x| <= 6n 2^-53 |R| |x| as for R itself (the residual of the
    rescaled solution in extended precision).  Values below the normal numbers are
    absolute errors of 2^-1074, 2^-74 of the matrix's unit at the most."""
    import _golden as G
    n = 150
    p = make_packing(n, 0.45, 31)
    o = oracle.OracleSim(RATE_PARAMS, p.position, p.radius, p.lx, p.ly, p.lz)
    o.first_time()
    d15, r, c, o18 = o.assemble()
    R = G.dense_from_blocks(oracle, d15, r, c, o18, n)
    b = np.random.default_rng(3).standard_normal((2, 6 * n))
    f = 2.0 ** power
    s = engine.Solver(n, engine.PREC_FP64, leaf_size=leaf)
    s.set_blocks(f * d15, r, c, f * o18, True, positions=p.position)
    s.factorize()
    x = s.solve(b) * f
    res = np.abs(b - x.astype(np.longdouble) @ R.astype(np.longdouble)).max(axis=1)
    bound = 6 * n * 2.0 ** -53 * (np.abs(x) @ np.abs(R)).max(axis=1)
    assert (res <= bound).all(), (res / bound)
