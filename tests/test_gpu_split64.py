"""FP64 factorisation with its tile products on the tensor cores
(lfg_factor64.cu): backward error of the solve at sizes whose fronts leave
remainders of every tile edge, exact behaviour under power-of-two scaling of
the matrix, and NaN / infinite entries still reported."""
import numpy as np
import pytest

from _systems import RATE_PARAMS, make_packing

pytestmark = pytest.mark.gpu


def _system(oracle, n, vf=0.45, seed=31):
    import _golden as G
    p = make_packing(n, vf, seed)
    o = oracle.OracleSim(RATE_PARAMS, p.position, p.radius, p.lx, p.ly, p.lz)
    o.first_time()
    d15, r, c, o18 = o.assemble()
    return p, d15, r, c, o18, G.dense_from_blocks(oracle, d15, r, c, o18, n)


def _solve(engine, p, d15, r, c, o18, b, leaf=16):
    s = engine.Solver(p.n, engine.PREC_FP64, leaf_size=leaf)
    s.set_blocks(d15, r, c, o18, True, positions=p.position)
    s.factorize()
    return s.solve(b)


@pytest.mark.parametrize("n,leaf", [(40, 16), (61, 1), (85, 64), (128, 7), (200, 22), (333, 16), (500, 200),
                                    (700, 16)])
def test_backward_error(oracle, engine, n, leaf):
    """|b - R x| <= 6n 2^-53 (|R| |x|) per row-sum norm, the classical bound of
    Cholesky in FP64 (the residual in extended precision); leaf sizes make
    fronts from 6 to 1200 pivot columns."""
    p, d15, r, c, o18, R = _system(oracle, n)
    b = np.random.default_rng(n).standard_normal((2, 6 * n))
    x = _solve(engine, p, d15, r, c, o18, b, leaf)
    Rl, xl = R.astype(np.longdouble), x.astype(np.longdouble)
    res = np.abs(b - xl @ Rl).max(axis=1)
    bound = 6 * n * 2.0 ** -53 * (np.abs(x) @ np.abs(R)).max(axis=1)
    assert (res <= bound).all(), (res / bound)


@pytest.mark.parametrize("power", [-400, -2, 2, 400])
def test_power_of_two_scaling_is_exact(oracle, engine, power):
    """R times 2^power (even) scales L by 2^(power/2): every rounding is the
    same, so x scales exactly."""
    p, d15, r, c, o18, _ = _system(oracle, 150)
    b = np.random.default_rng(3).standard_normal((1, 900))
    f = 2.0 ** power
    x = _solve(engine, p, d15, r, c, o18, b)
    y = _solve(engine, p, f * d15, r, c, f * o18, b)
    assert np.array_equal(y * f, x)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("where", ["diagonal", "offdiagonal"])
def test_nan_and_infinity_are_reported(oracle, engine, bad, where):
    p, d15, r, c, o18, _ = _system(oracle, 150)
    d, o = d15.copy(), o18.copy()
    if where == "diagonal":
        d[11, 0] = bad
    else:
        o[len(r) // 2, 0] = bad
    s = engine.Solver(p.n, engine.PREC_FP64)
    s.set_blocks(d, r, c, o, True, positions=p.position)
    with pytest.raises(engine.LFGError) as ei:
        s.factorize()
    assert ei.value.code == engine.LFG_ERR_NOT_SPD
