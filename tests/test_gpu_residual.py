"""The FP64 residual of the refinement and its norms: rows with no, few and many
off-diagonal blocks (a hub coupled to every particle), one to five right-hand
sides (the kernels take four at a time)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIAGONAL = [0, 5, 8, 9, 12, 14]   # of the 15 values of a diagonal block


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n,hub", [(1, 0), (5, 4), (6, 5), (11, 10), (40, 0), (40, 23), (700, 20)])
def test_residual_norm(oracle, engine, n, hub, k):
    """After one FP32 solve the reported residual is that of the returned x: the
    largest |b - A x| / |b|, to the rounding of the FP64 products (a row has at most
    30 (1 + blocks) of them, each sum within that many units of 2^-53)."""
    import _golden as G
    rng = np.random.default_rng([n, hub, k])
    pairs = sorted({(max(hub, j), min(hub, j)) for j in range(n) if j != hub} |
                   {(j, j - 1) for j in range(1, n) if j % 3 == 0}) if hub else []
    if n == 700:
        pairs = [p for p in pairs if hub not in p or p[0] < 90]
    r = np.array([p[0] for p in pairs], np.int32)
    c = np.array([p[1] for p in pairs], np.int32)
    d15 = rng.uniform(-1, 1, (n, 15))
    d15[:, DIAGONAL] = 18.0 * n
    o18 = rng.uniform(-1, 1, (len(pairs), 18))
    R = G.dense_from_blocks(oracle, d15, r, c, o18, n)
    b = rng.standard_normal((k, 6 * n))
    s = engine.Solver(n, engine.PREC_FP32_REFINE, refine_max_iter=1, refine_tol=1.0)
    s.set_blocks(d15, r, c, o18, True)
    s.factorize()
    x = s.solve(b)
    res = np.linalg.norm(b - x @ R, axis=1) / np.linalg.norm(b, axis=1)
    terms = 30 * (1 + np.bincount(np.r_[r, c], minlength=n).max())
    bound = terms * 2.0 ** -53 * (np.linalg.norm(np.abs(b) + np.abs(x) @ np.abs(R), axis=1) / np.linalg.norm(b, axis=1)).max()
    assert abs(s.last.refine_residual - res.max()) <= 2 * bound
    assert res.max() > 2 * bound   # the FP32 solve's error, well above the bound
