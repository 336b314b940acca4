"""FP32 fronts that are updated two-level (lfg_factor32.cu): more than 4000 rows and
more than one outer block of panels.  One dense front, whose columns leave
remainders of panels, outer blocks and tiles; two cliques around a separator,
whose fronts have update rows and uneven panel counts, one of them too small for
the path; three unknowns per particle; entries that are not finite.  The launch
counts show that the path was taken."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PANEL, OUTER, ROWS = 64, 4, 4000
# dense positions of the compact values (diagonal block; off-diagonal block)
DIAG = [(0, 0), (0, 1), (0, 2), (0, 4), (0, 5), (1, 1), (1, 2), (1, 5), (2, 2), (3, 3), (3, 4), (3, 5), (4, 4), (4, 5),
        (5, 5)]
SEED = 11


def cliques(a, b, s):
    """Two cliques of a and b particles, both coupled to all of s between them, the
    couplings of a particle's row about as large as its diagonal entry."""
    n = a + s + b
    part = np.repeat([0, 1, 2], [a, s, b])
    r, c = np.tril_indices(n, -1)
    keep = part[r] - part[c] < 2
    r, c = r[keep].astype(np.int32), c[keep].astype(np.int32)
    rng = np.random.default_rng([a, b, s, SEED])
    d15, o18 = rng.uniform(-1, 1, (n, 15)), rng.uniform(-1, 1, (len(r), 18))
    o18 *= 0.8 / np.sqrt(n)
    d15[:, [0, 5, 8, 9, 12, 14]] = 6.0
    pos = np.column_stack([10.0 * part + 1 + 1e-3 * np.arange(n), np.ones(n), np.ones(n)])
    return n, d15, r, c, o18, pos


def dense(n, d15, r, c, o18, dof):
    """The matrix from its compact blocks (MatrixBlocks.h's layout)."""
    sym = np.zeros((6, 6), int)
    for q, (i, j) in enumerate(DIAG):
        sym[i, j] = sym[j, i] = q + 1
    sym[1, 3] = sym[3, 1] = -4
    sym[2, 3] = sym[3, 2] = -5
    sym[2, 4] = sym[4, 2] = -8
    off = np.array([[1, 2, 3, 0, -10, -11], [2, 6, 7, 10, 0, -15], [3, 7, 9, 11, 15, 0], [0, -4, -5, 12, 13, 14],
                    [4, 0, -8, 13, 16, 17], [5, 8, 0, 14, 17, 18]])
    keep = np.arange(6) if dof == 6 else np.array([0, 2, 4])
    A = np.zeros((n, dof, n, dof))

    def expand(v, t):
        e = np.where(t == 0, 0.0, np.sign(t) * v[:, np.abs(t) - 1])
        return e[:, keep][:, :, keep]
    i = np.arange(n)
    A[i, :, i, :] = expand(d15, sym)
    B = expand(o18, off)
    A[r, :, c, :] = B
    A[c, :, r, :] = B.transpose(0, 2, 1)
    return A.reshape(dof * n, dof * n)


def launches(fronts):
    """Launches of a factorisation of the levels of fronts (columns, rows)."""
    total = 0
    for level in fronts:
        total += 2 + any(m > n for n, m in level)   # assembly, panel 0, Schur complements
        for k in range(max(-(-n // PANEL) for n, _ in level)):
            more = [(n > 256 and m > ROWS and (k + 1) % OUTER == 0) for n, m in level if n > (k + 1) * PANEL]
            total += 1 + (False in more) + 2 * (True in more)   # solve; update; tiles and diagonal blocks
    return total


# particles of one dense front, or of (clique, clique, separator)
ONE = [667, 672, 683, 768]
TREES = [(430, 420, 250), (430, 300, 250), (480, 431, 240)]


def solver(engine, system, leaf, dof=6, **opts):
    n, d15, r, c, o18, pos = system
    s = engine.Solver(n, engine.PREC_FP32_REFINE, dof=dof, leaf_size=leaf, **opts)
    s.set_blocks(d15, r, c, o18, True, positions=pos)
    return s


def check(engine, s, t, system, fronts, dof):
    """Higham and Mary (2019): a computed inner product of length n is within
    lambda sqrt(n) u of its absolute values' with a probability of 1 - 2
    exp(-lambda^2 / 2) (lambda = 6: 1e-8 each).  Factor and two solves: the residual
    is within three times that of |L| |L^T| |x|, and a factor of two for the inverses of the
    diagonal blocks that the solves multiply with."""
    n, d15, r, c, o18, _ = system
    comp = np.arange(6) if dof == 6 else np.array([0, 2, 4])
    s.factorize()
    assert s.stats()["n_factor_launches"] == launches(fronts)
    assert s.stats()["max_front"] == max(m for level in fronts for _, m in level)
    b = np.zeros((2, n, 6))
    b[:, :, comp] = np.random.default_rng(n).standard_normal((2, n, len(comp)))
    x = s.solve(b.reshape(2, -1))
    A = dense(n, d15, r, c, o18, dof)
    L = np.abs(np.linalg.cholesky(A))
    xs, bs = x.reshape(2, n, 6)[:, :, comp].reshape(2, -1), b[:, :, comp].reshape(2, -1)
    bound = 3 * 2 * 6 * np.sqrt(dof * n) * 2.0 ** -24 * (L @ (L.T @ np.abs(xs).T)).T
    assert (np.abs(bs - xs @ A) <= bound).all()
    s.factorize()
    assert np.array_equal(s.solve(b.reshape(2, -1)), x)
    t.factorize()
    t.solve(b.reshape(2, -1))
    assert t.last.refine_residual <= 1e-12


ONCE, TIGHT = {"refine_max_iter": 1, "refine_tol": 1.0}, {"refine_tol": 1e-12}


@pytest.mark.parametrize("n", ONE)
def test_dense_front(engine, n):
    system = cliques(n, 0, 0)
    check(engine, solver(engine, system, n, **ONCE), solver(engine, system, n, **TIGHT), system, [[(6 * n, 6 * n)]], 6)


@pytest.mark.parametrize("a,b,s", TREES)
def test_fronts_with_update_rows(engine, a, b, s):
    system = cliques(a, b, s)
    fronts = [[(6 * a, 6 * (a + s)), (6 * b, 6 * (b + s))], [(6 * s, 6 * s)]]
    leaf = max(a, b)
    check(engine, solver(engine, system, leaf, **ONCE), solver(engine, system, leaf, **TIGHT), system, fronts, 6)


def test_three_unknowns(engine):
    system = cliques(1340, 0, 0)
    n = system[0]
    check(engine, solver(engine, system, n, 3, **ONCE), solver(engine, system, n, 3, **TIGHT), system,
          [[(3 * n, 3 * n)]], 3)


@pytest.mark.parametrize("n", [667, 683, 768])
def test_factor_against_64_bits(engine, n):
    """A component common to all particles makes the updates cancel the entries from 100
    to about 6, so a digit of the products that was lost (2^-17 of a row's
    largest) would show.  L b in FP32 is as close to L b in FP64 as LAPACK's FP32 factor
    of the same matrix is to its FP64 one: as many roundings of the same size, and a
    factor of four."""
    _, d15, r, c, o18, pos = cliques(n, 0, 0)
    d15[:, [0, 5, 8, 9, 12, 14]] += 100.0
    o18[:, [0, 5, 8, 11, 15, 17]] += 100.0
    v = np.random.default_rng(n).standard_normal((4, 6 * n))
    got = []
    for prec in (engine.PREC_FP32_REFINE, engine.PREC_FP64):
        t = engine.Solver(n, prec, leaf_size=n)
        t.set_blocks(d15, r, c, o18, True, positions=pos)
        t.factorize()
        got.append(t.multiply_L(v))
    A = dense(n, d15, r, c, o18, 6)
    ref = [np.linalg.cholesky(A.astype(t)).astype(t) @ v.T.astype(t) for t in (np.float32, np.float64)]
    assert np.linalg.norm(got[0] - got[1]) <= 4 * np.linalg.norm(ref[0] - ref[1])


def test_rows_up_to_the_largest_exponents(engine):
    """A chain of particles with R = L L^T, L's diagonal 1 and its entries between
    neighbours -2: the rows of its inverse grow to 2^125, in one dense front.  Everything is
    a power of two, so the solution is exact.  The chain ends two particles after an outer
    block (column 1024), whose rows of 2^123 are multiplied with entries of -2."""
    n, first, last = 667, 47, 172
    d15, o18 = np.zeros((n, 15)), np.zeros((last - first, 18))
    d15[:, [0, 5, 8, 9, 12, 14]] = 1.0
    d15[first + 1:last + 1, [0, 5, 8, 9, 12, 14]] += 4.0
    o18[:, [0, 5, 8, 11, 15, 17]] = -2.0
    r = np.arange(first + 1, last + 1, dtype=np.int32)
    s = engine.Solver(n, engine.PREC_FP32_REFINE, leaf_size=n, **ONCE)
    s.set_blocks(d15, r, r - 1, o18, True)
    s.factorize()
    assert s.stats()["max_front"] == 6 * n
    b, x = np.zeros((2, n, 6)), np.zeros((2, n, 6))
    for q, comp in enumerate((0, 3)):
        b[q, last, comp] = 1.0
        x[q, first:last + 1, comp] = 2.0 ** (last - np.arange(first, last + 1))
    assert np.array_equal(s.solve(b), x)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("where", ["diagonal", "offdiagonal"])
def test_not_finite_is_reported(engine, bad, where):
    n, d15, r, c, o18, pos = cliques(667, 0, 0)
    if where == "diagonal":
        d15[300, 0] = bad
    else:
        o18[len(r) // 2, 0] = bad
    s = solver(engine, (n, d15, r, c, o18, pos), n, **ONCE)
    with pytest.raises(engine.LFGError) as ei:
        s.factorize()
    assert ei.value.code == engine.LFG_ERR_NOT_SPD


def test_patterns_of_other_sizes_in_between(engine):
    """The workspaces of a larger analysis serve the smaller ones after it."""
    b = np.random.default_rng(3).standard_normal((1, 6 * 980))
    s = engine.Solver(980, engine.PREC_FP32_REFINE, leaf_size=430, **ONCE)
    for a, bb, sep in [(430, 300, 250), (300, 400, 280), (430, 420, 130), (430, 300, 250)]:
        system = cliques(a, bb, sep)
        n, d15, r, c, o18, pos = system
        assert n == 980
        s.set_blocks(d15, r, c, o18, True, positions=pos)
        s.factorize()
        t = solver(engine, system, 430, **ONCE)
        t.factorize()
        assert np.array_equal(s.solve(b), t.solve(b)) and np.array_equal(s.multiply_L(b), t.multiply_L(b))


def test_a_front_is_its_own_matter(engine):
    """A front that is not updated two-level itself has the same factor, bit for bit, in a
    level with one that is and in a level without."""
    a, b, sep = 430, 300, 250
    system = cliques(a, b, sep)
    n, d15, r, c, o18, pos = system
    keep = np.r_[0:260, a:n]   # the same separator and second clique beside a smaller first one
    new = np.full(n, -1)
    new[keep] = np.arange(len(keep))
    e = (new[r] >= 0) & (new[c] >= 0)
    small = (len(keep), d15[keep], new[r[e]].astype(np.int32), new[c[e]].astype(np.int32), o18[e], pos[keep])
    v = np.random.default_rng(9).standard_normal((2, n, 6))
    v[:, :a + sep] = 0   # the second clique's columns
    got = []
    for sys_, rows, fronts in ((system, slice(None), [[(6 * a, 6 * (a + sep)), (6 * b, 6 * (b + sep))], [(6 * sep, 6 * sep)]]),
                               (small, keep, [[(1560, 6 * (260 + sep)), (6 * b, 6 * (b + sep))], [(6 * sep, 6 * sep)]])):
        t = solver(engine, sys_, a, **ONCE)
        t.factorize()
        assert t.stats()["n_factor_launches"] == launches(fronts)
        y = t.multiply_L(v[:, rows].reshape(2, -1)).reshape(2, -1, 6)
        got.append(y[:, -(b + sep):])
    assert np.array_equal(got[0], got[1])
