"""Solvers on several host threads at once: their kernels share the SMs, so the
lanes of a warp leave its barrier waits at different turns.  Every result is the
one the solver gives alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIAGONAL = [0, 5, 8, 9, 12, 14]   # of the 15 values of a diagonal block


def _run(engine, precision, n, seed, turns, out):
    rng = np.random.default_rng([n, seed])
    pairs = [(i, j) for i in range(n) for j in range(max(0, i - 3), i)]
    pairs += [(i, i - 5 - i % 11) for i in range(20, n, 7)]
    r, c = (np.array(v, np.int32) for v in zip(*sorted(pairs)))
    d15, o18 = rng.uniform(-1, 1, (n, 15)), rng.uniform(-1, 1, (len(r), 18))
    d15[:, DIAGONAL] = 100.0
    b = rng.standard_normal((2, 6 * n))
    opts = {} if precision == engine.PREC_FP64 else {"refine_max_iter": 2, "refine_tol": 1.0}
    s = engine.Solver(n, precision, leaf_size=64, **opts)
    s.set_blocks(d15, r, c, o18, True)
    for turn in range(turns):
        s.set_blocks((1.0 + turn % 3) * d15, r, c, o18, False)
        s.factorize()
        out.append(s.solve(b))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_threads_match_alone(engine, precision):
    prec = engine.PREC_FP64 if precision == "fp64" else engine.PREC_FP32_REFINE
    sizes = [130, 300, 700, 301]
    alone = []
    for n in sizes:
        ref = []
        _run(engine, prec, n, 5, 3, ref)
        alone.append(ref)
    got = [[] for _ in sizes]
    threads = [threading.Thread(target=_run, args=(engine, prec, n, 5, 30, got[q])) for q, n in enumerate(sizes)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for ref, g in zip(alone, got):
        assert len(g) == 30
        assert all(np.array_equal(x, ref[turn % 3]) for turn, x in enumerate(g))
