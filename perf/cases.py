"""Performance cases: what users of the engine have it do, through its public
entry points.

Two kinds of user stand behind them.  LF_DEM's own C++ with its StokesSolver
replaced hands over the resistance blocks of every half time step as host
arrays, factors, and solves for a few force components (the `solver` cases).
A simulation that lives on the device is stepped, and its particles are read
back (`sim`, `brownian` and `sweep` cases: one suspension under rate or stress
control, a monolayer, a Brownian run, a rheology sweep of many suspensions in
one fused batch).  Sizes run from the parity tests' (60-500 particles) over
the benchmark's (N = 4096 in FP32 + refinement and FP64, the N = 8192
monolayer) to the largest of the serving workload (N = 16384).

Packings are periodic repetitions of a small relaxed packing (quick to make at
any size) with every particle displaced at random, so no two cells are alike.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import lf_dem_gb300 as E
from lf_dem_gb300 import packing

JITTER = 2e-3   # random displacement of a particle, in radii of the small species


# ----------------------------------------------------------------------------
# cases
# ----------------------------------------------------------------------------
def listed():
    return [
        # StokesSolver of a very small run: one right-hand side, latency only
        _solver("solver_60_fp64", 60, 1, "fp64", phi=0.40),
        # ... of a parity-test sized rate-controlled run: 3 force components
        _solver("solver_500_fp64", 500, 3, "fp64", phi=0.50),
        # ... in the FP32 factor + FP64 refinement form to the tight tolerance
        _solver("solver_2047_fp32", 2047, 4, "fp32", phi=0.54),
        # ... of the benchmark's size, in plain FP64
        _solver("solver_4096_fp64", 4096, 4, "fp64", phi=0.56),
        # the parity tests' suspension stepped in the default fast form: five
        # steps between two looks at the particles
        _sim("sim_200_fp32", 200, "fp32", "rate", phi=0.45, steps=5),
        # a 3D rate-controlled run in FP64, each step with stresses (every
        # step written out)
        _sim("sim_500_fp64_stress", 500, "fp64", "rate", phi=0.50, stress_out=True),
        # the benchmark's stress-controlled suspension: FP32 + refinement, FP64
        _sim("sim_4096_fp32", 4096, "fp32", "stress", phi=0.56),
        _sim("sim_4096_fp64", 4096, "fp64", "stress", phi=0.56),
        # the benchmark's monolayer, 3 unknowns per particle
        _sim("mono_8192_fp32", 8192, "fp32", "rate", phi=0.78, twodim=True),
        # the largest suspension of the serving workload
        _sim("sim_16384_fp32", 16384, "fp32", "stress", phi=0.50),
        # a Brownian run: the factor is also multiplied with a random vector
        {"name": "brownian_1000_fp64", "kind": "brownian", "n": 1000, "phi": 0.45, "steps": 1},
        # a rheology sweep: suspensions of uneven N in one fused batch
        {"name": "sweep_12", "kind": "sweep", "count": 12, "nmin": 256, "nmax": 1400, "phi": 0.50,
         "precision": "fp32", "steps": 1},
    ]


def _solver(name, n, nrhs, precision, phi):
    return {"name": name, "kind": "solver", "n": n, "nrhs": nrhs, "precision": precision, "phi": phi}


def _sim(name, n, precision, control, phi, steps=1, stress_out=False, twodim=False):
    return {"name": name, "kind": "sim", "n": n, "precision": precision, "control": control, "phi": phi,
            "steps": steps, "stress_out": stress_out, "twodim": twodim}


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solver", "solver", "sim", "sim", "sim", "mono", "brownian", "sweep"])
    precision = rng.choice(["fp64", "fp32"])
    if kind == "solver":
        c = _solver("", size(60, 4000), rng.randint(1, 4), precision, phi=rng.choice([0.40, 0.45, 0.50, 0.54]))
    elif kind == "sim":
        c = _sim("", size(60, 4000 if precision == "fp64" else 16000), precision, rng.choice(["rate", "stress"]),
                 phi=rng.choice([0.45, 0.50, 0.54]), steps=rng.randint(1, 3), stress_out=rng.random() < 0.3)
        if c["n"] > 1500:
            c["steps"] = 1
    elif kind == "mono":
        c = _sim("", size(200, 8000), precision, rng.choice(["rate", "stress"]), phi=rng.choice([0.70, 0.78]),
                 twodim=True)
    elif kind == "brownian":
        c = {"kind": "brownian", "n": size(100, 3000), "phi": rng.choice([0.40, 0.45]), "steps": 1}
    else:
        c = {"kind": "sweep", "count": rng.randint(3, 14), "nmin": size(100, 300), "nmax": size(500, 1400),
             "phi": 0.50, "precision": precision, "steps": 1}
    c.pop("name", None)
    return c


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _base(n, phi, twodim):
    """A relaxed packing of n particles in its periodic box."""
    return packing.generate(n, phi, seed=7, twodim=twodim)


def _repeats(n, twodim):
    """Repetitions per axis so that one cell holds a few hundred particles."""
    axes = 2 if twodim else 3
    r = 1
    while n / (r + 1) ** axes >= 250:
        r += 1
    return r


def _suspension(n, phi, seed, twodim=False):
    """Positions, radii, box of n particles: a relaxed cell repeated, every
    particle displaced by its own random vector; what a cell short of n
    leaves over is dropped from the last cells."""
    r = _repeats(n, twodim)
    ry = 1 if twodim else r
    cell = _base(-(-n // (r * ry * r)), phi, twodim)
    off = np.array([(i * cell.lx, j * cell.ly, k * cell.lz) for i in range(r) for j in range(ry) for k in range(r)])
    pos = (cell.position[None] + off[:, None]).reshape(-1, 3)[:n]
    rad = np.tile(cell.radius, len(off))[:n]
    lx, ly, lz = r * cell.lx, ry * cell.ly, r * cell.lz
    rng = np.random.default_rng([seed, n])
    d = rng.uniform(-JITTER, JITTER, (n, 3))
    shift = rng.uniform(0, 1, 3) * (lx, ly, lz)
    if twodim:
        d[:, 1] = 0.0
    pos = pos + d + shift
    for ax, side in ((0, lx), (1, ly), (2, lz)):
        pos[:, ax] = np.mod(pos[:, ax], side) if side else 0.0
        pos[pos[:, ax] >= side, ax] = 0.0
    return np.ascontiguousarray(pos), np.ascontiguousarray(rad), lx, ly, lz


def _params(control, seed=0, brownian=0.0):
    p = dict(kn=1e4, kt=5e3, mu_static=1.0, mu_dynamic=1.0, friction_model=1, critical_load=0.0, ft_max=0.0,
             repulsion_on=1, repulsion=1.0, repulsive_length=0.05, repulsive_max_length=-1.0, lubrication_model=2,
             lub_reduce_parameter=1e-3, lub_max_gap=0.5, interaction_range=-1.0, sd_coeff=1.0,
             contact_relaxation_time=1e-3, contact_relaxation_time_tan=-1.0, disp_max=1e-3, dt=1e-4, dt_max=-1.0,
             dt_min=-1.0, fixed_dt=0, integration_method=1, control=0, shear_rate=1.0, target_stress=0.0,
             Ehat=(0, 0, 0.5, 0, 0, 0), Ohat=(0, 0.5, 0), init_strain_shear_rate_limit=0.0,
             init_shear_rate_limit=999.0)
    if control == "stress":
        p.update(friction_model=2, critical_load=1.0, repulsion_on=0, repulsion=0.0, control=1, shear_rate=0.0,
                 target_stress=10.0 / 6 / math.pi)
    if brownian:
        p.update(brownian=brownian, seed=seed % (1 << 31), fixed_dt=1, dt=1e-5)
    return p


def _precision(name):
    return E.PREC_FP64 if name == "fp64" else E.PREC_FP32_REFINE


def _blocks(n, phi, seed):
    """Resistance blocks of a suspension in LF_DEM's compact forms: for every
    pair in lubrication range a drag on the relative velocity of the two
    surfaces (1/h along the normal, log 1/h across it), and each particle's
    Stokes drag."""
    pos, rad, lx, ly, lz = _suspension(n, phi, seed)
    box = torch.tensor([lx, ly, lz], dtype=torch.float64)
    P, A = torch.from_numpy(pos), torch.from_numpy(rad)
    col, row = [], []
    for a in range(0, n, 512):
        d = P[None] - P[a:a + 512, None]
        d -= box * torch.round(d / box)
        near = (d * d).sum(2) < (1.25 * (A[a:a + 512, None] + A[None])) ** 2
        i, j = torch.nonzero(near, as_tuple=True)
        keep = j > i + a
        col.append(i[keep] + a)
        row.append(j[keep])
    i, j = torch.cat(col).numpy(), torch.cat(row).numpy()
    d = pos[j] - pos[i]
    d -= np.array([lx, ly, lz]) * np.round(d / np.array([lx, ly, lz]))
    r = np.sqrt((d * d).sum(1))
    n_ = d / r[:, None]
    ai, aj = rad[i], rad[j]
    h = np.maximum(2 * r / (ai + aj) - 2, 0.0) + 1e-3
    red = ai * aj / (ai + aj)
    an, at = 2 * red ** 2 / h, red * np.log(1 + 1 / h)
    nn = n_[:, :, None] * n_[:, None, :]
    eye = np.eye(3)[None]
    T = an[:, None, None] * nn + at[:, None, None] * (eye - nn)
    Q = at[:, None, None] * (eye - nn)
    N = np.zeros((len(i), 3, 3))   # N v = n x v
    N[:, 0, 1], N[:, 0, 2], N[:, 1, 2] = -n_[:, 2], n_[:, 1], -n_[:, 0]
    N[:, 1, 0], N[:, 2, 0], N[:, 2, 1] = n_[:, 2], -n_[:, 1], n_[:, 0]
    N *= at[:, None, None]
    u, v = ai[:, None, None], aj[:, None, None]
    od = np.zeros((len(i), 6, 6))   # rows: particle j, columns: particle i
    od[:, :3, :3], od[:, :3, 3:], od[:, 3:, :3], od[:, 3:, 3:] = -T, u * N, v * N, u * v * Q
    dia = np.zeros((n, 6, 6))
    k = np.arange(3)
    dia[:, k, k], dia[:, k + 3, k + 3] = rad[:, None], (4.0 / 3) * rad[:, None] ** 3
    for who, a, s in ((i, u, 1.0), (j, v, -1.0)):
        m = np.zeros((len(i), 6, 6))
        m[:, :3, :3], m[:, 3:, :3], m[:, 3:, 3:] = T, s * a * N, a * a * Q
        m[:, :3, 3:] = m[:, 3:, :3].transpose(0, 2, 1)
        np.add.at(dia, who, m)
    rc = [(0, 0), (1, 0), (2, 0), (4, 0), (5, 0), (1, 1), (2, 1), (5, 1), (2, 2), (3, 3), (4, 3), (5, 3), (4, 4),
          (5, 4), (5, 5)]
    d15 = np.stack([dia[:, a, b] for a, b in rc], 1)
    rc = [(0, 0), (1, 0), (2, 0), (4, 0), (5, 0), (1, 1), (2, 1), (5, 1), (2, 2), (1, 3), (2, 3), (3, 3), (4, 3),
          (5, 3), (2, 4), (4, 4), (5, 4), (5, 5)]
    o18 = np.stack([od[:, a, b] for a, b in rc], 1)
    return pos, dia, od, np.ascontiguousarray(d15), j.astype(np.int32), i.astype(np.int32), np.ascontiguousarray(o18)


def _sweep_sizes(case):
    k = case["count"]
    return [int(round(case["nmin"] * (case["nmax"] / case["nmin"]) ** (q / max(k - 1, 1)))) for q in range(k)]


def prepare(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "solver":
        pos, _, _, d15, row, col, o18 = _blocks(n, case["phi"], seed)
        rhs = np.random.default_rng([seed, n, 1]).standard_normal((case["nrhs"], 6 * n))
        opts = {"refine_tol": 1e-12} if case["precision"] == "fp32" else {}
        s = E.Solver(n, _precision(case["precision"]), **opts)
        s.set_blocks(d15, row, col, o18, True, positions=pos)   # the pattern is analysed once
        return {"case": case, "solver": s, "blocks": (d15, row, col, o18), "rhs": rhs}
    if kind == "sim":
        sus = _suspension(n, case["phi"], seed, case["twodim"])
        return {"case": case, "sim": E.Sim(_params(case["control"]), *sus, precision=_precision(case["precision"]))}
    if kind == "brownian":
        sus = _suspension(n, case["phi"], seed)
        return {"case": case, "sim": E.Sim(_params("rate", seed, brownian=1e-3), *sus, precision=E.PREC_FP64)}
    b = E.Batch(fused=True, precision=_precision(case["precision"]))
    for q, m in enumerate(_sweep_sizes(case)):
        p = _params("rate")
        p["shear_rate"] = 10.0 ** (-2 + 4 * q / max(case["count"] - 1, 1))
        b.add(p, *_suspension(m, case["phi"], seed + q))
    return {"case": case, "batch": b, "sims": [b.sim(q) for q in range(case["count"])]}


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------
def _read(sim):
    p = sim.particles()
    return {"pos": p["pos"], "vel": p["vel"], "ang": p["ang"]}


def run(state):
    case = state["case"]
    if case["kind"] == "solver":
        # a half time step of LF_DEM: new values in the known pattern, factor,
        # solve for the force components
        s = state["solver"]
        d15, row, col, o18 = state["blocks"]
        s.set_blocks(d15, row, col, o18, False)
        s.factorize()
        return {"x": s.solve(state["rhs"])}
    if case["kind"] == "sweep":
        state["batch"].run(case["steps"])
        return [_read(s) for s in state["sims"]]
    sim = state["sim"]
    if case.get("stress_out"):
        for _ in range(case["steps"]):
            sim.step(calc_stress=True)
        return dict(_read(sim), total_stress=sim.scalars()["total_stress"],
                    contact_stress=sim.particle_stress(0), hydro_stress=sim.particle_stress(2))
    sim.run(case["steps"])
    return _read(sim)


# ----------------------------------------------------------------------------
# what a pass cannot do without, and its values in 64 bits
# ----------------------------------------------------------------------------
def _factor(n, phi, twodim):
    """Flops of one Cholesky factorisation under nested dissection and the
    entries of its factor, fitted to symbolic analyses of these packings (48
    GFLOP and 24 million entries at N = 4096, phi = 0.56)."""
    if twodim:
        return 4.6e8 * (n / 8192) ** 1.5, 2.3e6 * (n / 8192) ** 1.2
    flops = 48e9 * (n / 4096) ** 2.1 * (phi / 0.56)
    nnz = 24e6 * (n / 4096) ** 1.47 * (phi / 0.56)
    return min(flops, (6 * n) ** 3 / 3), min(nnz, 18 * n * (n + 1))


def _one_step(n, phi, precision, nrhs, twodim, halves):
    """bytes, flops of `halves` factorisations, each with nrhs solves: the
    blocks read, the factor written once and read twice by the solves."""
    flops, nnz = _factor(n, phi, twodim)
    w = 8 if precision == "fp64" else 4
    unknowns = (3 if twodim else 6) * n
    pairs = (2.6 if twodim else 5.1) * n
    by = 8 * (15 * n + 18 * pairs) + 3 * w * nnz + 16 * nrhs * unknowns
    return halves * by, halves * (flops + 4.0 * nnz * nrhs)


def work(case):
    kind, phi = case["kind"], case["phi"]
    if kind == "solver":
        b, f = _one_step(case["n"], phi, case["precision"], case["nrhs"], False, 1)
    elif kind == "sweep":
        parts = [_one_step(m, phi, case["precision"], 1, False, 2 * case["steps"]) for m in _sweep_sizes(case)]
        b, f = (sum(x) for x in zip(*parts))
    else:
        nrhs = 4 if case.get("control") == "stress" or case.get("stress_out") else 1
        b, f = _one_step(case["n"], phi, case.get("precision", "fp64"), nrhs, case.get("twodim", False),
                         2 * case["steps"])
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """The solutions by a dense Cholesky factorisation in FP64, refined with
    residuals in extended precision; the stepped simulations have no closed
    form without the whole engine."""
    if case["kind"] != "solver":
        return None
    n, k = case["n"], case["nrhs"]
    _, dia, od, _, row, col, _ = _blocks(n, case["phi"], seed)
    rhs = np.random.default_rng([seed, n, 1]).standard_normal((k, 6 * n))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    A = torch.zeros((n, n, 6, 6), dtype=torch.float64, device=dev)
    at = torch.arange(n, device=dev)
    r, c = torch.from_numpy(row).long().to(dev), torch.from_numpy(col).long().to(dev)
    A[at, at] = torch.from_numpy(dia).to(dev)
    A[r, c] = torch.from_numpy(od).to(dev)
    A[c, r] = torch.from_numpy(od).to(dev).transpose(1, 2)
    A = A.permute(0, 2, 1, 3).reshape(6 * n, 6 * n)
    L = torch.linalg.cholesky(A)
    del A
    b = rhs.astype(np.longdouble)
    x = np.zeros_like(b)
    dl, ol = dia.astype(np.longdouble), od.astype(np.longdouble)
    res = b
    for _ in range(3):
        dx = torch.cholesky_solve(torch.from_numpy(res.astype(np.float64)).to(dev).T.contiguous(), L).T
        x = x + dx.cpu().numpy()
        xb = x.reshape(k, n, 6)
        y = np.einsum("nab,knb->kna", dl, xb)
        for q in range(k):
            np.add.at(y[q], row, np.einsum("eab,eb->ea", ol, xb[q, col]))
            np.add.at(y[q], col, np.einsum("eab,ea->eb", ol, xb[q, row]))
        res = b - y.reshape(k, -1)
    return {"x": x.astype(np.float64)}
