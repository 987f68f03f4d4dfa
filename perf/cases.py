"""What is measured: the Poisson-Boltzmann path's public entry points over the sizes they are used at.

A case is one call (or the short chain of calls) that a program makes through the Python binding:

  solve      Context.solve: atoms to solvation energy in one call (the reference's main program)
  batch      Context.batch_solve: several molecules at once
  electric   Tube.electric: plan, right-hand side, GMRES and energy on a tube that is there already
  matvec     Plan.matvec: one product with the boundary operator, as a caller's own solver makes it
  apply      Plan.apply: one scalar kernel's FMM, as a program of the black-box FMM makes it
  levelset   Context.levelset, Grid.download: atoms to the reinitialised level set

in the FP64 precision (the default, the reference's own) or the mixed one.  Molecules are the
repository's seeded synthetic proteins of 50 to 5,000 atoms and ions, orders 4 to 6, leaves of 64
to 160 points, kappa 0 to 0.15 / A.  The operator cases take their tubes from the atoms directly
(cells near the surface of the union of the atoms' spheres, projected onto it), so that their inputs
depend on nothing that is measured.

The mixed precision computes in single precision (level set, operator) or to the 1e-6 residual
of its solver; a program that chooses it keeps its results as single-precision numbers, and so
does run().  Iteration counts and times in the results are reports about a call, not its outputs.
"""

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ibim-levelset_gb300"))

import ibim  # noqa: E402
import synth  # noqa: E402

PROBE, BAND, REINIT_STEPS = 1.4, 8, 20
PRECISION = {"fp64": ibim.PRECISION_FP64, "mixed": ibim.PRECISION_MIXED}


def listed():
    return [
        # one ion on a 64^3 grid, FP64, order 4: the smallest whole call of the drop-in, where
        # launches, copies and host work count as much as arithmetic
        dict(name="solve_ion_fp64", kind="solve", precision="fp64", atoms=1, order=4, leaf=64, kappa=0.0, dI=1.0,
             thickness=3, cells=64),
        # a peptide through the default precision: what the drop-in's main program does
        dict(name="electric_protein100_fp64", kind="electric", precision="fp64", atoms=100, order=5, leaf=128,
             kappa=0.125, dI=2.0, thickness=2, cells=0),
        # one product of the FP64 operator, small, ordinary, large: a caller's own Krylov solver
        dict(name="matvec_protein60_fp64", kind="matvec", precision="fp64", atoms=60, order=4, leaf=160, kappa=0.1257,
             dI=1.0, thickness=2, cells=0),
        dict(name="matvec_protein500_fp64", kind="matvec", precision="fp64", atoms=500, order=5, leaf=128,
             kappa=0.125, dI=2.0, thickness=2, cells=0),
        dict(name="matvec_protein2000_fp64", kind="matvec", precision="fp64", atoms=2000, order=5, leaf=128,
             kappa=0.125, dI=2.0, thickness=2, cells=0),
        # one scalar kernel's FMM at order 6: a program of the black-box FMM alone
        dict(name="apply_protein150_fp64", kind="apply", precision="fp64", atoms=150, order=6, leaf=128, kappa=0.07,
             dI=2.0, thickness=2, cells=0, kernel="K3xy"),
        # the FP64 level set of a small protein
        dict(name="levelset_protein300_fp64", kind="levelset", precision="fp64", atoms=300, order=5, leaf=128,
             kappa=0.125, dI=2.0, thickness=2, cells=0),
        # the mixed path: a small molecule (latency) and the 2,000-atom benchmark protein
        dict(name="solve_protein60_mixed", kind="solve", precision="mixed", atoms=60, order=5, leaf=128, kappa=0.125,
             dI=2.0, thickness=2, cells=0),
        dict(name="solve_protein2000_mixed", kind="solve", precision="mixed", atoms=2000, order=5, leaf=128,
             kappa=0.125, dI=2.0, thickness=2, cells=0),
        # one product of the mixed operator: a small one at order 6, and the largest molecule of the batches
        dict(name="matvec_protein200_mixed", kind="matvec", precision="mixed", atoms=200, order=6, leaf=128,
             kappa=0.05, dI=2.0, thickness=2, cells=0),
        dict(name="matvec_protein5000_mixed", kind="matvec", precision="mixed", atoms=5000, order=5, leaf=128,
             kappa=0.125, dI=2.0, thickness=2, cells=0),
        # eight molecules of 50 to 400 atoms at once
        dict(name="batch_8x50_400_mixed", kind="batch", precision="mixed", atoms=400, order=5, leaf=128, kappa=0.15,
             dI=2.0, thickness=2, cells=0, molecules=8),
    ]


#: Per kind and precision of a drawn case: its weight and the range of its atom counts (log-uniform).
RANGES = {
    ("solve", "fp64"): (1, 1, 1),
    ("electric", "fp64"): (1, 20, 90),
    ("matvec", "fp64"): (2, 50, 1600),
    ("apply", "fp64"): (1, 50, 600),
    ("levelset", "fp64"): (1, 50, 400),
    ("levelset", "mixed"): (1, 100, 2000),
    ("solve", "mixed"): (2, 50, 1800),
    ("electric", "mixed"): (1, 50, 1500),
    ("matvec", "mixed"): (2, 50, 4500),
    ("batch", "mixed"): (1, 100, 400),
}


def draw(rng: random.Random):
    keys = list(RANGES)
    kind, precision = rng.choices(keys, weights=[RANGES[k][0] for k in keys])[0]
    _, lo, hi = RANGES[kind, precision]
    atoms = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    # order 6 holds 3 times order 5's operators: the whole solves draw 4 or 5
    order = rng.choice((4, 5)) if kind in ("solve", "electric", "batch") or atoms > 1000 else rng.choice((4, 5, 6))
    c = dict(kind=kind, precision=precision, atoms=atoms, order=order, leaf=rng.choice((64, 96, 128, 160)),
             kappa=round(rng.uniform(0.0, 0.15), 4), dI=rng.choice((1.0, 2.0)), thickness=2, cells=0)
    if atoms == 1:
        c.update(cells=rng.randrange(41, 65), thickness=3, kappa=0.0, order=4, leaf=64)
    if kind == "apply":
        c["kernel"] = rng.choice(ibim.KERNELS)
    if kind == "batch":
        c["molecules"] = rng.randrange(3, 9)
    return c


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------

_CTX = None


def _ctx():
    """The context that a program makes once and keeps."""
    global _CTX
    if _CTX is None:
        _CTX = ibim.Context(0)
    return _CTX


def _molecule(case, seed, atoms=None):
    atoms = case["atoms"] if atoms is None else atoms
    if atoms > 1:
        return synth.synthetic_protein(atoms, 1_000_003 * (seed + 1) + atoms)
    # an ion off the grid's and the octree's symmetry planes
    r = np.random.default_rng(seed)
    return synth.Molecule(r.uniform(-0.05, 0.05, (1, 3)), np.array([1.0 + 0.1 * r.random()]),
                          np.array([1.9 + 0.2 * r.random()]))


def _geometry(case):
    """The grid of a case: its own, or the cube that holds any synthetic protein of its size with the band's padding."""
    if case["cells"]:
        h = 12.0 / case["cells"]
        return synth.Geometry((-6.0, -6.0, -6.0), h, (case["cells"],) * 3)
    h = 0.5
    half = 2.2 * case["atoms"] ** (1.0 / 3.0) + 2.0 + 2.0 + PROBE + BAND * h + 2.0
    return synth.Geometry((-half,) * 3, h, (int(2 * half / h) + 2,) * 3)


def _config(case, geo, kappa=None):
    return ibim.default_config(lo=geo.lo, h=geo.h, n=geo.n, band=BAND, init=-2.0 * max(geo.n), probe=PROBE,
                               reinit_t=synth.reinit_time(REINIT_STEPS, geo.h), thickness=case["thickness"],
                               thres=1e-4, np=case["order"], maxpoint=case["leaf"], maxlevel=10,
                               kappa=case["kappa"] if kappa is None else kappa, dE=80.0, dI=case["dI"], tau=1.0,
                               restart=30, maxiter=200, tol=1e-6, precision=PRECISION[case["precision"]])


def _tube_points(mol, geo, count):
    """Tube quadrature of the surface of the union of the atoms, in FP64: (points, normals, cosine weights).
    The tube is as thick as `count` points make it (1.5 to 2 cells to either side)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    c = torch.as_tensor(mol.centers, dtype=torch.float64, device=dev)
    r = torch.as_tensor(mol.radii, dtype=torch.float64, device=dev)
    lo = torch.tensor(geo.lo, dtype=torch.float64, device=dev)
    n = torch.tensor(geo.n, device=dev)
    # every atom's signed distance at the cells around it, the smallest kept for each cell
    w = int(math.ceil((float(r.max()) + 4 * geo.h) / geo.h)) + 1
    off = torch.stack(torch.meshgrid(*[torch.arange(-w, w + 1, device=dev)] * 3, indexing="ij"), -1).reshape(-1, 3)
    phi = torch.full((int(n.prod()),), 1e9, dtype=torch.float64, device=dev)
    atom = torch.zeros(len(phi), dtype=torch.int64, device=dev)

    def around(i):
        ijk = ((c[i] - lo) / geo.h).round().long()[:, None, :] + off
        ok = ((ijk >= 0) & (ijk < n)).all(2)
        d = (lo + geo.h * ijk - c[i][:, None, :]).norm(dim=2) - r[i][:, None]
        cell = (ijk[..., 0] * n[1] + ijk[..., 1]) * n[2] + ijk[..., 2]
        return cell[ok], d[ok], i[:, None].expand_as(d)[ok]

    blocks = torch.arange(len(r), device=dev).split(512)
    for i in blocks:
        cell, d, _ = around(i)
        phi.scatter_reduce_(0, cell, d, "amin")
    for i in blocks:
        cell, d, k = around(i)
        own = d == phi[cell]
        atom[cell[own]] = k[own]
    size, order = phi.abs().sort()
    eps = float(size[count])
    cell = order[:count].sort().values
    x = lo + geo.h * torch.stack([cell // (n[1] * n[2]), cell // n[2] % n[1], cell % n[2]], 1)
    d, k = phi[cell], atom[cell]
    nrm = (x - c[k]) / (d + r[k])[:, None]
    wgt = (1.0 + torch.cos(math.pi * d / eps)) / (2.0 * eps)
    return tuple(a.cpu().numpy() for a in (x - d[:, None] * nrm, nrm, wgt))


def _vector(seed, n):
    """A smooth-free, order-one vector in host memory, as a Krylov solver's vectors are."""
    return np.random.default_rng([seed, 7]).uniform(-1.0, 1.0, n)


def _operator_inputs(case, seed):
    mol, geo = _molecule(case, seed), _geometry(case)
    p, n, w = _tube_points(mol, geo, int(_points(case)))
    return mol, geo, p, n, w, _vector(seed, 2 * len(w) if case["kind"] == "matvec" else len(w))


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    s = dict(kind=kind, single=case["precision"] == "mixed", ctx=ctx)
    if kind == "batch":
        # one of each size between 50 atoms and the case's, in a shuffled order, each with its kappa
        rng = random.Random(seed)
        m = case["molecules"]
        sizes = [int(round(50 * (case["atoms"] / 50) ** (i / (m - 1)))) for i in range(m)]
        rng.shuffle(sizes)
        mols = [_molecule(case, seed + 101 * i, k) for i, k in enumerate(sizes)]
        s["molecules"] = [(m.centers, m.charges, m.radii) for m in mols]
        s["cfgs"] = [_config(case, _geometry(dict(case, atoms=len(m.charges))), rng.uniform(0.0, case["kappa"])) for m in mols]
    elif kind in ("solve", "levelset"):
        s["mol"] = _molecule(case, seed)
        s["cfg"] = _config(case, _geometry(case))
    else:
        s["mol"], geo, p, n, w, s["x"] = _operator_inputs(case, seed)
        s["cfg"] = _config(case, geo)
        s["tube"] = ctx.tube(p, n, w, geo.h)
        if kind != "electric":
            s["kp"] = ibim.kernel_params(case["kappa"], 80.0, case["dI"], 1.0)
            s["plan"] = s["tube"].plan(case["order"], case["leaf"], 10, precision=PRECISION[case["precision"]])
            s["kernel"] = ibim.KERNELS.index(case["kernel"]) if kind == "apply" else None
    return s


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------

def run(state):
    kind, m = state["kind"], state.get("mol")
    if kind == "solve":
        r = state["ctx"].solve(m.centers, m.charges, m.radii, state["cfg"])
        out = dict(energy=np.float64(r["energy"]), area=np.float64(r["area"]), n_points=r["n_points"],
                   inclusion=r["inclusion"], steps=np.array(r["reinit_steps"]))
    elif kind == "batch":
        res, status, _ = state["ctx"].batch_solve(state["molecules"], state["cfgs"])
        out = dict(energy=np.array([r["energy"] for r in res]), area=np.array([r["area"] for r in res]),
                   n_points=np.array([r["n_points"] for r in res]), status=np.array(status))
    elif kind == "electric":
        r = state["tube"].electric(m.centers, m.charges, state["cfg"], want_x=True)
        out = dict(energy=np.float64(r["energy"]), x=r["x"], potential=r["atom_potential"])
    elif kind == "matvec":
        out = dict(y=state["plan"].matvec(state["kp"], state["x"]))
    elif kind == "apply":
        out = dict(y=state["plan"].apply(state["kernel"], state["kp"], state["x"]))
    else:
        g, steps = state["ctx"].levelset(m.centers, m.radii, state["cfg"])
        out = dict(phi=g.download(), steps=np.array(steps))
    if state["single"]:
        out = {k: v.astype(np.float32) if getattr(v, "dtype", None) == np.float64 else v for k, v in out.items()}
    return out


# ------------------------------------------------------------------------------------------------
# the work that a pass cannot do without
# ------------------------------------------------------------------------------------------------

def _points(case):
    """Tube points of a case, about: a sphere for the ion, else what the synthetic proteins have."""
    if case["atoms"] == 1:
        h = 12.0 / case["cells"]
        return 4 * math.pi * 2.0 ** 2 * 2 * case["thickness"] / h ** 2
    return 190.0 * case["atoms"] * (1.0 + 1.5 * case["atoms"] ** (-1.0 / 3.0))


def _matvec_flops(case):
    # per point about 9 leaves' worth of near-field pairs at 70 flops, and 3 pairs of (4 p^3)^2 operators
    return _points(case) * (70.0 * 9 * case["leaf"] + 3 * 2.0 * (4 * case["order"] ** 3) ** 2)


def work(case):
    kind, n = case["kind"], _points(case)
    double = 4.0 if case["precision"] == "mixed" else 8.0
    cells = float(_geometry(case).cells)
    levelset = 160 * 350.0 * cells  # 54 third-order steps of three stages
    iters = 25
    if kind == "matvec":
        return dict(bytes=double * (7 + 4) * n, flops=_matvec_flops(case))
    if kind == "apply":
        # one of the 16 kernels: 20 flops a pair, one (p^3)^2 operator
        return dict(bytes=double * (3 + 2) * n, flops=n * (20.0 * 9 * case["leaf"] + 6.0 * case["order"] ** 6))
    if kind == "electric":
        return dict(bytes=double * (7 + 2) * n, flops=iters * _matvec_flops(case))
    if kind == "levelset":
        return dict(bytes=double * cells, flops=levelset)
    if kind == "batch":
        m = case["molecules"]
        sizes = [dict(case, atoms=50 * (case["atoms"] / 50) ** (i / (m - 1)), kind="solve") for i in range(m)]
        parts = [work(c) for c in sizes]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    return dict(bytes=double * 5 * case["atoms"] + double * cells, flops=levelset + iters * _matvec_flops(case))


# ------------------------------------------------------------------------------------------------
# 64-bit values: the direct sums that the FMM approximates
# ------------------------------------------------------------------------------------------------

def _radial(case, d2, h):
    """c1, c4, k2, hd, ho of the kernel set at squared distance d2 (K3 = ho d d + hd 1) and the cutoff's mask."""
    eps, ieps, kappa = 80.0 / case["dI"], case["dI"] / 80.0, case["kappa"]
    inside = d2 < h * h
    r = torch.where(inside, torch.ones_like(d2), d2).sqrt_()
    t = kappa * r
    e = torch.exp(-t)
    et1 = e * (t + 1)
    ir3 = 1.0 / (r * r * r)
    q = 1.0 / (4 * math.pi)
    k2in = (math.exp(-kappa * h) - 1 + kappa * h) / kappa / (2 * math.pi) / (h * h) if kappa else 0.0
    f = dict(c1=(eps * et1 - 1) * ir3 * q, c4=(1 - ieps * et1) * ir3 * q, k2=(1 - e) / r * q, hd=(1 - et1) * ir3,
             ho=(e * ((t + 3) * t + 3) - 3) * ir3 / (r * r))
    return {k: v.masked_fill_(inside, k2in if k == "k2" else 0.0) for k, v in f.items()}


def exact(case, seed):
    if case["kind"] not in ("matvec", "apply"):
        return None
    _, geo, p, n, w, x = _operator_inputs(case, seed)
    ns = len(w)
    if ns > 140_000:  # the direct sum takes too long
        return None
    P, N, W, X = (torch.as_tensor(a, dtype=torch.float64, device="cuda") for a in (p, n, w, x))
    out = []
    rows = max(1, int(1e8 / ns))
    for i0 in range(0, ns, rows):
        T = P[i0:i0 + rows]
        d = [P[None, :, a] - T[:, None, a] for a in range(3)]
        f = _radial(case, d[0] * d[0] + d[1] * d[1] + d[2] * d[2], geo.h)
        if case["kind"] == "apply":
            name, k = case["kernel"][:2], ["xyz".index(c) for c in case["kernel"][2:]]
            if name == "K1":
                K = f["c1"] * d[k[0]]
            elif name == "K2":
                K = f["k2"]
            elif name == "K3":
                K = f["ho"] * d[k[0]] * d[k[1]] + (f["hd"] if k[0] == k[1] else 0.0)
            else:
                K = f["c4"] * d[k[0]]
            out.append(K @ X)
            continue
        Wh = W * geo.h ** 3
        m = [X[:ns] * N[:, a] * Wh for a in range(3)]
        psi = X[ns:] * Wh
        dm = d[0] * m[0] + d[1] * m[1] + d[2] * m[2]
        F = (f["c1"] * dm).sum(1) - f["k2"] @ psi
        cm = f["ho"] * dm - f["c4"] * psi
        G = [f["hd"] @ m[a] + (d[a] * cm).sum(1) for a in range(3)]
        Nt = N[i0:i0 + rows]
        out.append(torch.stack([F, Nt[:, 0] * G[0] + Nt[:, 1] * G[1] + Nt[:, 2] * G[2]]))
    if case["kind"] == "apply":
        return dict(y=torch.cat(out))
    fg = torch.cat(out, 1)
    eps = 80.0 / case["dI"]
    return dict(y=torch.cat([X[:ns] + fg[0] / (0.5 * (1 + eps)), X[ns:] + fg[1] / (0.5 * (1 + 1 / eps))]))
