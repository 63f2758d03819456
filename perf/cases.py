"""The work a user of this package has it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``kind`` names the public entry point:

  nk       ``mmff_minimize_nk``: host arrays in, host arrays out (packing, upload, launches, read-back)
  step     ``BinnedMinimizer.minimize_device``: tables resident, positions on the device
  eg       ``Minimizer.energy_grad``: energies and gradients of given conformers
  multi    ``mmff_optimize_metal_multi_mol``: the multi-molecule L-BFGS, molecules in and out
  dg, etk  ``DGDeviceBatch`` / ``ETKDeviceBatch.minimize_device``: the embedding stages, resident

``mols`` molecules of ``lo`` to ``hi`` atoms with ``confs`` conformers each, minimised for ``iters``
iterations.  A minimisation run to its end settles, for some conformers, in another basin after any
change of the order of a sum, so budgets are those of a short relaxation: the work of an iteration
is that of a long run, and hardly any conformer ends before its budget.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "mlxmolkit-archive_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from mlxmolkit_b200 import mmff_minimize as mm  # noqa: E402
from mlxmolkit_b200 import synth  # noqa: E402
from mlxmolkit_b200.conformer_metal import DGDeviceBatch  # noqa: E402
from mlxmolkit_b200.dg_extract import synth_dg_params  # noqa: E402
from mlxmolkit_b200.etk_extract import synth_etk_params  # noqa: E402
from mlxmolkit_b200.etk_metal import ETKDeviceBatch  # noqa: E402
from mlxmolkit_b200.mmff_metal_optimizer import mmff_optimize_metal_multi_mol  # noqa: E402
from mlxmolkit_b200.mmff_params import extract_mmff_params  # noqa: E402
from mlxmolkit_b200.shared_batch import add_etk_to_batch, pack_shared_dg_batch  # noqa: E402

NOISE = 0.1     # Gaussian noise of the starting coordinates, Angstrom


def listed():
    return [
        # one conformer of one small molecule through the drop-in call: what an interactive user waits for
        _case("nk", 1, 1, 18, 30, 10, name="nk_one"),
        # an ordinary drop-in call: a handful of drug-like molecules, ten conformers each, host to host
        _case("nk", 24, 10, 18, 150, 10, name="nk_ordinary"),
        # the small benchmark's shape (10-30 heavy atoms, 2500 conformers), tables resident
        _case("step", 24, 104, 23, 72, 5, name="step_small"),
        # uneven drug-like sizes (18-150 atoms), thousands of conformers: the main benchmark's step
        _case("step", 40, 125, 18, 150, 5, name="step_druglike"),
        # a few conformers of the largest dense sizes: a request on an idle GPU, bound by latency
        _case("step", 3, 5, 90, 150, 10, name="step_few"),
        # large and flexible molecules by L-BFGS (the optimizer from 150 atoms on)
        _case("step", 14, 48, 131, 400, 8, lbfgs=True, name="step_lbfgs"),
        # all-FP64 dense BFGS: the precision option that checks the others
        _case("step", 24, 21, 18, 110, 15, precision="fp64", name="step_fp64"),
        # scoring: energies and gradients of conformers in hand, host to host
        _case("eg", 40, 53, 18, 150, 0, name="energy_grad"),
        # the multi-molecule L-BFGS call on molecules (term extraction included, as users call it)
        _case("multi", 6, 31, 23, 72, 6, lbfgs=True, name="multi_mol"),
        # distance geometry in 4-D, 1000 conformers (the reference's 20 x 50 row)
        _case("dg", 20, 50, 23, 80, 3, lbfgs=True, name="dg_20x50"),
        # distance geometry of a larger batch of small molecules, more conformers than the GPU holds at once
        _case("dg", 20, 500, 18, 48, 2, lbfgs=True, name="dg_20x500"),
        # torsion-preference refinement (ETK) of embedded conformers
        _case("etk", 20, 50, 23, 80, 2, lbfgs=True, name="etk_20x50"),
    ]


def _case(kind, mols, confs, lo, hi, iters, lbfgs=False, precision="mixed", **name):
    return dict(name, kind=kind, mols=mols, confs=confs, lo=lo, hi=hi, iters=iters, lbfgs=lbfgs, precision=precision)


def draw(rng):
    """A case of the listed ranges: sizes log-uniform, atom ranges from narrow to wide."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["nk", "nk", "step", "step", "step", "step", "eg", "multi", "dg", "etk"])
    lbfgs = kind in ("multi", "dg", "etk") or (kind in ("nk", "step") and rng.random() < 0.3)
    precision = "fp64" if kind == "step" and not lbfgs and rng.random() < 0.25 else "mixed"
    lo, hi = 18, rng.choice([30, 48, 75, 110, 150])
    iters = rng.choice([4, 5, 6, 8])
    mols, total = log(1, 30), log(1, {"nk": 300, "step": 4000, "eg": 2000}.get(kind, 1000))
    if kind in ("nk", "step") and lbfgs:
        lo, hi, mols, total = 131, rng.choice([290, 400]), log(1, 14), log(1, 500)
    elif kind == "multi":
        hi, mols, total, iters = rng.choice([40, 64, 87]), log(1, 6), log(1, 200), rng.choice([4, 5, 6])
    elif kind in ("dg", "etk"):
        hi, iters = rng.choice([40, 64, 87]), rng.choice([2, 3]) if kind == "dg" else 2
        total = log(1, 8000 if kind == "dg" and hi == 40 else 600)
    elif precision == "fp64":
        hi, total, iters = min(hi, 110), log(1, 500), rng.choice([8, 11, 15])
    elif kind == "eg":
        iters = 0
    elif total > 1000:
        iters = rng.choice([4, 5])
    return _case(kind, mols, max(1, total // mols), lo, hi, iters, lbfgs, precision)


# ---------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=None)
def _bank(large: bool):
    """Seeded molecules with two clean conformers each, spread over the sizes: 18-150 atoms
    (6-70 heavy atoms), or 131-400 atoms (60-160 heavy atoms, some with a macrocycle)."""
    mols = []
    for i in range(14 if large else 44):
        rng = np.random.default_rng([2024, int(large), i])
        if large:
            h = 60 + (100 * i) // 13
            mol = synth.generate_molecule(rng, h, h, macrocycle=i % 3 == 0, max_atoms=400, ring_density=0.12)
        else:
            h = int(round(7 * (66 / 7.0) ** (i / 43.0)))
            mol = synth.generate_molecule(rng, h, h, max_atoms=150)
        mols.append((mol, synth.embed_conformers(mol, 2, rng, noise=0.0)))
    return mols


@functools.lru_cache(maxsize=None)
def _dg_terms(i: int):
    mol, xyz = _bank(False)[i]
    m = mol.copy()
    m.RemoveAllConformers()
    m.AddConformer(xyz[0])
    dg = synth_dg_params(m)
    return dg, synth_etk_params(m, dg.bounds_mat)


@functools.lru_cache(maxsize=None)
def _mmff_terms(large: bool, i: int, variant: str):
    mol, xyz = _bank(large)[i]
    m = mol.copy()
    m.RemoveAllConformers()
    m.AddConformer(xyz[0])
    return extract_mmff_params(m, mmff_variant=variant)


def _choose(case, seed):
    """Indices into the bank of the case's molecules (spread evenly over its sizes, the same for
    every seed, so that outputs have one shape), and the generator of the seed's coordinates."""
    large, n = case["lo"] > 100, case["mols"]
    fit = [i for i, (m, _) in enumerate(_bank(large)) if case["lo"] <= m.GetNumAtoms() <= case["hi"]]
    fit.sort(key=lambda i: _bank(large)[i][0].GetNumAtoms())
    pick = [fit[((2 * k + 1) * len(fit)) // (2 * n)] for k in range(n)]
    return large, pick, np.random.default_rng([seed, n, case["confs"], case["hi"]])


def _coords(large, i, k, rng):
    xyz = _bank(large)[i][1]
    x = xyz[rng.integers(0, len(xyz), size=k)]
    return x + rng.normal(scale=NOISE, size=x.shape)


def _variant(m):
    return "MMFF94" if m % 2 == 0 else "MMFF94s"


def prepare(case, seed):
    large, pick, rng = _choose(case, seed)
    kind, k = case["kind"], case["confs"]
    if kind in ("dg", "etk"):
        dim = 4 if kind == "dg" else 3
        batch = pack_shared_dg_batch([_dg_terms(i)[0] for i in pick], [k] * len(pick), dim=dim)
        pos = []
        for i in pick:
            x = _coords(False, i, k, rng)
            if kind == "dg":       # a rough embedding: metric-matrix starts are about this far off
                x = np.concatenate([x + rng.normal(scale=0.5, size=x.shape),
                                    rng.normal(scale=0.3, size=x.shape[:2] + (1,))], axis=2)
            pos.append(x.reshape(-1))
        if kind == "etk":
            add_etk_to_batch(batch, [_dg_terms(i)[1] for i in pick])
        dev = (DGDeviceBatch if kind == "dg" else ETKDeviceBatch)(batch)
        start = torch.from_numpy(np.concatenate(pos).astype(np.float32)).cuda()
        prm = dev.params(case["iters"], 1e-4, 1.0 if kind == "dg" else 0.0, 0.1 if kind == "dg" else 0.0)
        return dict(kind=kind, dev=dev, prm=prm, start=start)
    if kind == "multi":
        mols = []
        for i in pick:
            m = _bank(False)[i][0].copy()
            m.RemoveAllConformers()
            for x in _coords(False, i, k, rng):
                m.AddConformer(x)
            mols.append(m)
        return dict(kind=kind, mols=mols, start=[[c.pos.copy() for c in m.GetConformers()] for m in mols],
                    iters=case["iters"])
    params = [_mmff_terms(large, i, _variant(n)) for n, i in enumerate(pick)]
    pos = np.concatenate([_coords(large, i, k, rng).reshape(-1) for i in pick]).astype(np.float32)
    s = dict(kind=kind, counts=[k] * len(pick), iters=case["iters"], lbfgs=case["lbfgs"], pos=pos,
             precision=case["precision"])
    if kind == "nk":
        s["params"] = params
    elif kind == "eg":
        s["m"] = mm.Minimizer(params, s["counts"])
    else:
        s["m"] = mm.BinnedMinimizer(params, s["counts"])
        s["start"] = torch.from_numpy(pos).cuda()
    return s


# ---------------------------------------------------------------- one pass

def run(state):
    kind = state["kind"]
    if kind == "nk":
        return mm.mmff_minimize_nk(state["params"], state["counts"], state["pos"], max_iters=state["iters"],
                                   use_lbfgs=state["lbfgs"])
    if kind == "eg":
        e, g = state["m"].energy_grad(state["pos"], precision=state["precision"])
        return e.astype(np.float32), g       # the terms are 32-bit: the drop-in call's energy type
    if kind == "multi":
        for m, xyz in zip(state["mols"], state["start"]):
            for c, x in zip(m.GetConformers(), xyz):
                c.pos[:] = x
        r = mmff_optimize_metal_multi_mol([(m, None) for m in state["mols"]], max_iters=state["iters"])
        return [[x.energies, x.positions, x.grad_norms, x.per_conf_iters, x.converged] for x in r.mol_results]
    x = state["start"].clone()
    if kind in ("dg", "etk"):
        e, st = state["dev"].minimize_device(x, state["prm"])
        return x, e, st
    e, st, it = state["m"].minimize_device(x, max_iters=state["iters"], precision=state["precision"],
                                           history_m=mm.LBFGS_M if state["lbfgs"] else 0)
    # mixed precision: the terms are 32-bit, so the drop-in call's energy type
    return x, e if state["precision"] == "fp64" else e.float(), st, it


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    """Inputs read once, outputs written once; per iteration one energy and gradient (about 70
    operations a non-bonded pair, 250 a bonded term), one pass over the inverse Hessian (8 operations
    an element) or 8 history pairs.  The first evaluation comes before the first iteration."""
    large = case["lo"] > 100
    sizes = [m.GetNumAtoms() for m, _ in _bank(large) if case["lo"] <= m.GetNumAtoms() <= case["hi"]]
    kind, conf = case["kind"], case["mols"] * case["confs"]
    dim = 4 if kind == "dg" else 3
    nb = fl = 0.0
    for n in sizes:
        nb += 2 * 4 * dim * n + 12 + case["mols"] / conf * (16 * n * n / 2 if kind in ("dg", "etk") else n * (16 * 14 + n / 4))
        pairs, bonded = n * (n - 1) / 2 - 3 * n, 6.2 * n
        ev = 30 * n * n / 2 if kind == "dg" else 250 * 2 * n + 20 * 8 * n if kind == "etk" else 70 * pairs + 250 * bonded
        it = 0 if kind == "eg" else 32 * 3 * n * 2 if case["lbfgs"] else 8 * (3 * n) ** 2
        fl += ev + case["iters"] * (ev + it)
    return {"bytes": nb * conf / len(sizes), "flops": fl * conf / len(sizes)}


# ---------------------------------------------------------------- the same in 64 bits

def _mmff64(p, x):
    """MMFF94 energies (C,) and gradients (C, N, 3) of one molecule's conformers x in 64 bits:
    the seven terms written out over the extracted term lists, gradients by differentiation."""
    def t(a, dt=torch.float64):
        return torch.as_tensor(np.asarray(a), device=x.device).to(dt)

    def at(a):
        return x[:, t(a, torch.int64)]

    def unit(v):
        return v / v.norm(dim=-1, keepdim=True)

    def angle(i, j, k):
        u, v = unit(at(i) - at(j)), unit(at(k) - at(j))
        c = (u * v).sum(-1).clamp(-1, 1)
        return c, torch.rad2deg(torch.acos(c))

    x = x.clone().requires_grad_(True)
    md, deg = 143.9325, math.pi / 180.0
    d = (at(p.bond_idx1) - at(p.bond_idx2)).norm(dim=-1) - t(p.bond_r0)
    e = (0.5 * md * t(p.bond_kb) * d * d * (1 - 2 * d + 7.0 / 3.0 * d * d)).sum(1)
    if len(p.angle_idx1):
        c, a = angle(p.angle_idx1, p.angle_idx2, p.angle_idx3)
        da, ka = a - t(p.angle_theta0), t(p.angle_ka)
        bend = 0.5 * md * deg * deg * ka * da * da * (1 - 0.4 * deg * da)
        e = e + torch.where(t(p.angle_is_linear, torch.bool), md * ka * (1 + c), bend).sum(1)
    sb = torch.zeros_like(e)
    if len(p.strbend_idx1):
        i, j, k = p.strbend_idx1, p.strbend_idx2, p.strbend_idx3
        da = angle(i, j, k)[1] - t(p.strbend_theta0)
        di, dk = (at(i) - at(j)).norm(dim=-1) - t(p.strbend_r0_ij), (at(k) - at(j)).norm(dim=-1) - t(p.strbend_r0_kj)
        sb = (2.51210 * da * (di * t(p.strbend_kba_ijk) + dk * t(p.strbend_kba_kji))).sum(1)
    if len(p.oop_idx1):
        j = at(p.oop_idx2)
        nrm = unit(torch.linalg.cross(unit(j - at(p.oop_idx1)), unit(at(p.oop_idx3) - j), dim=-1))
        chi = torch.rad2deg(torch.asin((unit(at(p.oop_idx4) - j) * nrm).sum(-1).clamp(-1, 1)))
        e = e + (0.5 * md * deg * deg * t(p.oop_koop) * chi * chi).sum(1)
    if len(p.torsion_idx1):
        p1, p2, p3, p4 = (at(v) for v in (p.torsion_idx1, p.torsion_idx2, p.torsion_idx3, p.torsion_idx4))
        n1 = unit(torch.linalg.cross(p1 - p2, p3 - p2, dim=-1))
        n2 = unit(torch.linalg.cross(p2 - p3, p4 - p3, dim=-1))
        c = (n1 * n2).sum(-1)
        e = e + (0.5 * (t(p.torsion_V1) * (1 + c) + t(p.torsion_V2) * (2 - 2 * c * c)
                        + t(p.torsion_V3) * (1 + c * (4 * c * c - 3)))).sum(1)
    if len(p.vdw_idx1):
        q = (at(p.vdw_idx1) - at(p.vdw_idx2)).norm(dim=-1) / t(p.vdw_R_star)
        e = e + (t(p.vdw_eps) * (1.07 / (q + 0.07)) ** 7 * (1.12 / (q ** 7 + 0.12) - 2)).sum(1)
    if len(p.ele_idx1):
        r = (at(p.ele_idx1) - at(p.ele_idx2)).norm(dim=-1) + 0.05
        sc = torch.where(t(p.ele_is_1_4, torch.bool), 0.75, 1.0) * 332.0716 * t(p.ele_charge_term)
        e = e + (sc / r ** (2 if p.ele_diel_model == 2 else 1)).sum(1)
    # the stretch-bend gradient's prefactor is the exact 143.9325 pi / 180, its energy's the rounded one
    (g,) = torch.autograd.grad((e + sb * (md * deg / 2.51210)).sum(), x)
    return (e + sb).detach(), g


def exact(case, seed):
    """Energies and gradients in 64 bits.  A minimisation has no such value: its iterates are decided
    by accept / reject tests that an all-64-bit run meets differently."""
    if case["kind"] != "eg":
        return None
    large, pick, rng = _choose(case, seed)
    es, gs = [], []
    for n, i in enumerate(pick):
        x = torch.from_numpy(_coords(large, i, case["confs"], rng).astype(np.float32)).cuda().double()
        e, g = _mmff64(_mmff_terms(large, i, _variant(n)), x)
        es.append(e)
        gs.append(g.reshape(-1))
    return torch.cat(es), torch.cat(gs)
