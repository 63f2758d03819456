"""Algorithmic bytes of a minimisation, the numerator of the HBM roofline."""
from __future__ import annotations

import numpy as np


def term_bytes(p) -> int:
    """Bytes of one molecule's term records in the reference's packed sizes."""
    return (16 * len(p.bond_idx1) + 24 * len(p.angle_idx1) + 32 * len(p.strbend_idx1)
            + 20 * len(p.oop_idx1) + 28 * len(p.torsion_idx1) + 16 * len(p.vdw_idx1)
            + 20 * len(p.ele_idx1))


def algorithmic_bytes(params, conf_mol, iters, evals, history_m: int = 0) -> float:
    """Algorithmic HBM bytes of minimising the conformers ``conf_mol`` (molecule indices): what
    ``iters`` iterations with ``evals`` line-search trials cannot do without.

    The term records and 12 B per atom of coordinates once for the start and once per trial (the
    accepted trial's evaluation is also the next iteration's gradient); 12 B per atom of gradient for
    the start and per iteration; 40 n for the vectors per iteration (n = 3N coordinates).  Between
    iterations, dense BFGS (history_m == 0): nothing while the inverse Hessian is the identity
    (the first pass), 4 n^2 where its first update is written, 8 n^2 in each later pass (4-byte
    elements read and written once).  L-BFGS: the two-loop recursion's reads of the S and Y held so far
    twice (16 n a pair) and the new pair (8 n).  Not counted, though run: the second evaluation of a
    trial that was evaluated without its gradient and then accepted, that of a failed search's
    point, and a restart's passes are taken for ordinary ones.
    """
    conf_mol = np.asarray(conf_mol)
    it, ev = np.asarray(iters, np.float64), np.asarray(evals, np.float64)
    n_atoms = np.array([p.n_atoms for p in params], dtype=np.float64)[conf_mol]
    tb = np.array([term_bytes(p) for p in params], dtype=np.float64)[conf_mol]
    n = 3 * n_atoms
    passes = np.maximum(it - 1, 0)
    if history_m > 0:
        filling = np.minimum(passes, history_m)
        pairs = filling * (filling + 1) / 2 + (passes - filling) * history_m
        quasi = 16 * n * pairs + 8 * n * passes
    else:
        quasi = 4 * n * n * np.maximum(2 * passes - 3, 0)
    return float(np.sum(quasi + (1 + ev) * (tb + 12 * n_atoms) + (1 + it) * 12 * n_atoms + it * 40 * n))
