"""The roofline's numerator counts what a run cannot do without, against a walk over its iterations."""
from types import SimpleNamespace

import numpy as np
import pytest

from mlxmolkit_b200.roofline import algorithmic_bytes, term_bytes


def _mol(n):
    fields = ("bond", "angle", "strbend", "oop", "torsion", "vdw", "ele")
    p = {f"{f}_idx1": np.zeros(3 * n + i) for i, f in enumerate(fields)}
    return SimpleNamespace(n_atoms=n, **p)


def _walk(p, iters, trials, hist):
    """Bytes of one run: the start, then per iteration its trials, the gradient of the accepted one, the
    vectors, and -- where another iteration follows -- the inverse Hessian or the history."""
    n, tb = 3 * p.n_atoms, term_bytes(p)
    total = tb + 4 * n + 4 * n                       # the start: terms, coordinates, its gradient
    total += trials * (tb + 4 * n)                   # a trial evaluates the terms once
    for it in range(iters):
        total += 4 * n + 40 * n
        passes = it + 1
        if it + 1 == iters:
            continue                                 # nothing follows that would need the pass
        if hist:
            total += 16 * min(passes, hist) * n + 8 * n
        elif passes == 2:
            total += 4 * n * n                       # made from the identity: written
        elif passes > 2:
            total += 8 * n * n                       # (the first, an identity's, moves nothing)
    return total


@pytest.mark.parametrize("hist", [0, 1, 8])
@pytest.mark.parametrize("iters", [0, 1, 2, 3, 4, 9, 10, 200])
def test_bytes_are_those_of_the_evaluations_and_passes_that_run(hist, iters):
    mols = [_mol(5), _mol(40)]
    conf_mol = [0, 1, 1]
    trials = np.array([iters, iters + iters // 3, 2 * iters])
    want = sum(_walk(mols[m], iters, int(t), hist) for m, t in zip(conf_mol, trials))
    assert algorithmic_bytes(mols, conf_mol, np.full(3, iters), trials, hist) == pytest.approx(want, rel=1e-12)
