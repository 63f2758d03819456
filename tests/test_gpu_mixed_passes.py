"""The mixed-precision H passes against the FP64 oracle in positions and iteration counts: eight dense
iterations, six of them behind the two identity passes, in every instance (H in shared memory four
rows at a time or in register-cached columns, streamed row pairs with 8 or 16 warps or in
register-cached columns), for odd and even row counts; and runs that restart, over an old H.

Tolerance: 2e-3 A.  The oracle itself, started 1e-6 A off, ends 8 iterations at most 5.3e-5 A away, with
the same iteration counts and statuses (12 starts a batch); an FP32 run is off by about 2e-6 A anew in each
iteration (coordinates of 10 A, gradients to 1e-5 of a step of 0.1 A), so by 8 x 53 x 2e-6 = 9e-4 at the
most.  The oracle with a mistake planted in its passes (a row's product dropped, its update left
out, a neighbour's taken, a column left out, for the last or a middle row) is 4.6e-2 A or more away
in some conformer of each batch.
"""
import numpy as np
import pytest

from mlxmolkit_b200 import mmff_minimize as mm
from mlxmolkit_b200 import synth
from mlxmolkit_b200.mmff_params import extract_mmff_params
from oracle import oracle

pytestmark = pytest.mark.gpu

TOL = 2e-3
SIZES = [(1, 2), (3, 5), (6, 9), (14, 18), (20, 24), (27, 34), (45, 66)]   # heavy atoms: 5 to 138 atoms


def _batch(lo, hi):
    mols = synth.make_molecules(5, 2, 61, lo, hi, workers=1)
    params = [extract_mmff_params(m) for m in mols]
    pos = np.concatenate([np.stack([c.pos for c in m.GetConformers()]).reshape(-1) for m in mols])
    return params, [2] * 5, pos.astype(np.float32)


@pytest.mark.parametrize("lo,hi", SIZES)
@pytest.mark.parametrize("instance", [{}, {"threads": 64}, {"threads": 128}, {"threads": 512},
                                      {"hpass_lean": False}])
def test_mixed_passes_keep_to_the_oracle(lo, hi, instance):
    params, counts, pos = _batch(lo, hi)
    xo, _, so, io = oracle.minimize(params, counts, pos.astype(np.float64), max_iters=8, consts=oracle.TG_CONSTS)
    r = mm.BinnedMinimizer(params, counts).minimize(pos, max_iters=8, **instance)
    assert np.array_equal(r.iters, io) and np.array_equal(r.status, so)
    assert np.abs(r.positions - xo).max() <= TOL


@pytest.mark.parametrize("lo,hi", [s for s in SIZES if s != (27, 34)])   # none of those run on after a restart
def test_mixed_restarts_keep_to_the_oracle(lo, hi):
    """The smallest step allowed is large, so searches fail early and start again from the identity."""
    params, counts, pos = _batch(lo, hi)
    consts = list(oracle.TG_CONSTS)
    consts[2] = 0.02
    x = pos.astype(np.float64)
    xo, _, so, io = oracle.minimize(params, counts, x, max_iters=12, consts=consts, max_restarts=3)
    x0, _, _, _ = oracle.minimize(params, counts, x, max_iters=12, consts=consts)
    assert np.abs(xo - x0).max() > 10 * TOL                  # some runs did restart
    r = mm.BinnedMinimizer(params, counts).minimize(pos, max_iters=12, consts=consts, max_restarts=3)
    assert np.array_equal(r.iters, io) and np.array_equal(r.status, so)
    assert np.abs(r.positions - xo).max() <= TOL
