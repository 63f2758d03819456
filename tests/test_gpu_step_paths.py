"""The optimizer's evaluation and H-pass paths at the sizes where they can go wrong, against the
FP64 oracle: molecules of a few atoms (fewer rows than a group or the warps take), odd and even row
counts of the shared-memory and the streamed pass, the first passes while H is the identity, a
restart back to it, and L-BFGS histories that wrap.

Tolerances.  FP64 kernel against the FP64 oracle after a few iterations: 1e-7 relative, as in the
large fixture's test (rounding of 1e-16 grown by the first, strongly curved steps); mixed: 2e-4, the
same test's (FP32 terms of 1e-7 grown likewise).  An energy with and without its gradient sums the
same FP32 terms in FP64 in two orders: at most some 220 terms a thread and a tree, so within
220 x 1.1e-16 of the sum of the terms' sizes, 1e5 at the most here: 2.5e-9.
"""
import numpy as np
import pytest

from mlxmolkit_b200 import mmff_minimize as mm
from mlxmolkit_b200 import synth
from mlxmolkit_b200.mmff_params import extract_mmff_params
from oracle import oracle

pytestmark = pytest.mark.gpu

SIZES = [(1, 2), (3, 5), (6, 9), (14, 18), (20, 24), (27, 34)]   # heavy atoms: 5 to 76 atoms


def _batch(lo, hi, n_mols=5, k=2, seed=61):
    mols = synth.make_molecules(n_mols, k, seed, lo, hi, workers=1)
    params = [extract_mmff_params(m) for m in mols]
    pos = np.concatenate([np.stack([c.pos for c in m.GetConformers()]).reshape(-1) for m in mols])
    return params, [k] * n_mols, pos.astype(np.float32)


def _close(e, eo, tol):
    assert np.all(np.abs(e - eo) <= tol * np.maximum(1.0, np.abs(eo))), (e, eo)


@pytest.mark.parametrize("lo,hi", SIZES)
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_energy_is_the_same_with_and_without_its_gradient(lo, hi, precision):
    params, counts, pos = _batch(lo, hi)
    m = mm.Minimizer(params, counts)
    e, _ = m.energy_grad(pos, precision=precision)
    e0, _ = m.energy_grad(pos, precision=precision, want_grad=False)
    np.testing.assert_allclose(e0, e, rtol=0, atol=2.5e-9)


@pytest.mark.parametrize("lo,hi", SIZES)
@pytest.mark.parametrize("iters", [1, 3, 8])
def test_first_dense_iterations_follow_the_oracle(lo, hi, iters):
    params, counts, pos = _batch(lo, hi)
    m = mm.BinnedMinimizer(params, counts)
    _, eo, _, io = oracle.minimize(params, counts, pos.astype(np.float64), max_iters=iters,
                                   consts=oracle.TG_CONSTS)
    r64 = m.minimize(pos, max_iters=iters, precision="fp64")
    _close(r64.energies, eo, 1e-7)
    assert np.array_equal(r64.iters, io)
    _close(m.minimize(pos, max_iters=iters).energies, eo, 2e-4)


@pytest.mark.parametrize("hist", [1, 2, 5, 16])
def test_lbfgs_histories_wrap_as_the_oracle_s(hist):
    params, counts, pos = _batch(8, 20)
    m = mm.BinnedMinimizer(params, counts)
    _, eo, _, io = oracle.minimize(params, counts, pos.astype(np.float64), max_iters=9, history_m=hist,
                                   consts=oracle.TG_CONSTS)
    r64 = m.minimize(pos, max_iters=9, history_m=hist, precision="fp64")
    _close(r64.energies, eo, 1e-7)
    assert np.array_equal(r64.iters, io)
    _close(m.minimize(pos, max_iters=9, history_m=hist).energies, eo, 2e-4)


@pytest.mark.parametrize("lo,hi", [(6, 9), (14, 18), (27, 34)])
def test_a_restart_goes_back_to_the_identity(lo, hi):
    """A line search that may not go below a large step fails early; with restarts the run goes on
    from steepest descent, as the oracle's does."""
    params, counts, pos = _batch(lo, hi)
    consts = list(oracle.TG_CONSTS)
    consts[2] = 0.02                                        # MOVETOL: the smallest relative step
    m = mm.BinnedMinimizer(params, counts)
    x = pos.astype(np.float64)
    _, eo, so, io = oracle.minimize(params, counts, x, max_iters=12, consts=consts, max_restarts=3)
    _, _, s0, i0 = oracle.minimize(params, counts, x, max_iters=12, consts=consts)
    assert np.any((io != i0) | (so != s0))                  # some runs did restart
    r = m.minimize(pos, max_iters=12, consts=consts, max_restarts=3, precision="fp64")
    _close(r.energies, eo, 1e-7)
    assert np.array_equal(r.iters, io) and np.array_equal(r.status, so)
