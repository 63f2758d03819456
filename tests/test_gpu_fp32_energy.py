"""The all-FP32 option sums an energy in one order: its line search compares an energy evaluated
alone with one evaluated with its gradient, and in FP32 two orders differ by more than the decrease
that the search looks for near a minimum.  The same terms in the same order are the same bits.
"""
import numpy as np
import pytest

from mlxmolkit_b200 import mmff_minimize as mm
from mlxmolkit_b200 import synth
from mlxmolkit_b200.mmff_params import extract_mmff_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(1, 2), (3, 5), (6, 9), (14, 18), (27, 34), (60, 70)])
def test_fp32_energy_is_the_same_bits_with_and_without_its_gradient(lo, hi):
    mols = synth.make_molecules(5, 4, 67, lo, hi, workers=1)
    params = [extract_mmff_params(m) for m in mols]
    pos = np.concatenate([np.stack([c.pos for c in m.GetConformers()]).reshape(-1) for m in mols])
    m = mm.Minimizer(params, [4] * len(mols))
    e, _ = m.energy_grad(pos.astype(np.float32), precision="fp32")
    e0, _ = m.energy_grad(pos.astype(np.float32), precision="fp32", want_grad=False)
    np.testing.assert_array_equal(e0, e)
