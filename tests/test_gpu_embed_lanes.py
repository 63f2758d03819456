"""The embedding kernels' block-shared state: repeat runs with several warps per conformer give the
same bits (the L-BFGS rho of the newest pair is read behind the barrier that publishes it), and the
ETK gradient, whose incidence lists a few lanes share, matches the FP64 oracle where the lane count
changes (atoms below, at and above the threads, one atom's list shorter than the lanes).

Tolerances: the gradient's is the ETK suite's, 1e-4 of the largest component (FP32 sums of about
100 terms of up to 1e3 relative to it); repeat runs are compared exactly.
"""
import numpy as np
import pytest

from mlxmolkit_b200 import synth
from mlxmolkit_b200.conformer_metal import DGDeviceBatch
from mlxmolkit_b200.dg_extract import synth_dg_params
from mlxmolkit_b200.etk_extract import synth_etk_params
from mlxmolkit_b200.etk_metal import ETKDeviceBatch
from mlxmolkit_b200.shared_batch import add_etk_to_batch, pack_shared_dg_batch
from oracle import dg

pytestmark = pytest.mark.gpu


def _batch(stage, n_mols, k, lo, hi, seed=41):
    mols = synth.make_molecules(n_mols, 1, seed, lo, hi, workers=1)
    dgp = [synth_dg_params(m) for m in mols]
    dim = 4 if stage == "dg" else 3
    b = pack_shared_dg_batch(dgp, [k] * n_mols, dim=dim)
    rng = np.random.default_rng(seed)
    x = np.concatenate([np.tile(m.GetConformers()[0].pos, (k, 1)) for m in mols])
    x = x + rng.normal(0, 0.3, x.shape)
    if dim == 4:
        x = np.concatenate([x, rng.normal(0, 0.3, (len(x), 1))], axis=1)
    else:
        add_etk_to_batch(b, [synth_etk_params(m, p.bounds_mat) for m, p in zip(mols, dgp)])
    return b, x.astype(np.float32).reshape(-1)


@pytest.mark.parametrize("stage", ["dg", "etk"])
@pytest.mark.parametrize("tpm", [64, 128, 256])
def test_repeat_runs_give_the_same_bits(stage, tpm):
    import torch
    b, x0 = _batch(stage, 6, 200, 18, 30)
    dev = (DGDeviceBatch if stage == "dg" else ETKDeviceBatch)(b)
    prm = dev.params(8, 1e-4, 1.0, 0.1, tpm=tpm)
    start = torch.from_numpy(x0).cuda()
    runs = []
    for _ in range(4):
        x = start.clone()
        e, s = dev.minimize_device(x, prm)
        runs.append((x, e, s))
    for other in runs[1:]:
        for a, c in zip(runs[0], other):
            assert torch.equal(a, c)


@pytest.mark.parametrize("tpm", [32, 64, 128, 256])
@pytest.mark.parametrize("lo,hi", [(1, 3), (10, 16), (26, 40)])
def test_etk_gradient_matches_the_oracle_at_every_lane_count(tpm, lo, hi):
    import torch
    b, x0 = _batch("etk", 4, 2, lo, hi)
    dev = ETKDeviceBatch(b)
    _, g = dev.energy_grad_device(torch.from_numpy(x0).cuda(), dev.params(0, 0.0, 0.0, 0.0, tpm=tpm))
    g = g.cpu().numpy()
    for c in range(b.n_confs_total):
        a0, a1 = int(b.conf_atom_starts[c]) * 3, int(b.conf_atom_starts[c + 1]) * 3
        _, ref = dg.energy_grad(b, x0.astype(np.float64), c, stage="etk")
        assert np.abs(g[a0:a1] - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max()), (c, tpm)
