"""How many conformers an SM holds at once.  A launch of one block per conformer that needs a
second wave takes at least a lone conformer's time more.  One conformer more per SM that still
fits shares the SM, at most (k + 1) / k times the time of k; one that does not adds a wave.
The line between the two lies at 1.5: a wave of few conformers takes more than half of a full
one's time, since one conformer's iterations are a chain of latencies.
"""
import ctypes

import numpy as np
import pytest

from mlxmolkit_b200 import _lib
from mlxmolkit_b200 import mmff_minimize as mm
from mlxmolkit_b200 import synth
from mlxmolkit_b200.mmff_metal_optimizer import _MultiMolRun
from mlxmolkit_b200.mmff_params import extract_mmff_params

pytestmark = pytest.mark.gpu


def _fill(per_sm):
    """One molecule of about 30 atoms with per_sm conformers for each SM."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    mol = synth.make_molecules(1, 1, 5, 12, 14, workers=1)[0]
    c = per_sm * sms
    x = np.tile(mol.GetConformers()[0].pos.reshape(-1), c).astype(np.float32)
    return mm.Minimizer([extract_mmff_params(mol)], [c]), x


def _ms(f):
    import torch
    f()
    ts = []
    for _ in range(9):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        ts.append(a.elapsed_time(b))
    return min(ts)


def _fused_sd_ms(per_sm):
    import torch
    m, x = _fill(per_sm)
    L = _lib.load()
    start = torch.from_numpy(x).cuda()
    y = start.clone()
    e = torch.empty(m.confs.n_conf, dtype=torch.float64, device="cuda")
    o = mm.opt_params(60, 0.0, 0, "mixed", mm.TG_CONSTS, mm.MODE_MEGA)
    sd = (ctypes.c_float * 2)(0.1, 1e-3)
    bd, cd = m.batch.desc(), m.confs.desc()

    def f():
        y.copy_(start)
        _lib.check(L.mmffb_fused_sd(ctypes.byref(bd), ctypes.byref(cd), ctypes.byref(o), sd, y.data_ptr(),
                                    e.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "sd")
    return _ms(f)


def test_steepest_descent_holds_four_conformers_an_sm():
    assert _fused_sd_ms(4) < 1.5 * _fused_sd_ms(3)


def _multi_mol_ms(per_sm):
    import torch
    m, x = _fill(per_sm)
    run = _MultiMolRun(m, x, 10, 0.1, 0.3, 1e-4, threads=64)
    start = torch.from_numpy(x).cuda()

    def f():
        run.x.copy_(start)
        run.hcount.zero_()
        run.converged.zero_()
        run.step(_lib.MM_START, 0, 0, 100)
        run.step(_lib.MM_RUN, 30, 30, 100)
    return _ms(f)


def test_multi_mol_with_64_threads_holds_eight_conformers_an_sm():
    assert _multi_mol_ms(8) < 1.5 * _multi_mol_ms(6)
