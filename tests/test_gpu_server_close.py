"""A closed server holds no page-locked memory: freeing it later would wait for the device to be
idle, in whatever thread the garbage collector happens to run, while another server's worker runs.
"""
import pytest

from mlxmolkit_b200 import synth

pytestmark = pytest.mark.gpu


def test_close_gives_the_mapped_flags_back():
    from mlxmolkit_b200.serve import MMFFServer
    mols = synth.make_molecules(2, 2, 35, 8, 30, workers=1)
    srv = MMFFServer(hbm_budget_bytes=1 << 30)
    for f in [srv.submit(m) for m in mols]:
        f.result(timeout=120)
    bufs = [h.done_buf for cs in srv.classes.values() for h in cs.halves]
    assert bufs and all(b.array is not None and b._host for b in bufs)
    srv.close()
    assert all(b.array is None and not b._host for b in bufs)
    bufs[0].free()                                       # a second call does nothing
