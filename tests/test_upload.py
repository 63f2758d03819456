"""One upload for many small arrays; a large one goes up from where it is."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mlxmolkit_b200 import mmff_minimize as mm

SMALL, LARGE = 1000, 1 << 20


@pytest.fixture(autouse=True)
def _on_the_host(monkeypatch):
    monkeypatch.setattr(mm, "_torch", lambda: torch)


def _storage(t):
    return t.untyped_storage().data_ptr()


def test_small_arrays_share_one_upload_and_large_ones_do_not_join_it():
    a = [np.arange(SMALL, dtype=np.int32), np.arange(LARGE, dtype=np.float32),
         np.arange(SMALL, dtype=np.float64), np.arange(LARGE, dtype=np.int64)]
    out = mm._upload(a, torch.device("cpu"))
    for x, t in zip(a, out):
        np.testing.assert_array_equal(t.numpy(), x)
        assert t.numpy().dtype == x.dtype
    assert _storage(out[0]) == _storage(out[2])
    # joining a large array costs a host copy of it, more than the copy call it saves
    assert len({_storage(t) for t in out}) == 3
    assert out[0].untyped_storage().nbytes() < 64 * SMALL


@pytest.mark.parametrize("shape", [(0,), (0, 4), (3, 5), (7, 11)])
@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.float32, np.float64])
def test_values_types_and_alignment(shape, dtype):
    rng = np.random.default_rng(3)
    a = [rng.integers(0, 100, size=s).astype(dt) for s, dt in ((shape, dtype), ((5,), np.int32), (shape, dtype))]
    a.append(np.asfortranarray(a[0]))                        # not contiguous in memory order
    a.append(np.repeat(np.arange(9, dtype=dtype), 2)[::2])
    out = mm._upload(a, torch.device("cpu"))
    base = _storage(out[1])
    for x, t in zip(a, out):
        np.testing.assert_array_equal(t.numpy(), np.ascontiguousarray(x).reshape(-1))
        if t.numel():
            assert (t.data_ptr() - base) % 512 == 0


def test_no_arrays_and_empty_arrays():
    assert mm._upload([], torch.device("cpu")) == []
    (t,) = mm._upload([np.zeros(0, np.int64)], torch.device("cpu"))
    assert t.numel() == 0 and t.dtype == torch.int64



@pytest.mark.filterwarnings("error")
def test_read_only_arrays_go_up_too():
    a = [np.zeros(4, np.float32), np.ones(LARGE, np.float32)]
    for x in a:
        x.flags.writeable = False
    out = mm._upload(a, torch.device("cpu"))
    assert out[0].sum() == 0 and out[1].sum() == LARGE
