"""GPU: nhw_get_field into every kind of host memory.

Page-locked memory is written by the packing kernel itself where it can be: at
addresses that are a multiple of the value's size.  A buffer in a packed record
or at any other odd offset, a registered one, and a buffer that ends with its
allocation must all receive the bytes that pageable memory does, and no byte
beside them.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["ETA", "U", "MASK", "FZ"]      # FP64 2-D, 3-D in the storage type, integers, one more level


def _scenario(precision):
    from nhwave_gb300 import lib, scenarios as S
    p, d, e, u = S.make("tiny_c3", precision=precision, seed=5)
    s = lib.Scenario(p, d, e, u)
    assert s.step() == 0
    return s


def _read(s, field, ptr):
    from nhwave_gb300 import lib
    st = lib.load().nhw_get_field(s._h, field, ctypes.c_void_p(ptr))
    assert st == lib.OK, lib.last_error()


@pytest.mark.parametrize("precision", [0, 1])
def test_any_host_address(precision, gpu_lib):
    torch = pytest.importorskip("torch")
    from nhwave_gb300 import fields as F
    s = _scenario(precision)
    for name in FIELDS:
        f = getattr(F, name)
        want = s.get(f).tobytes()      # pageable
        n = len(want)
        for offset in (0, 1, 2, 4, 8, 12, 64):
            buf = torch.full((n + 128,), 0xA5, dtype=torch.uint8, pin_memory=True)
            assert buf.data_ptr() % 64 == 0
            _read(s, f, buf.data_ptr() + offset)
            got = buf.numpy().tobytes()
            assert got[offset:offset + n] == want, f"{name} at offset {offset}"
            assert set(got[:offset]) | set(got[offset + n:]) == {0xA5}
    s.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_registered_memory(precision, gpu_lib):
    torch = pytest.importorskip("torch")
    from nhwave_gb300 import fields as F
    s = _scenario(precision)
    rt = torch.cuda.cudart()
    for name in FIELDS:
        f = getattr(F, name)
        want = s.get(f)
        out = np.empty(want.nbytes + 8, dtype=np.uint8)
        assert int(rt.cudaHostRegister(out.ctypes.data, out.nbytes, 0)) == 0
        try:
            for offset in (8, 3):      # to the end of the registration, and off the values' size
                _read(s, f, out.ctypes.data + offset)
                assert out[offset:offset + want.nbytes].tobytes() == want.tobytes(), f"{name} at offset {offset}"
        finally:
            assert int(rt.cudaHostUnregister(out.ctypes.data)) == 0
    s.close()


def test_unaligned_views_through_python(gpu_lib):
    torch = pytest.importorskip("torch")
    from nhwave_gb300 import fields as F
    s = _scenario(0)
    want = s.get(F.U)
    record = torch.zeros(want.nbytes + 16, dtype=torch.uint8, pin_memory=True).numpy()
    view = np.frombuffer(record.data, dtype=np.float64, count=want.size, offset=5)
    assert not view.flags["ALIGNED"] and view.flags["C_CONTIGUOUS"]
    assert np.array_equal(s.get(F.U, out=view), want)
    s.close()
