"""The ctypes mirror of the single-rank argument block has the compiled size."""
import ctypes as C


def test_local_struct_sizes():
    from moonep_b200 import _native
    lib = _native.load()
    assert C.sizeof(_native.MoeLocal) == lib.mep_sizeof_MoeLocal()
