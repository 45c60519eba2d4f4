"""The ctypes mirrors of the single-rank argument blocks have the compiled sizes."""
import ctypes as C


def test_local_struct_sizes():
    from moonep_b200 import _native
    lib = _native.load()
    for cls in (_native.LocalDispatchArgs, _native.LocalCombineArgs, _native.MoeLocal):
        assert C.sizeof(cls) == getattr(lib, f"mep_sizeof_{cls.__name__}")(), cls.__name__
