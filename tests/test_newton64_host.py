"""CPU test: the float64 step driver's descriptor has the library's layout."""
import ctypes


def test_descriptor_layout():
    import __graft_entry__
    from dpf_gb300 import _lib
    if not _lib.LIBRARY.exists():
        __graft_entry__.build()
    lib = _lib.load()
    assert lib.dpf_newton64_struct_size() == ctypes.sizeof(_lib.Newton64)
