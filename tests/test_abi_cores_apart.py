"""TTG_CORES_APART marks an input's layout; it is not ownership."""
import ctypes as C

import numpy as np


def test_free_leaves_an_input_alone(ttg):
    L = ttg.lib()
    src = ttg._In([np.full((1, 2, 3), 2.0), np.full((3, 4, 1), 5.0)])
    before = bytes(src.t)
    assert src.t.owned == ttg._CORES_APART
    # Buffers of the C allocator, so that a library that takes them for its
    # own frees them without harm to this process.
    libc = C.CDLL(None)
    libc.malloc.restype, libc.malloc.argtypes = C.c_void_p, [C.c_size_t]
    libc.free.restype, libc.free.argtypes = None, [C.c_void_p]
    t = ttg._Tensor.from_buffer_copy(before)
    held = {}
    for name, typ in (("ranks", C.c_int32), ("rows", C.c_int32), ("offsets", C.c_int64),
                      ("data", C.c_double)):
        held[name] = libc.malloc(256)
        setattr(t, name, C.cast(C.c_void_p(held[name]), C.POINTER(typ)))
    image = bytes(t)
    L.ttg_free(C.byref(t))
    assert bytes(t) == image
    for p in held.values():
        libc.free(p)
    # an output is still freed
    out = ttg._Tensor()
    modes = (C.c_int32 * 2)(2, 3)
    assert L.ttg_host_ones(2, modes, C.byref(out)) == 0 and out.owned
    L.ttg_free(C.byref(out))
    assert not out.owned and not out.data
