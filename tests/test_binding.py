"""The native call path of the Python binding (host/pycall.cpp): it covers every status-returning function of the headers,
reports errors like the ctypes path, and hands argument forms it does not convert to ctypes."""
import ctypes as C

import pytest


def test_every_status_function_has_a_native_entry(talos):
    status = {n for n, (res, _) in talos.lib.protos.items() if res is C.c_int32 and n not in talos._NOT_STATUS}
    native = {n for n in dir(talos.lib.native) if n.startswith("talos_")}
    assert native == status


def test_errors_and_argument_forms(talos):
    lib = talos.lib
    with pytest.raises(talos.TalosError) as e:
        lib.talos_gemm(None, 0, 0, 1, 1, 1, None, 1, None, 1, None, 1, 0, None)
    assert e.value.status == talos.ERR_ARG and "null context" in str(e.value)
    out = (C.c_float * 4)()                                              # an array: converted by ctypes
    lib.talos_rng_uniform_host(7, -1, 1.0, out, 4)                        # an int where a float is declared
    again = (C.c_float * 4)()
    lib.talos_rng_uniform_host(7, -1.0, 1.0, C.addressof(again), 4)       # the native path
    assert list(out) == list(again) and any(v != 0.0 for v in out)
    lib.talos_rng_uniform_host(7, -1.0, 1.0, C.c_void_p(C.addressof(out)), 4)
    assert list(out) == list(again)
    with pytest.raises(TypeError):
        lib.talos_rng_uniform_host(7, -1.0)                               # too few arguments
    with pytest.raises(C.ArgumentError):
        lib.talos_rng_uniform_host("seed", -1.0, 1.0, None, 0)
