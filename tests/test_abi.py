"""CPU checks of the C ABI library: it builds, loads, exports every symbol the
public header declares, and refuses to run without an sm_100 GPU (no fallback)."""
import ctypes as C

import pytest

from rest_b200 import _abi, build


@pytest.fixture(scope="module")
def L():
    build.build()
    return C.CDLL(str(_abi.LIB_PATH))


def test_every_declared_symbol_is_exported(L):
    names = _abi.header_symbols()
    assert len(names) >= 25
    missing = [n for n in names if not hasattr(L, n)]
    assert not missing, missing


def test_binding_signatures_cover_the_header():
    assert set(_abi.header_symbols()) <= set(_abi.SIGNATURES)


def test_status_strings(L):
    L.rijk_status_string.restype = C.c_char_p
    assert L.rijk_status_string(0) == b"ok"
    assert b"positive definite" in L.rijk_status_string(3)


def test_energy_contraction_runs_on_host(L):
    import numpy as np

    from oracle import rijk_oracle as O
    from rest_b200 import energy_contraction

    rng = np.random.default_rng(3)
    a = rng.standard_normal(28)
    b = rng.standard_normal(28)
    assert abs(energy_contraction(a, b) - O.par_energy_contraction(a, b)) < 1e-13


def test_context_creation_fails_loudly_without_a_gpu(L):
    import torch

    if torch.cuda.is_available():
        pytest.skip("a GPU is visible")
    from rest_b200 import RIJK, RijkError

    with pytest.raises(RijkError):
        RIJK(0)


def test_int8_launchers_report_operands_without_a_tensor_map(L):
    """A tensor map that cannot be encoded (no driver here, a null operand on a GPU
    box) makes the launchers return false; nothing is enqueued, no error word touched."""
    import subprocess

    names = subprocess.run(["nm", "-D", "--defined-only", str(_abi.LIB_PATH)], capture_output=True, text=True,
                           check=True).stdout.split()
    rank, half = (next(s for s in names if f"4rijk14launch_i8_{w}E" in s) for w in ("rank", "half"))

    class Cols(C.Structure):
        _fields_ = [("nw", C.c_int64 * 2), ("g", C.c_int * 2)]

    class Chunk(C.Structure):
        _fields_ = [("np", C.c_int64), ("B", C.c_void_p), ("digits", C.c_void_p), ("bmax", C.c_void_p),
                    ("X", C.c_void_p * 2), ("wpart", C.c_void_p)]

    class Next(C.Structure):
        _fields_ = [("np", C.c_int64), ("B", C.c_void_p), ("bmax", C.c_void_p), ("shared_max", C.c_bool),
                    ("digits", C.c_void_p)]

    n, ldx, k = C.c_int64(130), C.c_int64(256), C.c_int64(640)
    fn = getattr(L, rank)
    fn.restype = C.c_bool
    err = C.c_int(0)
    assert fn(n, ldx, k, None, None, None, None, 1, 0, None, C.byref(err), None, None) is False
    fn = getattr(L, half)
    fn.restype = C.c_bool
    cols = Cols((C.c_int64 * 2)(200, 0), (C.c_int * 2)(13, 0))  # four column blocks: digits through memory
    assert fn(C.byref(cols), n, C.c_int64(5), ldx, C.c_int64(15 * 1024), C.byref(Chunk(np=4)), C.byref(Next()), None,
              None, None, None, C.byref(err), None, None) is False
    assert err.value == 0


def test_exchange_form_needs_a_context(L):
    assert L.rijk_ctx_set_exchange(None, 0) == 1
