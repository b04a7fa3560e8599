"""The shared library loads and exports every symbol that include/macseek_b200.h declares (no compute calls)."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__ as ge
    ge.build()
    return ctypes.CDLL(os.path.join(ROOT, "macseek_b200", "libmacseek_b200.so"))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "macseek_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(msb_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(lib):
    names = declared_symbols()
    assert len(names) >= 8
    for n in names:
        assert hasattr(lib, n), n


def test_geometry_and_argument_errors(lib):
    lib.msb_row_bytes.restype = ctypes.c_size_t
    lib.msb_row_bytes.argtypes = [ctypes.c_int, ctypes.c_int64]
    lib.msb_last_error.restype = ctypes.c_char_p
    assert lib.msb_row_bytes(19, 4096) == 800 and lib.msb_row_bytes(16, 4096) == 1056
    assert lib.msb_row_bytes(14, 4096) == 3360 and lib.msb_row_bytes(8, 4096) == 4352
    assert lib.msb_block_elems(20) == 32 and lib.msb_block_elems(30) == 1
    # argument checks happen before any CUDA call
    lib.msb_matvec.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p,
                               ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    assert lib.msb_matvec(19, None, 8, 100, None, None, 0, 1, None) == -1      # cols not a multiple of 256
    assert b"bad shape" in lib.msb_last_error()
    assert lib.msb_matvec(99, None, 8, 256, None, None, 0, 1, None) == -2      # unknown type


def test_moe_prefill_types_are_refused_whatever_the_routing(lib):
    """One expert takes every token, so that its weights would be copied to half first: the types are checked all the same."""
    from macseek_b200 import _lib
    n, D = 2048, 256
    a = _lib.MoePrefillArgsC()
    slots = (_lib.ExpertSlotC * 1)()
    slots[0].gate = slots[0].up = slots[0].down = 4096      # never read: the call ends before any CUDA call
    offs = (ctypes.c_int * 2)(0, n)
    a.dim = a.inter = D
    a.n_tokens, a.n_exp, a.k_per_token, a.has_shared = n, 1, 1, 0
    a.slots, a.offs = slots, offs
    a.tok = a.wt = a.slot_of = a.X = a.Y = a.scratch = 4096
    a.scratch_bytes = 1 << 40
    for gu, dn, sh in ((13, 19, 14), (19, 20, 14), (19, 19, 30), (1, 1, 1), (30, 30, 14)):
        a.t_gate_up, a.t_down, a.t_shared = gu, dn, sh
        assert _lib.lib.msb_moe_prefill(ctypes.byref(a), None) == -2, (gu, dn, sh)
        assert b"unsupported" in _lib.lib.msb_last_error()
