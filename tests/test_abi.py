"""CPU: the C-ABI library loads, exports every symbol the header declares, and rejects bad
arguments with an error code before touching a device."""

import ctypes
import os
import re

import pytest

from flashomni_b200 import _native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    names = []
    inc = os.path.join(ROOT, "include")
    for f in sorted(os.listdir(inc)):
        if f.endswith(".h"):
            text = open(os.path.join(inc, f)).read()
            names += re.findall(r"FO_API\s+[\w\s\*]+?\b(fo_\w+)\s*\(", text)
    return names


def test_library_loads_and_exports_every_declared_symbol():
    lib = _native.load()
    declared = _declared_symbols()
    assert len(declared) >= 10
    for name in declared:
        assert hasattr(lib, name), f"{name} is declared in include/ but not exported"
    assert set(declared) == set(_native.SIGNATURES), "ctypes prototypes and header differ"
    assert lib.fo_abi_version() == 2


def test_argument_errors_are_reported_not_raised_as_faults():
    lib = _native.load()
    assert lib.fo_packbits(None, 8, 1, None, None) == _native.FO_ERR_INVALID_ARG
    assert b"null" in lib.fo_last_error()
    assert lib.fo_packbits(None, 0, 1, None, None) == _native.FO_OK
    assert lib.fo_gemm_q(None, None, None, None, 1, 1, 128, 128, 64, 1, 0, 128, 128, 0, 1, None, 0, None, None,
                         0, None) == _native.FO_ERR_INVALID_ARG
    rc = lib.fo_sparse_attn_fwd(*([None] * 5), 1, 128, 128, 1, 1, 128, 128, 128, 128, 128, 128, 128, 128, 128,
                                128, 128, *([None] * 3), 1, None, None, 0, 0, ctypes.c_float(1.0), None, None)
    assert rc == _native.FO_ERR_INVALID_ARG
    assert lib.fo_gemm_workspace_bytes(1, 128, 128, 128, 128) >= 64
    assert lib.fo_mask_compact_scratch_bytes(10, 3) >= 10 * 16


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setenv("FLASHOMNI_B200_LIB", str(tmp_path / "nope.so"))
    monkeypatch.setattr(_native, "_lib", None)
    with pytest.raises(RuntimeError, match="native library not found"):
        _native.load()


class _AttnCall(ctypes.Structure):   # fo_attn_call
    _fields_ = ([(n, ctypes.c_void_p) for n in ("plan", "sparse_info", "sparse_kv_info")]
                + [(n, ctypes.c_int64) for n in ("sparse_info_bytes", "sparse_kv_info_bytes")]
                + [(n, ctypes.c_void_p) for n in ("sparse_info_indptr", "sparse_kv_info_indptr")]
                + [(n, ctypes.c_int32) for n in ("is_full", "lists_ready", "zero_inactive", "dtype")]
                + [(n, ctypes.c_void_p) for n in ("q", "k", "v", "o", "lse")]
                + [(n, ctypes.c_int64) for n in ("total_q", "total_kv")]
                + [(n, ctypes.c_int32) for n in ("num_qo_heads", "num_kv_heads", "head_dim", "fp8_kind")]
                + [(n, ctypes.c_int64) for n in ("q_stride_n", "q_stride_h", "k_stride_n", "k_stride_h", "v_stride_n", "v_stride_h",
                                                 "o_stride_n", "o_stride_h")]
                + [(n, ctypes.c_void_p) for n in ("k16", "v16")] + [("kv_values", ctypes.c_int64), ("partials", ctypes.c_void_p)]
                + [(n, ctypes.c_float) for n in ("sm_scale", "logits_soft_cap")] + [("status", ctypes.c_void_p)])


@pytest.mark.parametrize("small", [True, False])
@pytest.mark.parametrize("bad", [
    dict(num_kv_heads=0), dict(num_kv_heads=-1), dict(num_kv_heads=3), dict(dtype=7), dict(head_dim=96), dict(sm_scale=0.0), dict(logits_soft_cap=-1.0),
    dict(q=None), dict(q=0x1008), dict(status=None), dict(q_stride_n=4), dict(k_stride_h=0), dict(o_stride_n=1024), dict(o_stride_h=256),
    dict(o=0x1008), dict(fp8_kind=2), dict(fp8_kind=0, k16=None), dict(fp8_kind=0, k=0x1004), dict(fp8_kind=1, v16=0x1008)])
def test_attention_call_is_refused_before_anything_is_launched(bad, small):
    """On a machine without a GPU a launch is an error of CUDA, so an argument error says that none was tried (and num_kv_heads = 0
    divides nothing). Nothing is read or written behind the pointers, small numbers that only have to be aligned."""
    n_cand, P = 4 if small else 40000, 0x1000
    plan = (ctypes.c_int64 * 27)(P, P, 1, 4, 0, 4, 128, 128, n_cand, 1, n_cand, n_cand, P, P, P, P, P, P, 1 << 30, 148, 1, 16, n_cand, 0, P, P, P)
    c = _AttnCall(plan=ctypes.addressof(plan), sparse_info=P, sparse_kv_info=P, sparse_info_bytes=1, sparse_kv_info_bytes=1, sparse_info_indptr=P,
                  sparse_kv_info_indptr=P, zero_inactive=1, dtype=1, q=P, k=P, v=P, o=P, total_q=128, total_kv=128, num_qo_heads=4, num_kv_heads=4,
                  head_dim=128, fp8_kind=-1, q_stride_n=512, q_stride_h=128, k_stride_n=512, k_stride_h=128, v_stride_n=512, v_stride_h=128,
                  o_stride_n=512, o_stride_h=128, k16=P, v16=P, kv_values=65536, sm_scale=1.0, status=P)
    for k, v in bad.items():
        setattr(c, k, v)
    lib = _native.load()
    before = lib.fo_launch_count()
    assert lib.fo_attn_run(ctypes.byref(c), None) in (_native.FO_ERR_INVALID_ARG, _native.FO_ERR_UNSUPPORTED)
    assert lib.fo_launch_count() == before
