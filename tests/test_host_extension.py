"""The native functions behind the public ops (csrc/host.cpp) against the Python code that they stand in for: the same
results for the calls they take, None (and so the Python code's own behaviour) for everything else."""

import numpy as np
import pytest
import torch

import flashomni_b200 as fo
from flashomni_b200 import _native
from flashomni_b200 import workloads as wl
from flashomni_b200.gemm import prepare_gemm_o_list, prepare_gemm_q_list
from helpers import masks_to_device


class _Nothing:
    """Stands in for the extension: every function leaves the call to the Python code."""

    def __getattr__(self, name):
        return lambda *a: None


def _both(monkeypatch, call):
    """Result (or exception) of `call` with the extension and without."""
    def run():
        try:
            return call()
        except Exception as e:  # noqa: BLE001 (compared below)
            return type(e), str(e)
    a = run()
    with monkeypatch.context() as m:
        m.setattr(_native, "host", lambda: _Nothing())
        b = run()
    return a, b


def _same(a, b):
    if isinstance(a, torch.Tensor):
        return isinstance(b, torch.Tensor) and a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)
    if isinstance(a, tuple):
        return isinstance(b, tuple) and len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    return a == b


def test_nothing_is_taken_without_cuda_tensors():
    h = _native.host()
    t, i = torch.zeros(4, 128, 128, dtype=torch.bfloat16), torch.zeros(2, dtype=torch.int32)
    for x in (t, None, "x", 3, np.zeros(3)):
        assert h.gemm_q(x, x, 1, None, None, 0, None, None, 128, True, 0, None, None, {}) is None
        assert h.gemm_o(x, x, 1, None, None, 0, None, False, 128, 0, None, None, None, {}) is None
        assert h.segment_packbits(x, i, 1) is None
        assert h.select_blocks(x, 1, 0.1, 0.1, True) is None
    for f in (h.gemm_q, h.gemm_o, h.segment_packbits, h.select_blocks, h.attn_run, h.attn_plan):
        with pytest.raises(TypeError):
            f(1)


def _attn(device, H=4, Hkv=4, D=128, lens=(300, 77), dtype=torch.bfloat16, layout="NHD", kv_dtype=None, seed=3, **plan):
    ip = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=device)
    T = int(ip[-1])
    g = torch.Generator(device=device).manual_seed(seed)
    mk = lambda h: torch.randn(T, h, D, generator=g, device=device).to(dtype)
    q, k, v = mk(H), mk(Hkv), mk(Hkv)
    if kv_dtype is not None:
        k, v = k.to(kv_dtype), v.to(kv_dtype)
    if layout == "HND":
        k, v = k.transpose(0, 1).contiguous(), v.transpose(0, 1).contiguous()
    rng = np.random.default_rng(seed)
    qt = 128 // (H // Hkv)
    qa = [(rng.random((-(-n // qt), Hkv)) < 0.7).astype(np.uint8) for n in lens]
    kk = [(rng.random((-(-n // qt), Hkv, -(-n // 128))) < 0.7).astype(np.uint8) for n in lens]
    m = wl.pack_masks(qa, kk)
    masks = masks_to_device(m, device)
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1 << 20, dtype=torch.uint8, device=device), layout)
    w.plan(ip, ip, H, Hkv, D, q_data_type=dtype, kv_data_type=kv_dtype, **plan)
    return w, q, k, v, masks


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "hnd", "grouped", "d64", "d256", "f16", "fp8", "fp8_hnd", "fp8_strided", "softcap", "scale", "causal"])
def test_attention_forms(cuda_device, monkeypatch, form):
    kw = {"hnd": dict(layout="HND"), "grouped": dict(H=8, Hkv=2), "d64": dict(D=64), "d256": dict(D=256), "f16": dict(dtype=torch.float16),
          "fp8": dict(kv_dtype=torch.float8_e4m3fn), "fp8_hnd": dict(kv_dtype=torch.float8_e5m2, layout="HND"),
          "fp8_strided": dict(kv_dtype=torch.float8_e4m3fn), "softcap": dict(logits_soft_cap=2.0), "scale": dict(sm_scale=0.05),
          "causal": dict(causal=True)}.get(form, {})
    w, q, k, v, masks = _attn(cuda_device, **kw)
    if form == "fp8_strided":
        k = torch.cat([k.view(torch.uint8)] * 2, 2).view(k.dtype)[:, :, :k.shape[2]]
    calls = [
        lambda: w.run(q, k, v, *masks),
        lambda: w.run(q, k, v, *masks, return_lse=True, lse=torch.zeros(q.shape[:2], device=cuda_device)),
        lambda: w.run(q, k, v, *masks, out=torch.ones_like(q)),
        lambda: w.run(q, k, v, is_full=True),
        lambda: w.run_return_lse(q, k, v, is_full=True),
        lambda: w.run(torch.nn.Parameter(q), k, v, *masks),
        lambda: w.run(q, k, v, masks[0], masks[1], masks[2].long(), masks[3].long()),
        lambda: w.run(torch.cat([q, q], 1)[:, :q.shape[1]], k, v, *masks),
        lambda: w.run(q, k, v, *masks, out=torch.zeros(q.shape[0], 2 * q.shape[1], q.shape[2], dtype=q.dtype, device=cuda_device)[:, 1::2]),
    ]
    for i, c in enumerate(calls):
        a, b = _both(monkeypatch, c)
        assert _same(a, b), f"{form}, call {i}: {a if not isinstance(a, torch.Tensor) else ''} {b if not isinstance(b, torch.Tensor) else ''}"
        w.check_status()
    w.prepare_masks(*masks)
    a = w.run(q, k, v, *masks, out=torch.ones_like(q))
    assert _same(a, w.run(q, k, v, *masks, out=torch.ones_like(q)))


@pytest.mark.gpu
def test_attention_refusals(cuda_device, monkeypatch):
    w, q, k, v, masks = _attn(cuda_device)
    si, skv, ip, kp = masks
    bad = [
        lambda: w.run(q[:-1], k, v, *masks), lambda: w.run(q, k[:-1], v, *masks), lambda: w.run(q.half(), k, v, *masks),
        lambda: w.run(q, k.half(), v, *masks), lambda: w.run(q, k, v.half(), *masks), lambda: w.run(q.cpu(), k, v, *masks),
        lambda: w.run(q, k, v), lambda: w.run(q, k, v, si, skv, ip, None), lambda: w.run(q, k, v, si.cpu(), skv, ip, kp),
        lambda: w.run(q, k, v, si.int(), skv, ip, kp), lambda: w.run(q, k, v, si, skv, ip[:-1], kp),
        lambda: w.run(q, k, v, *masks, out=torch.empty_like(q)[:, :-1]), lambda: w.run(q, k, v, *masks, out=torch.empty_like(q).half()),
        lambda: w.run(q, k, v, *masks, lse=torch.zeros(3, device=cuda_device), return_lse=True),
        lambda: w.run(q.transpose(1, 2).contiguous().transpose(1, 2), k, v, *masks),
    ]
    for i, c in enumerate(bad):
        a, b = _both(monkeypatch, c)
        assert isinstance(a, tuple) and isinstance(a[0], type) and issubclass(a[0], Exception), i
        assert a == b, f"call {i}: {a} {b}"


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_forms_and_refusals(cuda_device, monkeypatch, dtype):
    B, M, H, D, hid = 2, 256, 4, 128, 192
    g = torch.Generator(device=cuda_device).manual_seed(1)
    mk = lambda *s: torch.randn(*s, generator=g, device=cuda_device).to(dtype)
    rng = np.random.default_rng(2)
    flags = [(rng.random((M // 128, H)) < 0.6).astype(np.uint8) for _ in range(B)]
    m = wl.pack_masks(flags, [np.ones((M // 128, H, 1), np.uint8) for _ in range(B)])
    si, _, ip, _ = masks_to_device(m, cuda_device)
    x, wq, bias, out = mk(B, M, hid), mk(H * D, hid), mk(H * D), mk(B, M, H * D)
    a_o, wo, cache, b1 = mk(B, M, H * D), mk(256, H * D), mk(B, M, 256), mk(256)
    ql = prepare_gemm_q_list(B, M, H * D, H, si, ip, 0)
    ol = prepare_gemm_o_list(B, M, H * D, H, si, ip, 0, head_dim=D)
    q = lambda **kw: fo.flashomni_gemm(x, wq, H, si, ip, 0, out=out.clone(), **kw)
    o = lambda bias, cached=False, **kw: fo.flashomni_gemm_reduction(a_o, wo, H, si, ip, 0, bias, cached, head_dim=D, **kw)
    calls = [
        lambda: q(), lambda: q(bias=bias), lambda: q(is_full=True), lambda: q(worklist=ql), lambda: q(worklist=ol),
        lambda: fo.flashomni_gemm(x, wq, H, si, ip, 0), lambda: fo.flashomni_gemm(x, wq, H, si, ip.long(), 0, out=out.clone()),
        lambda: fo.flashomni_gemm(x[:, :, 32:], wq, H, si, ip, 0), lambda: fo.flashomni_gemm(x, wq[:-1], H, si, ip, 0),
        lambda: fo.flashomni_gemm(x, wq, H, None, None, 0, out=out.clone()), lambda: fo.flashomni_gemm(x, wq.float(), H, si, ip, 0),
        lambda: fo.flashomni_gemm(x, wq, H, si, ip, 0, out=out[:, :, :-1]), lambda: fo.flashomni_gemm(x.cpu(), wq, H, si, ip, 0),
        lambda: fo.flashomni_gemm(x, wq, H, si[:1], ip, 0, out=out.clone(), head_dim=96),
        lambda: o(cache), lambda: o(None), lambda: o(b1, True), lambda: o(cache, worklist=ol), lambda: o(cache, worklist=ql),
        lambda: o(cache, out=torch.zeros_like(cache)), lambda: o(b1), lambda: o(cache, True), lambda: o(cache.float()),
    ]
    for i, c in enumerate(calls):
        a, b = _both(monkeypatch, c)
        assert _same(a, b), f"call {i}: {a} {b}"


@pytest.mark.gpu
def test_masks_forms_and_refusals(cuda_device, monkeypatch):
    rng = np.random.default_rng(4)
    x = torch.from_numpy((rng.random(5000) < 0.5).astype(np.uint8)).to(cuda_device)
    ip = torch.tensor([0, 7, 7, 1000, 4999], dtype=torch.int32, device=cuda_device)
    p = fo.segment_packbits
    score = torch.randn(2, 3, 20, 20, device=cuda_device)
    s = fo.select_blocks
    calls = [
        lambda: p(x, ip), lambda: p(x, ip, "little"), lambda: p(x.bool(), ip.long(), "little"), lambda: p(x.to(torch.int8), ip),
        lambda: p(x.float(), ip), lambda: p(torch.stack([x, x], 1)[:, 0], ip), lambda: p(x, ip.cpu()), lambda: p(x, ip, "no"),
        lambda: p(x.cpu(), ip), lambda: p(x, ip + 10), lambda: p(x, ip.flip(0)), lambda: p(x[:1000], ip), lambda: p(x.repeat(2000), ip),
        lambda: s(score, 2, 0.2, 0.3), lambda: s(score, 2, 0.2, 0.3, False), lambda: s(score, 2, 1, 0), lambda: s(score.transpose(2, 3), 2, 0.2, 0.3),
        lambda: s(score, 2, torch.tensor([0.1, 0.2]), 0.3), lambda: s(score, 21, 0.2, 0.3), lambda: s(score.half(), 2, 0.2, 0.3),
        lambda: s(score, 2, 1e39, 0.3), lambda: s(score, 2, float("inf"), 0.3), lambda: s(score[:, :, :-1], 2, 0.2, 0.3),
    ]
    for i, c in enumerate(calls):
        a, b = _both(monkeypatch, c)
        assert _same(a, b), f"call {i}: {a} {b}"


@pytest.mark.gpu
@pytest.mark.parametrize("work_in_front", [False, True])
def test_packed_size_is_waited_for_whatever_is_queued(cuda_device, work_in_front):
    """The size is polled for and, behind some milliseconds of other work, waited for with the stream."""
    rng = np.random.default_rng(8)
    x = (rng.random(3000) < 0.5).astype(np.uint8)
    ip = [0, 13, 1500, 3000]
    a = torch.randn(8192, 8192, device=cuda_device)
    for _ in range(3):
        if work_in_front:
            a @ a
        y, new = fo.segment_packbits(torch.from_numpy(x).to(cuda_device), torch.tensor(ip, dtype=torch.int32, device=cuda_device), "little")
        want = np.concatenate([np.packbits(x[i:j], bitorder="little") for i, j in zip(ip, ip[1:])])
        assert np.array_equal(y.cpu().numpy(), want) and new.tolist() == [0, 2, 188, 376]


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["columns", "transposed", "rows", "expanded"])
def test_log_sum_exp_into_a_strided_buffer(cuda_device, monkeypatch, form):
    """The values land where the caller's view says, nothing beside it changes, and an expanded view is refused."""
    w, q, k, v, masks = _attn(cuda_device)
    T, H = q.shape[:2]
    want = torch.full((T, H), 3.0, device=cuda_device)
    w.run(q, k, v, *masks, lse=want, return_lse=True)
    buf = torch.full({"columns": (T, 2 * H), "transposed": (H, T), "rows": (2 * T, H), "expanded": (T, 1)}[form], 3.0, device=cuda_device)
    view = {"columns": lambda b: b[:, 1:H + 1], "transposed": lambda b: b.t(), "rows": lambda b: b[::2], "expanded": lambda b: b.expand(T, H)}[form]
    for return_lse in (True, False):
        def call():
            b = buf.clone()
            r = w.run(q, k, v, *masks, lse=view(b), return_lse=return_lse)
            return (b, *r) if return_lse else (b, r)
        a, b = _both(monkeypatch, call)
        assert _same(a, b)
        if form == "expanded":
            assert a[0] is ValueError
            continue
        full = buf.clone()
        view(full).copy_(want)
        assert torch.equal(a[0], full) and (not return_lse or torch.equal(a[2], want))


@pytest.mark.gpu
@pytest.mark.parametrize("indptr", [[0, 7, 5000], [0, 10_000_000]])
def test_flags_are_packed_once(cuda_device, monkeypatch, indptr):
    """Also where the packed bytes of a few segments are copied out of an allocation for all of x."""
    x = torch.from_numpy((np.random.default_rng(1).random(20_000_000) < 0.5).astype(np.uint8)).to(cuda_device)
    ip = torch.tensor(indptr, dtype=torch.int32, device=cuda_device)
    lib = _native.load()

    def call():
        before = lib.fo_launch_count()
        y, new = fo.segment_packbits(x, ip, "little")
        return y, new, torch.tensor(lib.fo_launch_count() - before), torch.tensor(y.untyped_storage().nbytes())
    a, b = _both(monkeypatch, call)
    assert _same(a, b) and int(a[2]) == 1 and int(a[3]) <= a[0].numel() + (2 << 20)
    want = np.concatenate([np.packbits(x[i:j].cpu().numpy(), bitorder="little") for i, j in zip(indptr, indptr[1:])])
    assert np.array_equal(a[0].cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("missing", [0, 1, 2, 3])
def test_missing_masks_are_refused_after_a_preparation_too(cuda_device, monkeypatch, missing):
    w, q, k, v, masks = _attn(cuda_device)
    some = [None if i == missing else m for i, m in enumerate(masks)]

    def call():
        w.prepare_masks(*masks)
        return w.run(q, k, v, *some)
    a, b = _both(monkeypatch, call)
    assert a == b and a[0] is ValueError and "required unless is_full=True" in a[1]
