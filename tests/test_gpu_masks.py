"""GPU: packbits / segment_packbits / mask compaction / GEMM work lists, bit-exact against the oracle."""

import numpy as np
import pytest
import torch

import flashomni_b200 as fo
from flashomni_b200 import _native, workloads as wl
from oracle import masks as om
from helpers import dev, masks_to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["big", "little"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 64, 1000, 4097, 1 << 20])
def test_packbits_matches_numpy(cuda_device, order, n):
    rng = np.random.default_rng(n)
    x = rng.integers(0, 2, n).astype(np.uint8)
    y = fo.packbits(dev(x, cuda_device).bool(), bitorder=order)
    assert np.array_equal(y.cpu().numpy(), om.packbits(x, order))


def test_packbits_reference_docstring_kat(cuda_device):
    x = torch.tensor([1, 0, 1, 1, 0, 0, 1, 1], dtype=torch.bool, device=cuda_device)
    assert fo.packbits(x).tolist() == [0b10110011]
    xs = torch.tensor([1, 0, 1, 1, 0, 0, 1, 1, 1, 0, 1], dtype=torch.bool, device=cuda_device)
    y, ip = fo.segment_packbits(xs, torch.tensor([0, 4, 7, 11], device=cuda_device), bitorder="big")
    assert y.tolist() == [0b10110000, 0b100000, 0b11010000]
    assert ip.tolist() == [0, 1, 2, 3]


@pytest.mark.parametrize("order", ["big", "little"])
def test_segment_packbits_ragged(cuda_device, order):
    rng = np.random.default_rng(1)
    lens = [0, 1, 7, 8, 9, 63, 64, 65, 1000, 0, 31104, 5]
    indptr = np.concatenate([[0], np.cumsum(lens)])
    x = rng.integers(0, 2, int(indptr[-1])).astype(np.uint8)
    y, ip = fo.segment_packbits(dev(x, cuda_device), dev(indptr, cuda_device), bitorder=order)
    ry, rip = om.segment_packbits(x, indptr, order)
    assert np.array_equal(ip.cpu().numpy(), rip)
    assert np.array_equal(y.cpu().numpy(), ry)
    # uint8 input whose non-zero values are not 1, and int32 indptr
    x2 = x * 200
    y2, _ = fo.segment_packbits(dev(x2, cuda_device), dev(indptr.astype(np.int32), cuda_device), bitorder=order)
    assert np.array_equal(y2.cpu().numpy(), ry)


# one empty segment; an indptr that starts past zero; the most segments of the one-launch path and one more;
# more inputs than the segments cover
@pytest.mark.parametrize("lens,start,extra", [([0], 0, 5), ([3, 40], 17, 0), ([13] * 1024, 0, 3), ([13] * 1025, 0, 0),
                                              ([0, 31, 32, 33, 0, 257], 1, 300), ([70001], 0, 0)])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("indptr_device", ["cuda", "cpu"])
def test_segment_packbits_sizes(cuda_device, lens, start, extra, dtype, indptr_device):
    indptr = start + np.concatenate([[0], np.cumsum(lens)])
    rng = np.random.default_rng(len(lens) + start)
    x = rng.integers(0, 2, int(indptr[-1]) + extra).astype(np.uint8)
    ip = torch.from_numpy(indptr).to(dtype)
    y, nip = fo.segment_packbits(dev(x, cuda_device), ip.to(cuda_device) if indptr_device == "cuda" else ip, bitorder="little")
    ry, rip = om.segment_packbits(x[start:], indptr - start, "little")
    assert nip.dtype == torch.int32 and nip.device == y.device and y.is_contiguous()
    assert np.array_equal(nip.cpu().numpy(), rip) and np.array_equal(y.cpu().numpy(), ry)


# a start and an end past the values, an end of few more, a negative start; on the one-launch path and past its segment count
@pytest.mark.parametrize("indptr", [[1000000, 1000100], [0, 50, 107], [-8, 100], [0] * 1100 + [101]])
@pytest.mark.parametrize("indptr_device", ["cuda", "cpu"])
def test_segments_outside_the_input_are_refused(cuda_device, indptr, indptr_device):
    x = torch.ones(100, dtype=torch.uint8, device=cuda_device)
    with pytest.raises(ValueError):
        fo.segment_packbits(x, torch.tensor(indptr, dtype=torch.int32, device=indptr_device))
    torch.cuda.synchronize()


def test_packed_bytes_of_a_few_segments_hold_no_memory_for_the_rest(cuda_device):
    x = torch.ones(1 << 24, dtype=torch.uint8, device=cuda_device)
    y, _ = fo.segment_packbits(x, torch.tensor([5, 5 + 16], dtype=torch.int32, device=cuda_device))
    assert y.tolist() == [255, 255] and y.untyped_storage().nbytes() <= 1 << 20


def test_segments_that_read_nothing_may_lie_anywhere(cuda_device):
    x = torch.ones(100, dtype=torch.uint8, device=cuda_device)
    for indptr, want in (([500, 500], []), ([96, 100, 97, 100], [240, 224])):   # (a step back of less than 8 packs nothing)
        y, ip = fo.segment_packbits(x, torch.tensor(indptr, dtype=torch.int32, device=cuda_device))
        assert y.tolist() == want and int(ip[-1]) == len(want)


def _compact_gpu(device, m, qo, kv, H, head_begin=0, head_count=None, is_full=False):
    hc = H - head_begin if head_count is None else head_count
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1024, dtype=torch.uint8, device=device))
    w.plan(dev(qo.astype(np.int32), device), dev(kv.astype(np.int32), device), hc, hc, 128, q_data_type=torch.bfloat16,
           mask_num_heads=H, mask_head_begin=head_begin)
    lib = _native.load()
    si, skv, ip, kp = masks_to_device(m, device)
    ws = w._ws
    rc = lib.fo_mask_compact(_native.ptr(si), si.numel(), _native.ptr(skv), skv.numel(), _native.ptr(ip), _native.ptr(kp),
                             _native.ptr(w._qo_indptr_buf), _native.ptr(w._kv_indptr_buf), len(qo) - 1, H, head_begin, hc,
                             128, 128, 1 if is_full else 0, w._n_cand, w._max_nkv, max(w._n_cand, 1), max(w._max_kept, 1),
                             _native.ptr(ws["items"]), _native.ptr(ws["kv_ptr"]), _native.ptr(ws["kv_idx"]),
                             _native.ptr(ws["order"]), _native.ptr(ws["counters"]), _native.ptr(ws["scratch"]),
                             w._scratch_bytes, torch.cuda.current_stream(device).cuda_stream)
    _native.check(rc, "fo_mask_compact")
    torch.cuda.synchronize()
    return w.work_lists()


def _assert_lists_equal(got, ref):
    assert got["status"] == 0
    assert got["n_items"] == len(ref["items"])
    assert got["total_kept"] == len(ref["kv_idx"])
    for k in ("items", "kv_indptr", "kv_idx", "order"):
        assert np.array_equal(got[k], ref[k]), k


@pytest.mark.parametrize("case", ["flux_b1", "flux_b2", "ragged", "window", "full", "sparse_extreme"])
def test_attention_compaction_bit_exact(cuda_device, case):
    H = 24
    if case == "flux_b1":
        m = wl.flux_masks(1, H, 36, 36, 0.5, seed=11); qo = kv = np.array([0, 4608])
        args = {}
    elif case == "flux_b2":
        m = wl.flux_masks(2, H, 36, 36, 0.5, seed=12); qo = kv = np.array([0, 4608, 9216])
        args = {}
    elif case == "ragged":
        H = 5
        lens_q, lens_kv = [300, 128, 1000, 77], [256, 700, 1300, 129]
        qo = np.concatenate([[0], np.cumsum(lens_q)]); kv = np.concatenate([[0], np.cumsum(lens_kv)])
        rng = np.random.default_rng(2)
        qa = [(rng.random((-(-a // 128), H)) < 0.6).astype(np.uint8) for a in lens_q]
        kk = [(rng.random((-(-a // 128), H, -(-b // 128))) < 0.5).astype(np.uint8) for a, b in zip(lens_q, lens_kv)]
        m = wl.pack_masks(qa, kk); args = {}
    elif case == "window":
        m = wl.flux_masks(2, H, 36, 36, 0.5, seed=13); qo = kv = np.array([0, 4608, 9216])
        args = {"head_begin": 6, "head_count": 3}
    elif case == "full":
        m = wl.flux_masks(1, H, 9, 11, 0.5, seed=14); qo = np.array([0, 9 * 128]); kv = np.array([0, 11 * 128])
        args = {"is_full": True}
    else:  # nothing active in most rows, long kv rows (more than 32 words per row)
        H = 3
        rng = np.random.default_rng(3)
        qa = [(rng.random((7, H)) < 0.2).astype(np.uint8)]
        kk = [(rng.random((7, H, 1100)) < 0.03).astype(np.uint8)]
        m = wl.pack_masks(qa, kk); qo = np.array([0, 7 * 128]); kv = np.array([0, 1100 * 128]); args = {}
    got = _compact_gpu(cuda_device, m, qo, kv, H, **args)
    ref = om.compact(m.sparse_info, m.sparse_kv_info, m.info_indptr, m.kv_info_indptr, qo, kv, H, 128, 128, **args)
    _assert_lists_equal(got, ref)


def test_attention_compaction_random_ragged_cases(cuda_device):
    """Forty seeded cases: ragged request lengths, densities from empty to full, head windows."""
    rng = np.random.default_rng(2025)
    for _ in range(40):
        B, H = int(rng.integers(1, 5)), int(rng.integers(1, 7))
        lens_q = [int(rng.integers(1, 1500)) for _ in range(B)]
        lens_kv = [int(rng.integers(1, 6000)) for _ in range(B)]
        dq, dk = float(rng.choice([0.0, 0.3, 0.8, 1.0])), float(rng.choice([0.0, 0.05, 0.5, 1.0]))
        qa = [(rng.random((-(-a // 128), H)) < dq).astype(np.uint8) for a in lens_q]
        kk = [(rng.random((-(-a // 128), H, -(-b // 128))) < dk).astype(np.uint8) for a, b in zip(lens_q, lens_kv)]
        hb = int(rng.integers(0, H))
        hc = int(rng.integers(1, H - hb + 1))
        qo = np.concatenate([[0], np.cumsum(lens_q)]); kv = np.concatenate([[0], np.cumsum(lens_kv)])
        m = wl.pack_masks(qa, kk)
        got = _compact_gpu(cuda_device, m, qo, kv, H, head_begin=hb, head_count=hc)
        ref = om.compact(m.sparse_info, m.sparse_kv_info, m.info_indptr, m.kv_info_indptr, qo, kv, H, 128, 128, hb, hc)
        _assert_lists_equal(got, ref)


# (request lengths q, kv, mask heads, head window, density): one candidate; a remainder of the 16 candidates per CTA;
# ragged with a request of no rows; a window; kv rows of more than one 64-bit word; more (group, length) buckets than
# lengths are ordered for (single heads, q-blocks ascending); the largest candidate count of one launch and the first one past
# it, for a few requests (2560), for many and with all blocks (4096)
@pytest.mark.parametrize("lens_q,lens_kv,H,hb,hc,density", [
    ([100], [77], 1, 0, 1, 1.0), ([17 * 128], [300], 1, 0, 1, 0.5), ([300, 0, 1000, 77], [256, 128, 1300, 129], 5, 0, 5, 0.4),
    ([4608, 4608], [4608, 4608], 24, 6, 3, 0.5), ([700], [64 * 128 + 1], 3, 0, 3, 0.3), ([512], [102400], 40, 0, 40, 0.4),
    ([128 * 128], [512], 32, 0, 32, 0.5), ([128 * 128 + 1], [512], 32, 0, 32, 0.5), ([80 * 128], [512], 32, 0, 32, 0.5),
    ([80 * 128 + 1], [512], 32, 0, 32, 0.5), ([2048] * 16, [512] * 16, 16, 0, 16, 0.5), ([2048] * 15 + [2049], [512] * 16, 16, 0, 16, 0.5)])
@pytest.mark.parametrize("is_full", [False, True])
def test_attention_lists_in_one_call_match_the_oracle(cuda_device, lens_q, lens_kv, H, hb, hc, density, is_full):
    rng = np.random.default_rng(len(lens_q) * 100 + H)
    qa = [(rng.random((-(-a // 128), H)) < density).astype(np.uint8) for a in lens_q]
    kk = [(rng.random((-(-a // 128), H, -(-b // 128))) < density).astype(np.uint8) for a, b in zip(lens_q, lens_kv)]
    qo = np.concatenate([[0], np.cumsum(lens_q)]); kv = np.concatenate([[0], np.cumsum(lens_kv)])
    m = wl.pack_masks(qa, kk)
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1024, dtype=torch.uint8, device=cuda_device))
    w.plan(dev(qo.astype(np.int32), cuda_device), dev(kv.astype(np.int32), cuda_device), hc, hc, 128,
           q_data_type=torch.bfloat16, mask_num_heads=H, mask_head_begin=hb)
    w.build_work_lists(*masks_to_device(m, cuda_device), is_full=is_full)
    torch.cuda.synchronize()
    got = w.work_lists()
    ref = om.compact(m.sparse_info, m.sparse_kv_info, m.info_indptr, m.kv_info_indptr, qo, kv, H, 128, 128, hb, hc,
                     is_full=is_full)
    _assert_lists_equal(got, ref)
    assert got["n_units"] == got["n_items"] and got["unit_status"] == 0
    for pos, it in enumerate(got["order"]):   # one record per item, in processing order
        b, h, qb, n = (int(x) for x in got["items"][it])
        ends = n > 0 and lens_kv[b] % 128 != 0 and int(got["kv_idx"][got["kv_indptr"][it] + n - 1]) == lens_kv[b] // 128
        valid = min(128, lens_q[b] - 128 * qb) | ((lens_kv[b] % 128) << 16 if ends else 0)
        want = [n, int(got["kv_indptr"][it]), h | b << 16, int(qo[b]) + 128 * qb, valid, int(kv[b]),
                128 * qb + lens_kv[b] - lens_q[b], -65535]
        assert got["units"][pos].tolist() == want


@pytest.mark.parametrize("H,group,D,lens", [(2, 1, 64, [300]), (4, 2, 128, [65, 700]), (24, 1, 128, [128 * 180])])
def test_allocated_output_is_zero_in_skipped_blocks(cuda_device, H, group, D, lens):
    """An output that run() allocates itself, over memory that held other values; the last case is past the one-launch
    builder's size."""
    rng = np.random.default_rng(3)
    toks = 128 // group
    qa = [(rng.random((-(-n // toks), H)) < 0.5).astype(np.uint8) for n in lens]
    kk = [(rng.random((-(-n // toks), H, -(-n // 128))) < 0.1).astype(np.uint8) for n in lens]
    m = wl.pack_masks(qa, kk)
    ip = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=cuda_device)
    total = sum(lens)
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1024, dtype=torch.uint8, device=cuda_device))
    w.plan(ip, ip, H * group, H, D, q_data_type=torch.bfloat16)
    g = torch.Generator(device=cuda_device).manual_seed(1)
    q = torch.randn(total, H * group, D, generator=g, device=cuda_device).bfloat16()
    k, v = (torch.randn(total, H, D, generator=g, device=cuda_device).bfloat16() for _ in range(2))
    masks = masks_to_device(m, cuda_device)
    junk = torch.full_like(q, 7.0)
    del junk
    got = w.run(q, k, v, *masks)
    want = w.run(q, k, v, *masks, out=torch.zeros_like(q))
    w.check_status()
    on = torch.cat([dev(a, cuda_device).bool().repeat_interleave(toks, 0)[:n] for a, n in zip(qa, lens)])
    off = ~on.repeat_interleave(group, 1)
    assert not got[off].any() and not want[off].any()
    # the order in which a q-block's row sums are added depends on the CTA that draws it: one bf16 step of values below 4
    assert (got.float() - want.float()).abs().max() <= 2 ** -6


def test_allocated_output_is_zero_where_the_lists_do_not_fit(cuda_device):
    """Lists that outgrow their room are reported and not run; the output is zeros, as ever."""
    H, D, S = 2, 64, 384
    ip = torch.tensor([0, S], dtype=torch.int32, device=cuda_device)
    masks = masks_to_device(wl.pack_masks([np.ones((3, H), np.uint8)], [np.ones((3, H, 3), np.uint8)]), cuda_device)
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1024, dtype=torch.uint8, device=cuda_device))
    w.plan(ip, ip, H, H, D, q_data_type=torch.bfloat16)
    args = list(w._list_args)
    assert args[9] == 3 * 3 * H   # room for the kept kv-blocks
    args[9] -= 1
    w._list_args = tuple(args)
    q = torch.randn(S, H, D, device=cuda_device).bfloat16()
    junk = torch.full_like(q, 7.0)
    del junk
    got = w.run(q, q, q, *masks)
    assert not got.any()
    with pytest.raises(RuntimeError):
        w.check_status()


def test_captured_output_is_zero_past_the_rows_of_a_later_plan(cuda_device):
    """Graph mode: the captured call is replayed with fewer rows than it was captured with; the rest of its output is zeros."""
    H, D = 2, 128
    sizes = [torch.tensor([0, n], dtype=torch.int32, device=cuda_device) for n in (300, 200)]
    bufs = [sizes[0].clone() for _ in range(2)]
    # every bit set, whatever the block counts
    masks = masks_to_device(wl.pack_masks([np.ones((3, H), np.uint8)], [np.ones((3, H, 3), np.uint8)]), cuda_device)
    masks[0].fill_(255), masks[1].fill_(255)
    q = torch.randn(300, H, D, device=cuda_device).bfloat16()
    new = lambda *a: fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1024, dtype=torch.uint8, device=cuda_device), "NHD", *a)
    w = new(True, *bufs)
    w.plan(sizes[0], sizes[0], H, H, D, q_data_type=torch.bfloat16)
    side = torch.cuda.Stream(cuda_device)
    side.wait_stream(torch.cuda.current_stream(cuda_device))
    with torch.cuda.stream(side):
        w.run(q, q, q, *masks)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        out = w.run(q, q, q, *masks)
    w.plan(sizes[1], sizes[1], H, H, D, q_data_type=torch.bfloat16)
    out.fill_(7.0)
    g.replay()
    ref = new()
    ref.plan(sizes[1], sizes[1], H, H, D, q_data_type=torch.bfloat16)
    want = ref.run(q[:200], q[:200], q[:200], *masks)
    torch.cuda.synchronize()
    assert torch.equal(out[:200], want) and not out[200:].any()


def test_gemm_worklists_bit_exact(cuda_device):
    lib = _native.load()
    B, H, nq = 2, 24, 36
    m = wl.flux_masks(B, H, nq, nq, 0.5, seed=21)
    si, _, ip, _ = masks_to_device(m, cuda_device)
    M, N, K = nq * 128, H * 128, H * 128
    nbytes = lib.fo_gemm_workspace_bytes(B, M, N, K, 128)
    ws = torch.zeros(nbytes, dtype=torch.uint8, device=cuda_device)
    st = torch.cuda.current_stream(cuda_device).cuda_stream
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    for ntt, m_rows in ((0, M), (512, M - 512)):
        # all heads, and head windows as a rank of 2 / 8 has them (few records: the rule cuts more of them)
        for hb, hc in ((0, H), (12, 12), (21, 3)):
            rc = lib.fo_gemm_q_worklist(B, m_rows, hc * 128, H, hb, 128, 128, ntt, 0, _native.ptr(si), si.numel(),
                                        _native.ptr(ip), _native.ptr(ws), ws.numel(), st)
            _native.check(rc, "fo_gemm_q_worklist")
            w = ws.view(torch.int32).cpu().numpy()
            ref = om.gemm_q_tile_pairs(m.sparse_info, m.info_indptr, B, m_rows, hc * 128, H, 128, ntt, head_begin=hb,
                                       head_dim=128, num_ctas=sms)
            assert w[0] == len(ref) and w[2] == 0
            assert w[1] == len(om.gemm_q_tiles(m.sparse_info, m.info_indptr, B, m_rows, hc * 128, H, 128, ntt,
                                               head_begin=hb, head_dim=128))
            assert w[3] == int((ref[:, 3] >= 0).sum())
            assert np.array_equal(w[8:8 + 4 * len(ref)].reshape(-1, 4), ref)
        for cache in (0, 1):
            rc = lib.fo_gemm_o_worklist(B, m_rows, K, H, 0, 128, 128, ntt, cache, _native.ptr(si), si.numel(),
                                        _native.ptr(ip), _native.ptr(ws), ws.numel(), st)
            _native.check(rc, "fo_gemm_o_worklist")
            w = ws.view(torch.int32).cpu().numpy()
            rip, rheads, rorder = om.gemm_o_rows(m.sparse_info, m.info_indptr, B, m_rows, K, H, 128, ntt, bool(cache))
            R = B * m_rows // 128
            assert w[0] == R and w[1] == len(rheads)
            assert np.array_equal(w[8:8 + R + 1], rip)
            assert np.array_equal(w[8 + R + 1:8 + R + 1 + len(rheads)], rheads)
            o0 = 8 + R + 1 + R * H
            assert np.array_equal(w[o0:o0 + R], rorder)


@pytest.mark.parametrize("rows", [1, 31, 33, 1024, 1025])   # one row block per thread of the list kernels, and one more
def test_gemm_worklists_row_counts(cuda_device, rows):
    lib = _native.load()
    H, rng = 5, np.random.default_rng(rows)
    m = wl.pack_masks([(rng.random((rows, H)) < 0.5).astype(np.uint8)], [np.zeros((rows, H, 1), np.uint8)])
    si, _, ip, _ = masks_to_device(m, cuda_device)
    ws = torch.zeros(lib.fo_gemm_workspace_bytes(1, rows * 128, H * 128, H * 128, 128), dtype=torch.uint8, device=cuda_device)
    st = torch.cuda.current_stream(cuda_device).cuda_stream
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    mask = (_native.ptr(si), si.numel(), _native.ptr(ip), _native.ptr(ws), ws.numel(), st)
    _native.check(lib.fo_gemm_q_worklist(1, rows * 128, H * 128, H, 0, 128, 128, 0, 0, *mask), "fo_gemm_q_worklist")
    w = ws.view(torch.int32).cpu().numpy()
    ref = om.gemm_q_tile_pairs(m.sparse_info, m.info_indptr, 1, rows * 128, H * 128, H, 128, 0, head_dim=128, num_ctas=sms)
    assert w[0] == len(ref) and w[2] == 0 and np.array_equal(w[8:8 + 4 * len(ref)].reshape(-1, 4), ref)
    for cache in (0, 1):
        _native.check(lib.fo_gemm_o_worklist(1, rows * 128, H * 128, H, 0, 128, 128, 0, cache, *mask), "fo_gemm_o_worklist")
        w = ws.view(torch.int32).cpu().numpy()
        rip, rheads, rorder = om.gemm_o_rows(m.sparse_info, m.info_indptr, 1, rows * 128, H * 128, H, 128, 0, bool(cache))
        o0 = 8 + rows + 1 + rows * H
        assert np.array_equal(w[8:8 + rows + 1], rip) and np.array_equal(w[8 + rows + 1:8 + rows + 1 + len(rheads)], rheads)
        assert np.array_equal(w[o0:o0 + rows], rorder)


# smallest; the image layer with a head window; past the one-launch size
@pytest.mark.parametrize("B,nb,H,hb,hc", [(1, 1, 1, 0, 1), (2, 36, 24, 6, 5), (1, 180, 23, 0, 23)])
def test_layer_lists_in_one_call_match_the_separate_ones(cuda_device, B, nb, H, hb, hc):
    from flashomni_b200.gemm import prepare_gemm_o_list, prepare_gemm_q_list
    masks = masks_to_device(wl.flux_masks(B, H, nb, nb, 0.5, seed=5, text_blocks=min(4, nb)), cuda_device)
    S, n = nb * 128, hc * 128
    indptr = torch.arange(B + 1, dtype=torch.int32, device=cuda_device) * S
    side, ev = torch.cuda.Stream(cuda_device), torch.cuda.Event()
    got = []
    for together in (False, True):
        w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1024, dtype=torch.uint8, device=cuda_device))
        w.plan(indptr, indptr, hc, hc, 128, q_data_type=torch.bfloat16, mask_num_heads=H, mask_head_begin=hb)
        lists = [f(B, S, n, H, masks[0], masks[2], 0, head_begin=hb, head_dim=128) for f in (prepare_gemm_q_list, prepare_gemm_o_list)]
        if together:
            for wlist in lists:
                wlist.ws.zero_()
            ev.record()
            w.prepare_layer_lists(*masks, *lists, S, n, side, ev)
        else:
            w.build_work_lists(*masks)
        torch.cuda.synchronize()
        got.append((w.work_lists(), [wlist.ws.cpu() for wlist in lists]))
    _assert_lists_equal(got[1][0], dict(got[0][0], items=got[0][0]["items"]))
    assert np.array_equal(got[0][0]["units"], got[1][0]["units"])
    for a, b in zip(got[0][1], got[1][1]):
        assert torch.equal(a, b)


# (batch, row blocks a request, mask heads, head window): as many row blocks as the one-launch kernel has threads (512), more,
# and more than twice as many (three passes of its scans), all within the one-launch size
@pytest.mark.parametrize("B,nb,H,hb,hc", [(16, 32, 3, 0, 3), (16, 36, 5, 1, 3), (64, 9, 7, 0, 7), (64, 17, 4, 2, 2)])
def test_layer_lists_of_many_row_blocks_match_the_oracle(cuda_device, B, nb, H, hb, hc):
    from flashomni_b200.gemm import prepare_gemm_o_list, prepare_gemm_q_list
    lib, rng = _native.load(), np.random.default_rng(nb)
    m = wl.pack_masks([(rng.random((nb, H)) < 0.6).astype(np.uint8) for _ in range(B)],
                      [(rng.random((nb, H, nb)) < 0.5).astype(np.uint8) for _ in range(B)])
    masks = masks_to_device(m, cuda_device)
    S, n, R = nb * 128, hc * 128, B * nb
    indptr = torch.arange(B + 1, dtype=torch.int32, device=cuda_device) * S
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1024, dtype=torch.uint8, device=cuda_device))
    w.plan(indptr, indptr, hc, hc, 128, q_data_type=torch.bfloat16, mask_num_heads=H, mask_head_begin=hb)
    ql, ol = (f(B, S, n, H, masks[0], masks[2], 0, head_begin=hb, head_dim=128) for f in (prepare_gemm_q_list, prepare_gemm_o_list))
    ql.ws.zero_(), ol.ws.zero_()
    side, ev = torch.cuda.Stream(cuda_device), torch.cuda.Event()
    ev.record()
    before = lib.fo_launch_count()
    w.prepare_layer_lists(*masks, ql, ol, S, n, side, ev)
    assert lib.fo_launch_count() == before + 1
    torch.cuda.synchronize()
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    got = ql.ws.view(torch.int32).cpu().numpy()
    ref = om.gemm_q_tile_pairs(m.sparse_info, m.info_indptr, B, S, n, H, 128, 0, head_begin=hb, head_dim=128, num_ctas=sms)
    assert got[0] == len(ref) and got[2] == 0 and np.array_equal(got[8:8 + 4 * len(ref)].reshape(-1, 4), ref)
    got = ol.ws.view(torch.int32).cpu().numpy()
    rip, rheads, rorder = om.gemm_o_rows(m.sparse_info, m.info_indptr, B, S, n, H, 128, 0, False, head_begin=hb, head_dim=128)
    assert got[0] == R and got[1] == len(rheads) and np.array_equal(got[8:8 + R + 1], rip)
    assert np.array_equal(got[9 + R:9 + R + len(rheads)], rheads)
    assert np.array_equal(got[9 + R + R * hc:9 + R + R * hc + R], rorder)
    qo = np.arange(B + 1) * S
    _assert_lists_equal(w.work_lists(), om.compact(m.sparse_info, m.sparse_kv_info, m.info_indptr, m.kv_info_indptr, qo, qo, H,
                                                   128, 128, hb, hc))


def test_strided_gather_matches_torch(cuda_device):
    """fo_strided_gather on local buffers: the two layouts of the sequence-parallel exchange."""
    from flashomni_b200.parallel import PeerExchange
    g = torch.Generator().manual_seed(5)
    H, D, hc = 8, 128, 2
    srcs = [torch.randn(n, H, D, generator=g).to(torch.bfloat16).to(cuda_device) for n in (256, 128, 384)]
    out = torch.zeros(sum(t.shape[0] for t in srcs), hc, D, dtype=torch.bfloat16, device=cuda_device)
    row = hc * D * 2
    offs = [0, 256, 384]
    PeerExchange.gather([t.data_ptr() + 3 * row for t in srcs], [H * D * 2] * 3, [t.shape[0] for t in srcs],
                        [out.data_ptr() + o * row for o in offs], [row] * 3, row)
    torch.cuda.synchronize()
    assert torch.equal(out, torch.cat([t[:, 6:8] for t in srcs]))
    # the way back: contiguous source rows into a column block of a wider destination
    back = torch.zeros(128, H, D, dtype=torch.bfloat16, device=cuda_device)
    PeerExchange.gather([out.data_ptr() + 256 * row], [row], [128], [back.data_ptr() + 3 * row], [H * D * 2], row)
    torch.cuda.synchronize()
    assert torch.equal(back[:, 6:8], srcs[1][:, 6:8]) and int(back[:, :6].abs().sum()) == 0
    with pytest.raises(ValueError):
        PeerExchange.gather([out.data_ptr() + 2], [row], [1], [back.data_ptr()], [row], row)   # misaligned


@pytest.mark.parametrize("case", ["few_items_cut", "many_items_whole", "ragged"])
def test_attention_work_units_bit_exact(cuda_device, case, monkeypatch):
    """The unit list the attention kernel walks (fo_attn_units) against the oracle's statement: long kv lists are
    cut into parts when the launch has few items per stream, never otherwise."""
    monkeypatch.setattr(fo.BatchFlashOmniFAWithRaggedKVWrapper, "UNITS_PER_SM", 2)   # list cutting on
    if case == "few_items_cut":
        H, lens = 6, [36 * 128]                      # about 195 items: between one and two per SM
        m = wl.flux_masks(1, H, 36, 36, 0.9, seed=21)
    elif case == "many_items_whole":
        H, lens = 24, [36 * 128, 36 * 128]
        m = wl.flux_masks(2, H, 36, 36, 0.9, seed=22)
    else:
        H, lens = 3, [700, 128 * 9 + 5, 40]
        rng = np.random.default_rng(23)
        qa = [(rng.random((-(-n // 128), H)) < 0.8).astype(np.uint8) for n in lens]
        kk = [(rng.random((-(-n // 128), H, -(-n // 128))) < 0.7).astype(np.uint8) * a[:, :, None] for n, a in zip(lens, qa)]
        m = wl.pack_masks(qa, kk)
    qo = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1024, dtype=torch.uint8, device=cuda_device))
    w.plan(dev(qo, cuda_device), dev(qo, cuda_device), H, H, 128, q_data_type=torch.bfloat16)
    w.build_work_lists(*masks_to_device(m, cuda_device))
    torch.cuda.synchronize()
    got = w.work_lists()
    ref = om.compact(m.sparse_info, m.sparse_kv_info, m.info_indptr, m.kv_info_indptr, qo, qo, H, 128, 128)
    _assert_lists_equal(got, ref)
    units, slots, chunk = om.attn_units(ref, qo, qo, w._num_streams, w.MIN_CHUNK, max_slots=w._partial_slots,
                                        min_items=w._min_items)
    assert got["unit_status"] == 0 and got["chunk_max"] == chunk and got["partial_slots_used"] == slots
    assert got["n_units"] == len(units) and np.array_equal(got["units"], units)
    if case == "many_items_whole":
        assert slots == 0 and len(units) == len(ref["items"])
    if case == "few_items_cut":
        assert slots > 0
    assert got["n_units"] <= w._max_units and slots <= w._partial_slots


@pytest.mark.parametrize("n", [3000, 147 * 8192, 149 * 8192, 40_000_000])
def test_packed_bytes_are_complete_on_return(cuda_device, n):
    """Whatever reads them next, on any stream: here a stream that is not ordered behind the packing, which itself waits behind
    other work. One block, a block short of and past one per SM (the words that are polled), more than eight per SM."""
    side = torch.cuda.Stream(cuda_device)
    a = torch.randn(4096, 4096, device=cuda_device)
    for seed in range(3):
        x = torch.from_numpy(np.random.default_rng(seed).random(n) < 0.5).to(cuda_device)
        ip = torch.tensor([0, 5, n // 2, n], dtype=torch.int32, device=cuda_device)
        a @ a
        y, new = fo.segment_packbits(x, ip, "little")
        x.zero_()   # (in stream order behind the packing)
        with torch.cuda.stream(side):
            y, new = y.clone(), new.clone()
        side.synchronize()
        want = np.random.default_rng(seed).random(n) < 0.5
        want = np.concatenate([np.packbits(want[i:j], bitorder="little") for i, j in ((0, 5), (5, n // 2), (n // 2, n))])
        assert np.array_equal(y.cpu().numpy(), want) and int(new[-1]) == len(want)


def test_lists_on_a_side_stream_are_built_from_masks_packed_after_the_event(cuda_device):
    """`prepare_masks(stream=, after=)` is ordered behind that event alone, and a GEMM list in storage of its own behind nothing:
    masks packed since then must be complete."""
    B, S, H, D = 2, 1024, 8, 128
    nb = S // 128
    side = torch.cuda.Stream(cuda_device)
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1 << 20, dtype=torch.uint8, device=cuda_device))
    ip = torch.arange(B + 1, dtype=torch.int32, device=cuda_device) * S
    w.plan(ip, ip, H, H, D, q_data_type=torch.bfloat16)
    q, k, v = (torch.randn(B * S, H, D, device=cuda_device).bfloat16() for _ in range(3))
    x, wq = torch.randn(B, S, 256, device=cuda_device).bfloat16(), torch.randn(H * D, 256, device=cuda_device).bfloat16()
    busy = torch.randn(4096, 4096, device=cuda_device)
    wl_q = None
    for seed in range(4):
        rng = np.random.default_rng(seed)
        qa, kk = (torch.from_numpy(rng.random(s) < 0.5).to(cuda_device) for s in ((B, nb, H), (B, nb, H, nb)))
        qi, ki = (torch.arange(B + 1, dtype=torch.int32, device=cuda_device) * t[0].numel() for t in (qa, kk))
        after = torch.cuda.Event()
        after.record()
        busy @ busy
        si, sp = fo.segment_packbits(qa.view(-1), qi, "little")
        sk, kp = fo.segment_packbits(kk.view(-1), ki, "little")
        w.prepare_masks(si, sk, sp, kp, stream=side, after=after)
        wl_q = fo.gemm.prepare_gemm_q_list(B, S, H * D, H, si, sp, 0, into=wl_q, stream=side)
        o = w.run(q, k, v, si, sk, sp, kp, out=torch.zeros_like(q))
        y = fo.flashomni_gemm(x, wq, H, si, sp, 0, out=torch.zeros(B, S, H * D, dtype=x.dtype, device=cuda_device), worklist=wl_q)
        assert torch.equal(o, w.run(q, k, v, si, sk, sp, kp, out=torch.zeros_like(q)))
        assert torch.equal(y, fo.flashomni_gemm(x, wq, H, si, sp, 0, out=torch.zeros_like(y)))
        w.check_status()
