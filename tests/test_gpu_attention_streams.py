"""GPU: the attention kernel with two streams of kv blocks per SM where it can go wrong: units of one, two and three kv
blocks in a row (a unit of one block belongs to one stream only), more units than CTAs, partial q-blocks and kv blocks,
rows whose maximum rises late (rescale), grouped heads, both head dimensions and types, NaN inputs."""

import numpy as np
import pytest
import torch

import flashomni_b200 as fo
from flashomni_b200 import workloads as wl
from oracle import attention as oa
from helpers import assert_close_bf16, dev, masks_to_device

pytestmark = pytest.mark.gpu


def _case(lens_q, lens_kv, H, Hkv, D, dtype, density, seed, q_scale=1.0):
    rng = np.random.default_rng(seed)
    qo = np.concatenate([[0], np.cumsum(lens_q)]); kv = np.concatenate([[0], np.cumsum(lens_kv)])
    qt = 128 // (H // Hkv)
    qa = [(rng.random((-(-a // qt), Hkv)) < 0.8).astype(np.uint8) for a in lens_q]
    kk = [(rng.random((-(-a // qt), Hkv, -(-b // 128))) < density).astype(np.uint8) for a, b in zip(lens_q, lens_kv)]
    q = (wl.randn_bf16((int(qo[-1]), H, D), seed + 1).float() * q_scale).to(dtype)
    k = wl.randn_bf16((int(kv[-1]), Hkv, D), seed + 2, dtype=dtype)
    v = wl.randn_bf16((int(kv[-1]), Hkv, D), seed + 3, dtype=dtype)
    return qo, kv, wl.pack_masks(qa, kk), q, k, v


def _plan(device, qo, kv, H, Hkv, D, dtype):
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1 << 20, dtype=torch.uint8, device=device))
    w.plan(dev(np.asarray(qo, np.int32), device), dev(np.asarray(kv, np.int32), device), H, Hkv, D, q_data_type=dtype)
    return w


@pytest.mark.parametrize("D,H,Hkv,dtype,q_scale", [
    (128, 8, 8, torch.bfloat16, 1.0), (128, 8, 8, torch.float16, 3.0), (128, 16, 4, torch.bfloat16, 1.0),
    (64, 8, 8, torch.bfloat16, 3.0), (64, 6, 3, torch.float16, 1.0)])
def test_many_short_units_against_the_oracle(cuda_device, D, H, Hkv, dtype, q_scale):
    """With q_scale 3 the logits are N(0, 9): maxima rise by more than the rescale threshold between blocks. The error
    of one value is at most two roundings to 16 bits (P and O), 2 * 2^-9 * max|v| < 0.02 for bf16 and |v| < 5."""
    lens_kv = [128, 77, 256, 1, 129, 128, 384, 300, 500, 64, 128, 128, 1100] * 3
    lens_q = [128, 77, 300, 1, 128, 200, 129, 64, 333, 127, 65, 500, 260] * 3
    qo, kv, m, q, k, v = _case(lens_q, lens_kv, H, Hkv, D, dtype, 0.7, 31, q_scale)
    w = _plan(cuda_device, qo, kv, H, Hkv, D, dtype)
    prior, lse_prior = wl.randn_bf16(q.shape, 9, dtype=dtype), torch.full((q.shape[0], H), 3.0)
    for _ in range(2):   # twice: the second launch starts from the cursor that the first one put back
        o, lse = w.run(dev(q, cuda_device), dev(k, cuda_device), dev(v, cuda_device), *masks_to_device(m, cuda_device),
                       out=dev(prior, cuda_device).clone(), lse=dev(lse_prior, cuda_device).clone(), return_lse=True)
        w.check_status()
    n = w.work_lists()["items"][:, 3]
    assert len(n) > 148 and {0, 1, 2, 3} <= set(n.tolist())
    ref, ref_lse = oa.sparse_attention(q, k, v, qo, kv, m.sparse_info, m.sparse_kv_info, m.info_indptr, m.kv_info_indptr,
                                       out_prior=prior, lse_prior=lse_prior, return_lse=True)
    assert_close_bf16(o, ref, f"D={D} H={H}/{Hkv} {dtype}", allow_ulp=1.0)
    assert torch.allclose(lse.cpu(), ref_lse, atol=2e-2, rtol=1e-4)


def test_the_same_bits_from_call_to_call(cuda_device):
    """Which units a CTA draws, and with them which stream a unit's first block belongs to, changes from call to call; sums and
    their rounding do not."""
    lens = [128, 700, 333, 1, 900, 77, 512, 1300]
    qo, kv, m, q, k, v = _case(lens, lens[::-1], 16, 16, 128, torch.bfloat16, 0.6, 5)
    w = _plan(cuda_device, qo, kv, 16, 16, 128, torch.bfloat16)
    args = [dev(t, cuda_device) for t in (q, k, v)] + list(masks_to_device(m, cuda_device))
    fresh = lambda: torch.full((q.shape[0], 16), 3.0, device=cuda_device)   # rows of skipped q-blocks keep what they hold
    first, first_lse = w.run(*args, lse=fresh(), return_lse=True)
    first = first.clone()
    for _ in range(20):
        o, lse = w.run(*args, lse=fresh(), return_lse=True)
        assert torch.equal(o.view(torch.int16), first.view(torch.int16)) and torch.equal(lse, first_lse)
    w.check_status()


@pytest.mark.parametrize("keep", [0.0, 0.02, 0.25])
def test_long_runs_of_units_that_keep_nothing(cuda_device, keep):
    """Active q-blocks without a kept kv-block sit at the end of the processing order, several per CTA behind each other."""
    S, H, D = 4992, 32, 64
    n = S // 128
    rng = np.random.default_rng(5)
    kk = np.zeros((n, H, n), np.uint8)
    some = rng.random((n, H)) < keep
    kk[some] = rng.random((int(some.sum()), n)) < 0.2
    m = wl.pack_masks([np.ones((n, H), np.uint8)], [kk])
    q, k, v = (wl.randn_bf16((S, H, D), s) for s in (1, 2, 3))
    w = _plan(cuda_device, [0, S], [0, S], H, H, D, torch.bfloat16)
    prior = wl.randn_bf16(q.shape, 9)
    o, lse = w.run(dev(q, cuda_device), dev(k, cuda_device), dev(v, cuda_device), *masks_to_device(m, cuda_device),
                   out=dev(prior, cuda_device).clone(), return_lse=True)
    w.check_status()
    kept = kk.any(2)
    blocks = o.cpu().view(n, 128, H, D).permute(0, 2, 1, 3)
    assert (blocks[torch.from_numpy(~kept)] == 0).all()
    assert (lse.cpu().view(n, 128, H).permute(0, 2, 1)[torch.from_numpy(~kept)] == -5e4).all()
    for h in np.flatnonzero(kept.any(0))[:6]:
        one = wl.pack_masks([np.ones((n, 1), np.uint8)], [np.ascontiguousarray(kk[:, h:h + 1])])
        ref = oa.sparse_attention(q[:, h:h + 1], k[:, h:h + 1], v[:, h:h + 1], [0, S], [0, S], one.sparse_info, one.sparse_kv_info,
                                  one.info_indptr, one.kv_info_indptr)
        assert_close_bf16(o[:, h:h + 1], ref, f"head {h}")


@pytest.mark.parametrize("blocks", [1, 2, 5])
def test_nan_in_a_key_reaches_every_row_that_attends_to_it(cuda_device, blocks):
    S, H, D = 128 * blocks, 2, 128
    q, k, v = (wl.randn_bf16((S, H, D), s) for s in (1, 2, 3))
    k[S - 20, 1, 7] = float("nan")
    w = _plan(cuda_device, [0, S], [0, S], H, H, D, torch.bfloat16)
    o = w.run(dev(q, cuda_device), dev(k, cuda_device), dev(v, cuda_device), is_full=True).cpu()
    w.check_status()
    assert torch.isnan(o[:, 1]).all() and torch.isfinite(o[:, 0]).all()


@pytest.mark.parametrize("blocks", [1, 2, 3])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["bf16", "f16", "e5m2"])
def test_infinities_in_v_reach_the_output_as_infinities(cuda_device, kind, D, blocks):
    """A row of V with +inf, -inf or both in a column: every weight is positive (|logit| < 8, so P > 2^-24 also in f16), so
    the column is +inf, -inf or NaN in every row that attends to it, and nothing else changes."""
    S, H = 128 * blocks, 2
    dtype = torch.float16 if kind == "f16" else torch.bfloat16
    q, k, v = (wl.randn_bf16((S, H, D), s).to(dtype) for s in (1, 2, 3))
    v[S - 20, 1, 7], v[3, 1, 9] = float("inf"), -float("inf")
    v[5, 1, D - 1], v[S - 1, 1, D - 1] = float("inf"), -float("inf")
    kv_dtype = torch.float8_e5m2 if kind == "e5m2" else dtype
    k, v = k.to(kv_dtype), v.to(kv_dtype)
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1 << 20, dtype=torch.uint8, device=cuda_device))
    ip = torch.tensor([0, S], dtype=torch.int32, device=cuda_device)
    w.plan(ip, ip, H, H, D, q_data_type=dtype, kv_data_type=kv_dtype)
    o = w.run(dev(q, cuda_device), dev(k, cuda_device), dev(v, cuda_device), is_full=True).float().cpu()
    w.check_status()
    qf, kf, vf = (t.float().transpose(0, 1) for t in (q, k, v))
    p = torch.softmax(qf @ kf.transpose(1, 2) / D ** 0.5, 2)
    ref = (p @ vf).transpose(0, 1)
    assert torch.isposinf(o[:, 1, 7]).all() and torch.isneginf(o[:, 1, 9]).all() and torch.isnan(o[:, 1, D - 1]).all()
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(o), fin)
    assert_close_bf16(o[fin], ref[fin], f"{kind} D={D} blocks={blocks}", allow_ulp=1.0)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_small_weights_add_up_in_the_row_sum(cuda_device, dtype, D):
    """One block of logits 0 and 71 blocks of logits -21, in base 2: 2^-21 is below the last bit of a sum that has reached 32, but
    the 9 088 of them are 3.4e-5 of the whole. The log-sum-exp is known to a few units of its last place: log2 and
    the sum with the maximum 2^-21 each at a magnitude below 8, the scaled logit 21 * 2^-23 times a weight of 3.4e-5."""
    blocks, H = 72, 1
    S = 128 * blocks
    q, k, v = torch.zeros(S, H, D), torch.zeros(S, H, D), torch.ones(S, H, D)
    q[:, :, 0] = 1.0
    k[128:, :, 0] = -21.0
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1 << 20, dtype=torch.uint8, device=cuda_device))
    ip = torch.tensor([0, S], dtype=torch.int32, device=cuda_device)
    w.plan(ip, ip, H, H, D, q_data_type=dtype, sm_scale=float(np.log(2.0)))
    o, lse = w.run(*(dev(t.to(dtype), cuda_device) for t in (q, k, v)), is_full=True, return_lse=True)
    w.check_status()
    want = np.log2(128 + (S - 128) * 2.0 ** -21)
    assert (lse.cpu().double() - want).abs().max() <= 2.0 ** -20
    assert (o == 1).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S", [128, 333, 1024])
def test_log_sum_exp_of_exact_sums_is_rounded_once(cuda_device, S, D):
    """Integer logits from -4 to 4 in base 2 (sm_scale * log2(e) is 1 in float32): exponentials, merge weights and sums (at most 19
    bits) are exact, so what is left is the rounding of the result, half a unit in its last place, and one unit of a logarithm
    below 1 (2^-24) with its addition (2^-25)."""
    H = 8
    g = torch.Generator().manual_seed(S + D)
    q, k = torch.zeros(S, H, D), torch.zeros(S, H, D)
    q[..., :4] = torch.randint(0, 2, (S, H, 4), generator=g).float()
    k[..., :4] = torch.randint(-1, 2, (S, H, 4), generator=g).float()
    v = torch.randn(S, H, D, generator=g)
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1 << 20, dtype=torch.uint8, device=cuda_device))
    ip = torch.tensor([0, S], dtype=torch.int32, device=cuda_device)
    w.plan(ip, ip, H, H, D, q_data_type=torch.bfloat16, sm_scale=float(np.log(2.0)))
    _, lse = w.run(*(dev(t.bfloat16(), cuda_device) for t in (q, k, v)), is_full=True, return_lse=True)
    w.check_status()
    want = torch.log2(torch.exp2(torch.einsum("qhd,khd->qhk", q.double(), k.double())).sum(2))
    half_ulp = torch.exp2(torch.floor(torch.log2(want)) - 24)
    assert ((lse.cpu().double() - want).abs() <= half_ulp + 1.5 * 2.0 ** -24).all()
