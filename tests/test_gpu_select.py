"""Block selection on the GPU: bit-exact against the CPU statement, and usable by the hot path as is."""

import numpy as np
import pytest
import torch

import flashomni_b200 as fo
from oracle import select as osel

pytestmark = pytest.mark.gpu


def _run(s, t2t, qthr, kthr, zero_inactive, device):
    out = fo.select_blocks(torch.from_numpy(s).to(device), t2t, qthr, kthr, zero_inactive=zero_inactive)
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in out]


@pytest.mark.parametrize("B,H,n,t2t", [(1, 2, 5, 2), (2, 3, 36, 4), (1, 4, 77, 3), (2, 24, 36, 4), (1, 2, 604, 4),
                                       (3, 1, 33, 0), (1, 3, 40, 40)])
@pytest.mark.parametrize("zero_inactive", [True, False])
def test_bit_exact(cuda_device, B, H, n, t2t, zero_inactive):
    rng = np.random.default_rng(1000 * n + H)
    s = (rng.standard_normal((B, H, n, n)) * 1.5).astype(np.float32)
    qthr = rng.uniform(0.05, 0.5, B).astype(np.float32)
    kthr = rng.uniform(0.05, 0.6, H).astype(np.float32)
    info, kv, ip, kp = _run(s, t2t, torch.from_numpy(qthr), torch.from_numpy(kthr), zero_inactive, cuda_device)
    qa, kk = osel.select_blocks(s, t2t, qthr, kthr, zero_inactive=zero_inactive)
    rinfo, rkv, rip, rkp = osel.pack_selection(qa, kk)
    assert np.array_equal(ip, rip) and np.array_equal(kp, rkp)
    assert np.array_equal(info, rinfo)
    assert np.array_equal(kv, rkv)


@pytest.mark.parametrize("H", [7, 8, 9, 13, 65])
@pytest.mark.parametrize("n,t2t", [(9, 2), (17, 9), (44, 3)])
def test_bytes_that_two_blocks_share(cuda_device, H, n, t2t):
    """A byte of sparse_info holds bits of one, two (8 heads and more) or several q-blocks, and ends short in the last one."""
    s = (np.random.default_rng(H * n).standard_normal((2, H, n, n)) * 1.5).astype(np.float32)
    got = _run(s, t2t, 0.35, 0.3, True, cuda_device)
    want = osel.pack_selection(*osel.select_blocks(s, t2t, 0.35, 0.3))
    assert all(np.array_equal(g, w) for g, w in zip(got, (want[0], want[1], want[2], want[3])))


def test_ties_and_extremes(cuda_device):
    n = 64
    s = np.zeros((1, 2, n, n), dtype=np.float32)          # all scores equal: ties broken by block index
    s[0, 1, :, ::2] = -200.0                                # masses that round to zero are switched off first
    for thr in (0.0, 0.25, 1.0):
        info, kv, ip, kp = _run(s, 2, thr, thr, False, cuda_device)
        qa, kk = osel.select_blocks(s, 2, thr, thr, zero_inactive=False)
        rinfo, rkv, _, _ = osel.pack_selection(qa, kk)
        assert np.array_equal(info, rinfo) and np.array_equal(kv, rkv)


# row lengths at the edges of the per-lane entry counts (4, 20 and 64), one threshold for all; scores that spread,
# that differ by less than a float step of their mass, that take three values (more than 32 equal masses), and with
# infinities of both signs
@pytest.mark.parametrize("n", [1, 2, 31, 128, 129, 640, 641])
@pytest.mark.parametrize("kind", ["normal", "flat", "three", "inf"])
@pytest.mark.parametrize("thr", [0.0, 0.3, 0.97])
def test_one_threshold_for_all(cuda_device, n, kind, thr):
    rng = np.random.default_rng(n)
    H, t2t = (2 if n < 600 else 1), min(2, n)
    s = rng.standard_normal((1, H, n, n)).astype(np.float32)
    if kind == "flat":
        s *= np.float32(1e-6)
    elif kind == "three":
        s = rng.integers(0, 3, s.shape).astype(np.float32)
    elif kind == "inf":
        s[rng.random(s.shape) < 0.5] = -np.inf
        s[:, :, :, 0] = np.where(s[:, :, :, 0] == -np.inf, 0, s[:, :, :, 0])
    info, kv, ip, kp = _run(s, t2t, thr, thr, True, cuda_device)
    with np.errstate(invalid="ignore"):
        qa, kk = osel.select_blocks(s, t2t, thr, thr)
    rinfo, rkv, rip, rkp = osel.pack_selection(qa, kk)
    assert np.array_equal(ip, rip) and np.array_equal(kp, rkp)
    assert np.array_equal(info, rinfo) and np.array_equal(kv, rkv)


@pytest.mark.parametrize("thr", [(1e39, 0.3), (0.3, -1e300)])
def test_thresholds_past_fp32_are_refused(cuda_device, thr):
    s = torch.zeros(1, 1, 4, 4, device=cuda_device)
    fo.select_blocks(s, 1, float("inf"), float("nan"))
    with pytest.raises(RuntimeError, match="overflow"):
        fo.select_blocks(s, 1, *thr)


# few text rows and more requests than fit on the GPU at once: the CTAs of a request reach the exchange of their scores right
# after they start, at different times
@pytest.mark.parametrize("B,n", [(1, 2), (3, 9), (200, 9)])
def test_scores_meet_across_the_cluster(cuda_device, B, n):
    rng = np.random.default_rng(B)
    s = (rng.standard_normal((B, 1, n, n)) * 2).astype(np.float32)
    want = osel.pack_selection(*osel.select_blocks(s, 1, 0.4, 0.3))
    x = torch.from_numpy(s).to(cuda_device)
    for got in [fo.select_blocks(x, 1, 0.4, 0.3) for _ in range(50)]:
        for g, r in zip(got, (want[0], want[1], want[2], want[3])):
            assert np.array_equal(g.cpu().numpy(), r)


def test_feeds_the_hot_path(cuda_device):
    """The emitted tensors go straight into the attention wrapper; the result equals the run on masks packed
    from the CPU statement."""
    from flashomni_b200 import workloads as wl
    from helpers import dev
    B, H, n, D = 1, 4, 8, 128
    S = n * 128
    rng = np.random.default_rng(7)
    s = rng.standard_normal((B, H, n, n)).astype(np.float32)
    masks = fo.select_blocks(torch.from_numpy(s).to(cuda_device), 1, 0.3, 0.4)
    qa, kk = osel.select_blocks(s, 1, 0.3, 0.4)
    ref_masks = [torch.from_numpy(a).to(cuda_device) for a in osel.pack_selection(qa, kk)]
    q, k, v = (dev(wl.randn_bf16((S, H, D), 20 + i), cuda_device) for i in range(3))
    indptr = torch.tensor([0, S], dtype=torch.int32, device=cuda_device)
    w = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1 << 20, dtype=torch.uint8, device=cuda_device))
    w.plan(indptr, indptr, H, H, D, q_data_type=torch.bfloat16)
    a = w.run(q, k, v, *masks).clone()
    b = w.run(q, k, v, *ref_masks)
    w.check_status()
    assert torch.equal(a, b)


def test_matches_the_reference_masks(cuda_device):
    """fo_select_blocks against the masks the reference's own torch + Triton path produced
    (tests/golden/reference_selection.npz), same rule for rows at the threshold as the CPU statement's test."""
    from helpers import check_selection_against_golden, load_selection_golden
    from oracle.masks import unpack_segment
    cases, _ = load_selection_golden()
    for c in cases:
        B, H, n = c["B"], c["H"], c["n"]
        info, kv, ip, kp = _run(c["score"], c["t2t"], torch.from_numpy(c["q_threshold"]),
                                torch.from_numpy(c["kv_threshold"]), False, cuda_device)
        qa = np.stack([unpack_segment(info, int(ip[b]), n * H).reshape(n, H) for b in range(B)])
        kk = np.stack([unpack_segment(kv, int(kp[b]), n * H * n).reshape(n, H, n) for b in range(B)])
        check_selection_against_golden(c, qa, kk)
