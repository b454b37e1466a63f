"""Timing cases of the framework's main path, through its public entry points.

One denoising step of a sparse DiT layer is: block selection (or the caller's own flags and `segment_packbits`),
GEMM-Q, dense K / V projections, block-sparse attention over ragged requests, GEMM-O with the cached contribution of
the heads that are skipped. The cases cover each of these calls alone and the assembled layers, from calls that are
all latency to the long video layer. Sizes are those of `flashomni_b200/workloads.py`, of `bench.py` and of the tests.

`sparse` attention cases have a mask per (128-row q-block, head) and per (q-block, head, kv-block) as
`workloads.flux_masks` makes it: Bernoulli(density), text blocks and the diagonal always on. `full` ones are the dense
steps that a sampler runs first (`is_full=True`)."""

import math

import torch

import flashomni_b200 as fo
from flashomni_b200.gemm import prepare_gemm_o_list, prepare_gemm_q_list
from flashomni_b200.layer import BlockWeights, SparseDiTAttentionBlock, UlyssesSparseDiTAttentionBlock

BLOCK = 128
_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "e4m3": torch.float8_e4m3fn}


def listed():
    return [
        # smallest: one short request, a handful of work items; launches and host time are all there is
        {"name": "attention_short", "kind": "attention", "lens": "333", "heads": 4, "kv_heads": 4, "dim": 64,
         "dtype": "f16", "kv_dtype": "f16", "density": 0.6, "text": 1, "full": False, "lse": False},
        # a batch of requests of unequal, odd lengths with grouped heads, K / V stored in 8 bits, log-sum-exp returned
        {"name": "attention_ragged", "kind": "attention", "lens": "2051,300,77,1531", "heads": 16, "kv_heads": 8,
         "dim": 128, "dtype": "f16", "kv_dtype": "e4m3", "density": 0.5, "text": 1, "full": False, "lse": True},
        # the image layer: 4096 image + 512 text tokens, half of the blocks
        {"name": "attention_image", "kind": "attention", "lens": "4608", "heads": 24, "kv_heads": 24, "dim": 128,
         "dtype": "bf16", "kv_dtype": "bf16", "density": 0.5, "text": 4, "full": False, "lse": False},
        # the same layer in the dense steps of a sampler
        {"name": "attention_image_full", "kind": "attention", "lens": "4608", "heads": 24, "kv_heads": 24, "dim": 128,
         "dtype": "bf16", "kv_dtype": "bf16", "density": 1.0, "text": 4, "full": True, "lse": False},
        # the two sparse projections of that layer, each called alone
        {"name": "gemm_q_image", "kind": "gemm_q", "batch": 1, "rows": 4608, "heads": 24, "dim": 128, "hidden": 3072,
         "dtype": "bf16", "density": 0.5, "text": 4, "bias": False},
        {"name": "gemm_o_image", "kind": "gemm_o", "batch": 1, "rows": 4608, "heads": 24, "dim": 128, "hidden": 3072,
         "dtype": "bf16", "density": 0.5, "text": 4, "for_cache": False},
        # a small layer, one step
        {"name": "layer_small", "kind": "layer", "batch": 1, "rows": 1024, "heads": 8, "own_heads": 8, "dim": 128,
         "hidden": 1024, "dtype": "bf16", "density": 0.5, "text": 1},
        # the image layer, one step of two requests
        {"name": "layer_image", "kind": "layer", "batch": 2, "rows": 4608, "heads": 24, "own_heads": 24, "dim": 128,
         "hidden": 3072, "dtype": "bf16", "density": 0.5, "text": 4},
        # one GPU's part of it when the heads are split over eight
        {"name": "layer_image_eighth", "kind": "layer", "batch": 2, "rows": 4608, "heads": 24, "own_heads": 3,
         "dim": 128, "hidden": 3072, "dtype": "bf16", "density": 0.5, "text": 4},
        # largest: the video layer, 20 frames of 30 blocks, frame-local mask with random blocks
        {"name": "layer_video", "kind": "video", "frames": 20, "frame_blocks": 30, "heads": 40, "dim": 128,
         "hidden": 5120, "dtype": "bf16", "density": 0.1, "text": 4},
        # block selection from the pooled scores of the video layer
        {"name": "select_video", "kind": "select", "batch": 1, "heads": 40, "blocks": 604, "text": 4},
        # packing of a caller's own flags for the image layer
        {"name": "pack_image", "kind": "pack", "batch": 2, "heads": 24, "blocks": 36, "text": 4, "density": 0.5},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "gemm_q", "gemm_o", "layer", "layer", "video", "select",
                       "pack"])
    if kind == "attention":
        batch = rng.choice([1, 1, 2, 3, 4])
        lens = [_log_int(rng, 65, 4608) for _ in range(batch)]
        group = rng.choice([1, 1, 1, 2])
        kv_heads = rng.randint(2, 24 // group)
        full = rng.random() < 0.2
        dtype = rng.choice(["bf16", "bf16", "f16"])
        return {"kind": kind, "lens": ",".join(map(str, lens)), "heads": kv_heads * group, "kv_heads": kv_heads,
                "dim": rng.choice([64, 128, 128]), "dtype": dtype,
                "kv_dtype": "e4m3" if rng.random() < 0.2 else dtype,
                "density": 1.0 if full else round(rng.uniform(0.2, 0.9), 3), "text": rng.randint(1, 4), "full": full,
                "lse": rng.random() < 0.3}
    if kind in ("gemm_q", "gemm_o"):
        heads = rng.randint(2, 24)
        case = {"kind": kind, "batch": rng.choice([1, 1, 2]), "rows": BLOCK * _log_int(rng, 1, 72), "heads": heads,
                "dim": 128, "hidden": 128 * rng.randint(max(2, heads // 2), 24), "dtype": rng.choice(["bf16", "bf16", "f16"]),
                "density": round(rng.uniform(0.2, 0.9), 3), "text": rng.randint(1, 4)}
        if kind == "gemm_q":
            case["bias"] = rng.random() < 0.4
        else:
            case["for_cache"] = rng.random() < 0.4
        return case
    if kind == "layer":
        heads = rng.randint(4, 24)
        return {"kind": kind, "batch": rng.choice([1, 2]), "rows": BLOCK * _log_int(rng, 4, 36), "heads": heads,
                "own_heads": heads if rng.random() < 0.6 else max(1, heads // rng.choice([2, 4, 8])), "dim": 128,
                "hidden": 128 * heads, "dtype": rng.choice(["bf16", "bf16", "f16"]),
                "density": round(rng.uniform(0.25, 0.75), 3), "text": rng.randint(1, 4)}
    if kind == "video":
        heads = rng.randint(8, 40)
        return {"kind": kind, "frames": rng.randint(4, 20), "frame_blocks": rng.randint(6, 30), "heads": heads,
                "dim": 128, "hidden": 128 * heads, "dtype": "bf16", "density": round(rng.uniform(0.05, 0.25), 3),
                "text": rng.randint(2, 4)}
    batch, heads = rng.choice([1, 1, 2]), rng.randint(4, 40)
    if kind == "select":
        return {"kind": kind, "batch": batch, "heads": heads, "blocks": _log_int(rng, 12, 604), "text": rng.randint(1, 4)}
    return {"kind": kind, "batch": batch, "heads": heads, "blocks": _log_int(rng, 12, 604), "text": rng.randint(1, 4),
            "density": round(rng.uniform(0.2, 0.9), 3)}


# ------------------------------------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _randn(gen, shape, dtype, std=1.0):
    """N(0, std) in `dtype`, made in slices so that the float32 source never doubles a large tensor's footprint."""
    out = torch.empty(shape, dtype=dtype, device=_dev())
    flat = out.view(-1)
    step = 1 << 26
    for i in range(0, flat.numel(), step):
        n = min(step, flat.numel() - i)
        flat[i:i + n] = torch.randn(n, generator=gen, device=_dev()) * std
    return out


def _image_flags(gen, nq, heads, nkv, density, text, q_tokens=BLOCK):
    """Flags of one request: [nq, heads] and [nq, heads, nkv] (text blocks and the diagonal always on, rows of
    inactive q-blocks zero)."""
    rand = lambda *s: torch.rand(*s, generator=gen, device=_dev())
    tq, tk = min(nq, (text * BLOCK + q_tokens - 1) // q_tokens), min(text, nkv)
    qa = rand(nq, heads) < density
    qa[:tq] = True
    kk = rand(nq, heads, nkv) < density
    kk[:, :, :tk] = True
    rows = torch.arange(nq, device=_dev())
    kk[rows, :, torch.clamp(rows * q_tokens // BLOCK, max=nkv - 1)] = True
    return qa, kk & qa[:, :, None]


def _video_flags(gen, text, frames, frame_blocks, heads, density):
    n = text + frames * frame_blocks
    frame = torch.full((n,), -10, device=_dev())
    frame[text:] = torch.arange(n - text, device=_dev()) // frame_blocks
    local = ((frame[:, None] - frame[None, :]).abs() <= 1) & (frame[:, None] >= 0) & (frame[None, :] >= 0)
    qa = torch.ones(n, heads, dtype=torch.bool, device=_dev())
    kk = (torch.rand(n, heads, n, generator=gen, device=_dev()) < density) | local[:, None, :]
    kk[:, :, :text] = True
    return qa, kk


def _flat(flags):
    """Concatenated flags of the requests and their element indptr, as callers hand them to segment_packbits."""
    indptr = [0]
    for f in flags:
        indptr.append(indptr[-1] + f.numel())
    return torch.cat([f.reshape(-1) for f in flags]), torch.tensor(indptr, dtype=torch.int32, device=_dev())


def _packed(flags):
    qa, kk = _flat([f[0] for f in flags]), _flat([f[1] for f in flags])
    si, ip = fo.segment_packbits(*qa, bitorder="little")
    sk, kp = fo.segment_packbits(*kk, bitorder="little")
    return si, sk, ip, kp


def _lens(case):
    return [int(x) for x in case["lens"].split(",")]


def prepare(case, seed):
    gen = torch.Generator(device=_dev()).manual_seed(int(seed))
    kind = case["kind"]
    if kind == "attention":
        lens, group, dt = _lens(case), case["heads"] // case["kv_heads"], _DTYPES[case["dtype"]]
        q_tokens = BLOCK // group
        total, D = sum(lens), case["dim"]
        q = _randn(gen, (total, case["heads"], D), dt)
        k, v = (_randn(gen, (total, case["kv_heads"], D), dt).to(_DTYPES[case["kv_dtype"]]) for _ in range(2))
        indptr = torch.tensor([0] + [sum(lens[:i + 1]) for i in range(len(lens))], dtype=torch.int32, device=_dev())
        wrapper = fo.BatchFlashOmniFAWithRaggedKVWrapper(torch.empty(1 << 20, dtype=torch.uint8, device=_dev()))
        wrapper.plan(indptr, indptr, case["heads"], case["kv_heads"], D, q_data_type=dt,
                     kv_data_type=_DTYPES[case["kv_dtype"]])
        masks = (None,) * 4
        if not case["full"]:
            masks = _packed([_image_flags(gen, -(-n // q_tokens), case["kv_heads"], -(-n // BLOCK), case["density"],
                                          case["text"], q_tokens) for n in lens])
        # the log-sum-exp buffer is the caller's: rows of inactive q-blocks are not written
        lse = torch.zeros(total, case["heads"], device=_dev()) if case["lse"] else None
        return {"case": case, "wrapper": wrapper, "q": q, "k": k, "v": v, "masks": masks, "lse": lse}
    if kind in ("gemm_q", "gemm_o"):
        dt, n, hid = _DTYPES[case["dtype"]], case["heads"] * case["dim"], case["hidden"]
        nb = case["rows"] // BLOCK
        si, _, ip, _ = _packed([_image_flags(gen, nb, case["heads"], 1, case["density"], case["text"])
                                for _ in range(case["batch"])])
        state = {"case": case, "masks": (si, ip)}
        if kind == "gemm_q":
            state["x"] = _randn(gen, (case["batch"], case["rows"], hid), dt)
            state["w"] = _randn(gen, (n, hid), dt, hid ** -0.5)
            state["out"] = _randn(gen, (case["batch"], case["rows"], n), dt)   # the tiles of earlier steps
            state["bias"] = _randn(gen, (n,), dt) if case["bias"] else None
        else:
            state["x"] = _randn(gen, (case["batch"], case["rows"], n), dt)
            state["w"] = _randn(gen, (hid, n), dt, n ** -0.5)
            state["init"] = _randn(gen, (hid,) if case["for_cache"] else (case["batch"], case["rows"], hid), dt)
        return state
    if kind in ("layer", "video"):
        dt, D, hid, H = _DTYPES[case["dtype"]], case["dim"], case["hidden"], case["heads"]
        own = case.get("own_heads", H)
        w = BlockWeights(*(_randn(gen, (own * D, hid), dt, hid ** -0.5) for _ in range(3)),
                         _randn(gen, (hid, own * D), dt, (H * D) ** -0.5))
        if kind == "layer":
            B, S = case["batch"], case["rows"]
            nb = S // BLOCK
            masks = _packed([_image_flags(gen, nb, H, nb, case["density"], case["text"]) for _ in range(B)])
            block = SparseDiTAttentionBlock(w, H, D, B, S, 0, own, device=_dev(), dtype=dt)
            # the storage of the GEMM work lists, which a layer keeps from its first step on
            block._q_list = prepare_gemm_q_list(B, S, own * D, H, masks[0], masks[2], 0, head_dim=D)
            block._o_list = prepare_gemm_o_list(B, S, own * D, H, masks[0], masks[2], 0, head_dim=D)
        else:
            B, S = 1, BLOCK * (case["text"] + case["frames"] * case["frame_blocks"])
            masks = _packed([_video_flags(gen, case["text"], case["frames"], case["frame_blocks"], H, case["density"])])
            block = UlyssesSparseDiTAttentionBlock(w, H, D, S, 0, 1, _dev(), dt)
        # a sampler in the middle of its steps: the cache and the outputs of skipped q-blocks hold earlier values
        block.cache.copy_(_randn(gen, tuple(block.cache.shape), dt))
        block.attn.copy_(_randn(gen, tuple(block.attn.shape), dt))
        return {"case": case, "block": block, "x": _randn(gen, (B, S, hid), dt), "masks": masks}
    if kind == "select":
        B, H, n = case["batch"], case["heads"], case["blocks"]
        # pooled q k^T / sqrt(d) of the blocks: near the diagonal higher, as neighbouring blocks attend to each other
        score = torch.randn(B, H, n, n, generator=gen, device=_dev())
        pos = torch.arange(n, device=_dev(), dtype=torch.float32)
        score += 2.0 * torch.exp(-(pos[:, None] - pos[None, :]).abs() / (0.05 * n + 1.0))
        return {"case": case, "score": score}
    flags = [_image_flags(gen, case["blocks"], case["heads"], case["blocks"], case["density"], case["text"])
             for _ in range(case["batch"])]
    return {"case": case, "q_flags": _flat([f[0] for f in flags]), "kv_flags": _flat([f[1] for f in flags])}


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "attention":
        return state["wrapper"].run(state["q"], state["k"], state["v"], *state["masks"], case["full"],
                                    lse=state["lse"], return_lse=case["lse"])
    if kind == "gemm_q":
        return fo.flashomni_gemm(state["x"], state["w"], case["heads"], *state["masks"], 0, state["bias"],
                                 out=state["out"])
    if kind == "gemm_o":
        return fo.flashomni_gemm_reduction(state["x"], state["w"], case["heads"], *state["masks"], 0, state["init"],
                                           is_for_cache=case["for_cache"], head_dim=case["dim"])
    if kind in ("layer", "video"):
        y = state["block"].forward(state["x"], *state["masks"])
        return y, state["block"].attn
    if kind == "select":
        return fo.select_blocks(state["score"], case["text"], 0.2, 0.3)
    return fo.segment_packbits(*state["q_flags"], bitorder="little") + fo.segment_packbits(*state["kv_flags"],
                                                                                          bitorder="little")


# ------------------------------------------------------------------------------------------------ what a pass needs
def _image_shares(n_q, n_kv, density, text):
    """(expected share of active (q-block, head) pairs, expected kept kv-blocks of one request and head)."""
    tq, tk = min(n_q, text), min(n_kv, text)
    active = (tq + (n_q - tq) * density) / n_q
    image_kv = n_kv - tk
    kept_text_row = tk + image_kv * density
    diag = 1 if image_kv > 0 else 0
    kept_image_row = tk + diag + max(0, image_kv - diag) * density
    return active, tq * kept_text_row + (n_q - tq) * density * kept_image_row


def work(case):
    kind, two = case["kind"], 2
    if kind == "attention":
        flops = nbytes = 0.0
        kv_size = 1 if case["kv_dtype"] == "e4m3" else two
        for n in _lens(case):
            nb = -(-n // BLOCK)
            active, kept = (1.0, nb * nb) if case["full"] else _image_shares(nb, nb, case["density"], case["text"])
            flops += 4.0 * case["heads"] * case["dim"] * kept * (n / nb) ** 2
            nbytes += n * case["dim"] * (case["heads"] * two * (active + 1.0) + 2 * case["kv_heads"] * kv_size)
            nbytes += 0 if case["full"] else nb * case["kv_heads"] * (nb + 1) / 8
        return {"bytes": nbytes, "flops": flops}
    if kind in ("gemm_q", "gemm_o"):
        rows, n, hid = case["batch"] * case["rows"], case["heads"] * case["dim"], case["hidden"]
        nb = case["rows"] // BLOCK
        active = _image_shares(nb, nb, case["density"], case["text"])[0]
        if kind == "gemm_q":
            return {"bytes": two * (rows * hid + n * hid + rows * n * active), "flops": 2.0 * rows * n * hid * active}
        share = 1.0 - active if case["for_cache"] else active
        init = hid if case["for_cache"] else rows * hid
        return {"bytes": two * (rows * n * share + n * hid + init + rows * hid), "flops": 2.0 * rows * n * hid * share}
    if kind in ("layer", "video"):
        D, hid, own = case["dim"], case["hidden"], case.get("own_heads", case["heads"])
        if kind == "layer":
            rows, nb = case["batch"] * case["rows"], case["rows"] // BLOCK
            active, kept = _image_shares(nb, nb, case["density"], case["text"])
            kept *= case["batch"]
        else:
            nb = case["text"] + case["frames"] * case["frame_blocks"]
            rows, active = nb * BLOCK, 1.0
            f, fb, t, d = case["frames"], case["frame_blocks"], case["text"], case["density"]
            local = (3 * f - 2) * fb * fb                      # same frame and its neighbours
            kept = nb * t + local + ((f * fb) ** 2 - local + t * f * fb) * d
        n = own * D
        flops = 2.0 * rows * n * hid * (2 + 2 * active) + 4.0 * own * D * BLOCK * BLOCK * kept
        # hidden state, weights, cache in; output, attention output out
        nbytes = two * (rows * hid * 3 + 4.0 * n * hid + rows * n * active) + case["heads"] * kept / 8
        return {"bytes": nbytes, "flops": flops}
    B, H, n = case["batch"], case["heads"], case["blocks"]
    bits = B * H * n * (n + 1)
    if kind == "select":
        return {"bytes": 4.0 * B * H * n * n + bits / 8, "flops": 0.0}
    return {"bytes": bits + bits / 8, "flops": 0.0}


def tolerance(case):
    if case["kind"] in ("select", "pack"):
        return "exact"
    # Four times what the path shows against itself in 64 bits. bf16: attention 0.0024, GEMMs 0.0012-0.0017, active
    # blocks of a layer's attention 0.0035 (q, k, v and P rounded one after the other), single values up to 0.03 (GEMMs
    # 0.004). f16 has three bits more: attention 0.0003, single values 0.004.
    if case["dtype"] == "f16":
        return {"rel": 2e-3, "max": 3e-2}
    if case["kind"] in ("gemm_q", "gemm_o"):
        return {"rel": 7e-3, "max": 2e-2}
    return {"rel": 1e-2, "max": 1.2e-1}
