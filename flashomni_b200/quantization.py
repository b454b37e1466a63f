"""Bit packing of the block masks (drop-in for flashomni/quantization.py:68-159)."""

from __future__ import annotations

from typing import Tuple

import torch

from . import _native


def _little(bitorder: str) -> int:
    if bitorder not in ("big", "little"):
        raise ValueError(f"bitorder must be 'big' or 'little', got {bitorder!r}")
    return 1 if bitorder == "little" else 0


def _as_bytes(x: torch.Tensor) -> torch.Tensor:
    x = x.contiguous().view(-1)
    if x.dtype == torch.bool:
        return x.view(torch.uint8)
    if x.dtype in (torch.uint8, torch.int8):
        return x.view(torch.uint8)
    return (x != 0).view(torch.uint8)


def packbits(x: torch.Tensor, bitorder: str = "big") -> torch.Tensor:
    """Packs a 1-D binary-valued tensor into bits, same semantics as numpy.packbits
    (reference: flashomni/quantization.py:68-99)."""
    little = _little(bitorder)
    _native.require_cuda(x)
    xb = _as_bytes(x)
    n = xb.numel()
    y = torch.empty((n + 7) // 8, dtype=torch.uint8, device=x.device)
    with torch.cuda.device(x.device):
        rc = _native.load().fo_packbits(_native.ptr(xb), n, little, _native.ptr(y),
                                        _native.current_stream(x.device))
    _native.check(rc, "packbits")
    return y


def segment_packbits(x: torch.Tensor, indptr: torch.Tensor, bitorder: str = "big") -> Tuple[torch.Tensor, torch.Tensor]:
    """Packs each segment x[indptr[i]:indptr[i+1]] separately; returns (y, new_indptr) with
    new_indptr[i+1]-new_indptr[i] == ceil(len_i/8) (reference: flashomni/quantization.py:102-159,
    including its one wait of the host, which here is for the packed bytes as well as for their number)."""
    little = _little(bitorder)
    # the usual call in one native function; it returns None for anything else
    r = _native.host().segment_packbits(x, indptr, little)
    if r is not None:
        if type(r) is int:
            _native.check(r, "segment_packbits")
        return r
    _native.require_cuda(x)
    n_seg = len(indptr) - 1
    refused = False
    # The usual call: the byte indptr, its total and the packed bytes in one launch and one wait. The output is allocated
    # for the most that these segments can need and shortened; anything else takes the general path below.
    if (indptr.dim() == 1 and 1 <= n_seg <= 1024 and indptr.dtype in (torch.int32, torch.int64)
            and indptr.device == x.device and 0 < x.numel() < 1 << 33):
        device = x.device
        xb, ip = _as_bytes(x), indptr.contiguous()
        capacity = (xb.numel() + 7 * n_seg) // 8
        y = torch.empty(capacity, dtype=torch.uint8, device=device)
        indptr_new = torch.empty(n_seg + 1, dtype=torch.int32, device=device)
        words = torch.empty(_native.PACK_WORDS, dtype=torch.int64, pin_memory=True)
        with torch.cuda.device(device):
            rc = _native.load().fo_segment_packbits_polled(
                xb.data_ptr(), xb.numel(), ip.data_ptr(), int(ip.dtype == torch.int64), n_seg, capacity, little, y.data_ptr(),
                indptr_new.data_ptr(), words.data_ptr(), words.numel(), _native.current_stream(device))
        _native.check(rc, "segment_packbits")
        nbytes = int(words[0])
        if nbytes >= 0:
            y = y.narrow(0, 0, nbytes)
            # segments that cover little of x: the result does not keep the rest of the allocation alive (below a megabyte,
            # the allocator's own granularity, the copy would cost more than it frees)
            if capacity - nbytes > max(nbytes, 1 << 20):
                y = y.clone()
                torch.cuda.current_stream(device).synchronize()
            return y, indptr_new
        refused = True
    seglen = indptr[1:] - indptr[:-1]
    packed_len = (seglen + 7) // 8
    indptr_new = torch.zeros(len(indptr), dtype=indptr.dtype, device=indptr.device)
    torch.cumsum(packed_len, 0, dtype=indptr.dtype, out=indptr_new[1:])
    # No segment may leave x. An indptr on the device is taken to ascend here, as its ends come with the size at no further
    # wait; every entry is looked at on the host, and after the kernel above has found something wrong.
    if indptr.is_cuda and not refused:
        output_nnzs, lo, hi = (int(v) for v in torch.cat((indptr_new[-1:], indptr[:1], indptr[-1:])).tolist())
    else:
        output_nnzs = int(indptr_new[-1].item())
        v = indptr.tolist() if n_seg <= 64 else indptr.aminmax()   # (a few entries: cheaper than a tensor op)
        lo, hi = int(min(v)), int(max(v))
    if lo < 0 or hi > x.numel():   # (an empty segment may lie anywhere)
        if bool(((seglen > 0) & ((indptr[:-1] < 0) | (indptr[1:] > x.numel()))).any()):
            raise ValueError(f"segment_packbits: a segment leaves the {x.numel()} values of x")
    device = x.device
    indptr32 = indptr.to(device=device, dtype=torch.int32).contiguous()
    indptr_new = indptr_new.to(device=device, dtype=torch.int32).contiguous()
    xb = _as_bytes(x)
    y = torch.empty(output_nnzs, dtype=torch.uint8, device=device)
    with torch.cuda.device(device):
        rc = _native.load().fo_segment_packbits(_native.ptr(xb), _native.ptr(indptr32), _native.ptr(indptr_new),
                                                len(indptr) - 1, output_nnzs, little, _native.ptr(y),
                                                _native.current_stream(device))
    _native.check(rc, "segment_packbits")
    return y, indptr_new
