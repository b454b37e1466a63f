"""GPU: GEMM-O with the cached contribution as init, whose slabs come in by TMA: an odd number of column blocks (a single
last tile), row blocks without any active head (y = init), more tiles than CTAs, one tile, result written over the init."""

import numpy as np
import pytest
import torch

import flashomni_b200 as fo
from flashomni_b200 import workloads as wl
from helpers import dev, masks_to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,rows,heads,hidden,in_place", [
    (1, 128, 1, 128, False), (1, 256, 3, 384, True), (2, 384, 2, 640, False), (1, 2688, 4, 1920, False), (3, 1024, 6, 2304, True)])
def test_cached_contribution(cuda_device, dtype, batch, rows, heads, hidden, in_place):
    D, nb = 128, rows // 128
    rng = np.random.default_rng(rows + heads)
    flags = [(rng.random((nb, heads)) < 0.5).astype(np.uint8) for _ in range(batch)]
    flags[0][0] = 0                      # a row block of skipped heads only
    m = wl.pack_masks(flags, [f[:, :, None] for f in flags])
    si, _, ip, _ = masks_to_device(m, cuda_device)
    x, w = wl.randn_bf16((batch, rows, heads * D), 1, dtype=dtype), wl.randn_bf16((hidden, heads * D), 2, dtype=dtype)
    w = (w.float() * (heads * D) ** -0.5).to(dtype)
    cache = wl.randn_bf16((batch, rows, hidden), 3, dtype=dtype)
    c = dev(cache, cuda_device).clone()
    for _ in range(2):   # (the second launch starts from the tile cursor that the first one put back)
        if in_place:
            c = dev(cache, cuda_device).clone()
        y = fo.flashomni_gemm_reduction(dev(x, cuda_device), dev(w, cuda_device), heads, si, ip, 0, c, head_dim=D,
                                        out=c if in_place else None)
    mask = torch.from_numpy(np.stack(flags)).repeat_interleave(128, 1).repeat_interleave(D, 2)
    ref = (x.double() * mask) @ w.double().T + cache.double()
    # sums in fp32 and one rounding to 16 bits: half a unit in the last place of the result, and 1e-5 for the sum
    tol = ref.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) + 1e-4
    assert ((y.cpu().double() - ref).abs() <= tol).all()
    none = ~torch.from_numpy(np.stack(flags)).bool().any(2)
    assert torch.equal(y.cpu().view(batch, nb, 128, hidden)[none], cache.view(batch, nb, 128, hidden)[none])
