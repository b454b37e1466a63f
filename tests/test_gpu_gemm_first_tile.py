"""Calls that build their list themselves: every CTA of the GEMM kernel works its first tile out of the mask, the rest come from
the list. The same tiles with the same order of additions as with a prepared list, so the results are the same bits."""
import pytest
import torch

from flashomni_b200.gemm import flashomni_gemm, flashomni_gemm_reduction, prepare_gemm_o_list, prepare_gemm_q_list

pytestmark = pytest.mark.gpu


def _mask(batch, nq, heads, density, gen):
    flags = torch.rand(batch, nq * heads, generator=gen) < density
    pad = (-flags.shape[1]) % 8
    bits = torch.nn.functional.pad(flags, (0, pad)).view(batch, -1, 8).to(torch.int32)
    packed = (bits << torch.arange(8)).sum(-1).to(torch.uint8)
    indptr = torch.arange(batch + 1, dtype=torch.int32) * packed.shape[1]
    return packed.reshape(-1).cuda(), indptr.cuda()


# rows, heads, local heads, first local head, text tokens, density: one tile, fewer and more tiles than CTAs, 191..193 row
# blocks (the last thread that has one, and one too many), a window of the heads, 64 and 65 local heads, empty and full masks
SHAPES = [(1, 128, 2, 2, 0, 0, 0.7), (1, 128, 65, 64, 1, 0, 0.5), (1, 256, 65, 65, 0, 0, 0.5), (2, 384, 24, 24, 0, 100, 0.5), (1, 1024, 8, 3, 4, 512, 0.3),
          (3, 1536, 12, 12, 0, 0, 0.9), (1, 191 * 128, 3, 3, 0, 0, 0.5), (2, 96 * 128, 5, 4, 1, 0, 0.4), (1, 193 * 128, 3, 2, 0, 0, 0.6),
          (1, 4608, 24, 24, 0, 0, 0.0), (1, 4608, 24, 24, 0, 0, 1.0), (2, 4608, 24, 24, 0, 0, 0.05)]


@pytest.mark.parametrize("batch,rows,heads,local,first,text,density", SHAPES)
def test_same_bits_as_with_a_prepared_list(batch, rows, heads, local, first, text, density):
    gen = torch.Generator().manual_seed(rows + heads)
    info, indptr = _mask(batch, (rows + text) // 128 + 1, heads, density, gen)
    hidden, width = 256, local * 128
    x = torch.randn(batch, rows, hidden, generator=gen).to(torch.bfloat16).cuda()
    w = torch.randn(width, hidden, generator=gen).to(torch.bfloat16).cuda()
    q_list = prepare_gemm_q_list(batch, rows, width, heads, info, indptr, text, head_begin=first, head_dim=128)
    want = torch.zeros(batch, rows, width, dtype=torch.bfloat16, device="cuda")
    got = torch.zeros_like(want)
    flashomni_gemm(x, w, heads, info, indptr, text, None, out=want, head_begin=first, head_dim=128, worklist=q_list)
    flashomni_gemm(x, w, heads, info, indptr, text, None, out=got, head_begin=first, head_dim=128)
    assert torch.equal(got, want)

    a = torch.randn(batch, rows, width, generator=gen).to(torch.bfloat16).cuda()
    wo = torch.randn(hidden, width, generator=gen).to(torch.bfloat16).cuda()
    full, row = (torch.randn(*shape, generator=gen).to(torch.bfloat16).cuda() for shape in ((batch, rows, hidden), (hidden,)))
    for for_cache, inits in ((False, (None, full)), (True, (None, row))):
        for init in inits:
            o_list = prepare_gemm_o_list(batch, rows, width, heads, info, indptr, text, is_for_cache=for_cache,
                                         head_begin=first, head_dim=128)
            y = [flashomni_gemm_reduction(a, wo, heads, info, indptr, text, init, is_for_cache=for_cache, head_begin=first,
                                          head_dim=128, worklist=lst) for lst in (o_list, None)]
            assert torch.equal(y[0], y[1])
