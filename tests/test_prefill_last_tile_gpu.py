"""tcgen05 prompt attention where V comes late: the last key tile's product must be waited for, not the one before it.

Scores that do not grow from tile to tile (queries of zeros) pass over the only other wait on a product, and a V that is not in L2 beside a
K that is lets the softmax of the last tile finish before the product of the tile before it."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"


@pytest.mark.parametrize("H,G,d", [(16, 2, 128), (28, 4, 128), (8, 2, 64)])
@pytest.mark.parametrize("tokens,start", [(129, 0), (268, 0), (40, 230), (130, 300), (9, 500)])
def test_last_tile_is_complete(H, G, d, tokens, start):
    from qwen_decoder_b200 import kernels
    page, n = 16, start + tokens
    pages = (n + page - 1) // page
    g = torch.Generator(device=DEV).manual_seed(n + d)
    kv = torch.empty(pages, 2, G, page, d, device=DEV).normal_(generator=g).bfloat16()
    table = torch.randperm(pages, device=DEV, generator=g).to(torch.int32).view(1, -1)
    cu = torch.tensor([0, tokens], dtype=torch.int32, device=DEV)
    first = torch.tensor([start], dtype=torch.int32, device=DEV)
    k, v = (kv[table[0].long(), i].transpose(0, 1).reshape(G, -1, d)[:, :n].double().repeat_interleave(H // G, dim=0) for i in (0, 1))
    later = torch.arange(n, device=DEV) > (start + torch.arange(tokens, device=DEV))[:, None]
    flush = torch.empty(1 << 28, dtype=torch.int8, device=DEV)          # twice the L2
    for scale in (0.0, 1.0):
        q = (scale * torch.empty(tokens, H * d, device=DEV).normal_(generator=g)).bfloat16()
        s = torch.einsum("thd,hnd->htn", q.double().view(tokens, H, d), k) * d ** -0.5
        want = torch.einsum("htn,hnd->thd", s.masked_fill(later, float("-inf")).softmax(-1), v)
        kept = None
        for _ in range(20):
            out = torch.empty(tokens, H * d, dtype=torch.bfloat16, device=DEV)
            flush.zero_()
            kv[:, 0].float().sum()                                       # K is in L2, V is not
            kernels.prefill_attention_tc5(q, H * d, out, kv, table, cu, first, 1, tokens, H, G, d, page, d ** -0.5, 0)
            kept = out if kept is None else kept
            assert torch.equal(out, kept)
        assert kernels.prefill_attention_tc5_status() == 0
        # weights and results are rounded to bfloat16, 2^-9 each; a product that is missing leaves a tenth or more of the result out
        err = (kept.double().view(tokens, H, d) - want).norm(dim=-1) / want.norm(dim=-1)
        assert float(err.max()) <= 2.0 ** -6
