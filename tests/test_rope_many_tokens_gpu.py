"""Rotation and cache write of many tokens (a thread takes several heads) against the same call on a few tokens at a time."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"


@pytest.mark.parametrize("T", [1536, 8201])
@pytest.mark.parametrize("H,G,d,page", [(16, 2, 128, 16), (28, 4, 128, 32), (30, 2, 16, 16), (5, 5, 80, 16), (4, 3, 48, 8)])
@pytest.mark.parametrize("bias,write", [(True, True), (False, True), (True, False)])
def test_many_tokens_as_few(T, H, G, d, page, bias, write):
    from qwen_decoder_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(T + d)
    qkv = torch.empty(T, (H + 2 * G) * d, device=DEV).normal_(generator=g).bfloat16()
    b = torch.empty((H + 2 * G) * d, device=DEV).normal_(generator=g) if bias else None
    ang = torch.empty(2 * T, d // 2, device=DEV).uniform_(0, 6, generator=g)
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    pos = torch.randperm(2 * T, device=DEV, generator=g)[:T].to(torch.int32)
    pages = (T + page - 1) // page + 2
    slots = torch.randperm(pages * page, device=DEV, generator=g)[:T].to(torch.int32)
    got, kv = qkv.clone(), torch.zeros(pages, 2, G, page, d, dtype=torch.bfloat16, device=DEV)
    want, kv2 = qkv.clone(), torch.zeros_like(kv)
    call = lambda x, p, s, cache: kernels.rope_kv_write_biased(x, b, H, G, d, d, 1, cos, sin, p, cache if write else None, s, page, write)
    call(got, pos, slots, kv)
    for i in range(0, T, 700):
        call(want[i:i + 700], pos[i:i + 700].contiguous(), slots[i:i + 700].contiguous(), kv2)
    # what is left in the rows of k and v when they go to the cache is nobody's business
    n = H * d if write else (H + 2 * G) * d
    assert torch.equal(got[:, :n], want[:, :n]) and torch.equal(kv, kv2)
