"""Decode attention whose CTAs go by the requests' lengths: ragged batches against one unsplit call through the kernel that shares
nothing.  Few long requests among many short ones, all equal, all short (more CTAs than the grid holds: equal shares), windows."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"

LENGTHS = {
    "two": lambda T: [3, 2000] + [17] * (T - 2),
    "rising": lambda T: [1 + 37 * i % 1999 for i in range(T)],
    "one_long": lambda T: [40] * (T - 1) + [4095],
    "short": lambda T: [1 + 16 * (i % 3) for i in range(T)],
    "equal": lambda T: [777] * T,
}


@pytest.mark.parametrize("T", [2, 7, 33, 128])
@pytest.mark.parametrize("kind", list(LENGTHS))
@pytest.mark.parametrize("H,G,d,page,window,splits", [(16, 2, 128, 16, 0, 4), (28, 4, 128, 32, 0, 1), (4, 4, 64, 16, 0, 64), (8, 2, 64, 64, 300, 3)])
def test_shares_by_length(T, kind, H, G, d, page, window, splits, monkeypatch):
    from qwen_decoder_b200 import kernels
    lens = LENGTHS[kind](T)
    g = torch.Generator(device=DEV).manual_seed(T + splits)
    pages = [(n + page - 1) // page for n in lens]
    perm = torch.randperm(sum(pages), device=DEV, generator=g).to(torch.int32)
    table = torch.full((T, max(pages)), -1, dtype=torch.int32, device=DEV)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = perm[at:at + n]
        at += n
    kv = torch.empty(at, 2, G, page, d, device=DEV).normal_(generator=g).bfloat16()
    q = torch.empty(T, H * d, device=DEV).normal_(generator=g).bfloat16()
    req = torch.arange(T, dtype=torch.int32, device=DEV)
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    call = lambda out, s, by: kernels.decode_attention(q, H * d, out, kv, table, req, pos, T, H, G, d, page, d ** -0.5, window, s, by_length=by)
    got, again, want = (torch.empty_like(q) for _ in range(3))
    assert kernels.decode_by_tma(T, d) == (True, True)
    call(got, splits, True)
    call(again, splits, True)                # the tickets are zero again
    monkeypatch.setattr(kernels, "_DECODE_TMA", False)
    call(want, 1, False)
    assert kernels.library("attention_flash").qd_decode_attention_tma_status() == 0
    assert torch.equal(got, again)
    # both round weights and results to bfloat16: four times 2^-9 of the largest value
    err = float((got.float() - want.float()).abs().max())
    assert err <= 2.0 ** -7 * float(kv[:, 1].float().abs().max()), err
