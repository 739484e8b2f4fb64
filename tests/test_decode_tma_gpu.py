"""Decode attention fed by TMA copies against the form fed by cp.async: which of the two a step takes must not show in its results.
Ragged batches, one chunk, shares without a chunk, windows; and against float64, each request by its own values."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"

LENGTHS = {
    "two": lambda T: [3, 2000] + [17] * (T - 2),
    "rising": lambda T: [1 + 37 * i % 1999 for i in range(T)],
    "one_long": lambda T: [40] * (T - 1) + [4095],
    "equal": lambda T: [777] * T,
}


@pytest.mark.parametrize("T", [2, 7, 33])
@pytest.mark.parametrize("kind", list(LENGTHS))
@pytest.mark.parametrize("H,G,d,page,window,splits", [(16, 2, 128, 16, 0, 4), (28, 4, 128, 32, 0, 1), (4, 4, 64, 16, 0, 64), (8, 2, 64, 64, 300, 3)])
def test_both_feeds_agree(T, kind, H, G, d, page, window, splits, monkeypatch):
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
    call = lambda out: kernels.decode_attention(q, H * d, out, kv, table, req, pos, T, H, G, d, page, d ** -0.5, window, splits)
    got, again, other = (torch.empty_like(q) for _ in range(3))
    assert kernels.decode_by_tma(d)
    call(got)
    call(again)                              # the tickets are zero again
    monkeypatch.setattr(kernels, "_DECODE_TMA", False)
    call(other)
    assert kernels.library("attention_flash").qd_decode_attention_tma_status() == 0
    assert torch.equal(got, again) and torch.equal(got, other)
    for t, n in enumerate(lens):
        rows = kv[table[t, :pages[t]].long()].double()                   # [pages, 2, G, page, d]
        k, v = (rows[:, j].transpose(0, 1).reshape(G, -1, d)[:, :n].repeat_interleave(H // G, dim=0) for j in (0, 1))
        s = torch.einsum("hd,hnd->hn", q[t].double().view(H, d), k) * d ** -0.5
        if window:
            s[:, :max(0, n - window)] = float("-inf")
        want = torch.einsum("hn,hnd->hd", s.softmax(-1), v)
        # weights and results are rounded to bfloat16, 2^-9 each: a sum of n rounded weights times values is off by a small share of
        # that; a lost, doubled or shifted share of the keys moves it by the size of the result itself
        err = float((got[t].double().view(H, d) - want).norm() / want.norm())
        assert err <= 2.0 ** -7, (t, n, err)
