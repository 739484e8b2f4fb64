"""Decode attention with its CTAs dealt out by the tokens' lengths: the list against the rule it states, the attention against float64 at
lengths that differ a lot, end inside chunks and pages, fill a batch with padding, or need more shares than one round of the combine."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"


def rule(keys, n_list, least=10, most=64):
    """Shares of each token: of at most S chunks of 16 keys, S the smallest that needs no more than ``n_list``."""
    chunks = [(k + 15) // 16 for k in keys]
    S = max(least, -(-max(chunks) // most))
    while sum(-(-c // S) for c in chunks) > n_list:
        S += 1
    return [[(c * s // n, c * (s + 1) // n) for s in range(n)] for c in chunks for n in (-(-c // S),)]


CASES = {
    "short": ([1, 2, 16], 0), "one long": ([40, 4095, 17, 1], 0), "equal": ([2049] * 33, 31),
    "rising": ([1 + 131 * i for i in range(23)], 9), "many": ([1 + 37 * i % 700 for i in range(200)], 0),
    "as many as there may be": ([1 + i % 50 for i in range(1024)], 0), "very long": ([30000, 300], 0), "padded": ([161] + [5] * 16, 15),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("H,G,d,page", [(16, 2, 128, 16), (28, 4, 128, 32), (8, 8, 64, 16)])
def test_shares_by_length(name, H, G, d, page):
    from qwen_decoder_b200 import kernels
    keys, pads = CASES[name]
    n, T = len(keys), len(keys) + pads
    g = torch.Generator(device=DEV).manual_seed(n + d)
    need = [-(-k // page) for k in keys]
    order = torch.randperm(sum(need), device=DEV, generator=g).to(torch.int32)
    table = torch.full((T, max(need)), -1, dtype=torch.int32, device=DEV)
    at = 0
    for i, c in enumerate(need):
        table[i, :c] = order[at:at + c]
        at += c
    table[n:] = table[0]
    pos = torch.tensor([k - 1 for k in keys] + [keys[0] - 1] * pads, dtype=torch.int32, device=DEV)
    slot = torch.tensor([3] * n + [at * page] * pads, dtype=torch.int32, device=DEV)
    kv = torch.empty(at, 2, G, page, d, device=DEV).normal_(generator=g).bfloat16()
    q = torch.empty(T, H * d, device=DEV).normal_(generator=g).bfloat16()
    q[n:] = q[0]
    assert kernels.decode_shares_supported(q.dtype, T, H, G, d, page, max(keys))
    shares = kernels.decode_shares(pos, slot, at * page, T, G, d)
    rows = shares.cpu().numpy().view("uint16").reshape(-1, 8).astype(int)       # token, share, first, end, keys (2), shares, copies
    want = rule(keys, len(rows))
    flat = [[t, s, a, b, keys[t] & 65535, keys[t] >> 16, len(w), 0 if t else pads] for t, w in enumerate(want) for s, (a, b) in enumerate(w)]
    assert rows[:len(flat)].tolist() == flat and not rows[len(flat):].any()
    for fresh in (True, False):                          # the second launch: the tickets are zero again
        out = torch.full_like(q, float("nan"))
        kernels.decode_attention_shares(q, H * d, out, kv, table, T, H, G, d, page, d ** -0.5, shares, fresh)
        assert kernels.library("attention_flash").qd_decode_attention_tma_status() == 0
        for t in range(0, n, max(1, n // 40)):
            k, v = (kv[table[t, :need[t]].long(), i].double().transpose(0, 1).reshape(G, -1, d)[:, :keys[t]].repeat_interleave(H // G, 0)
                    for i in (0, 1))
            p = torch.softmax((k @ q[t].double().view(H, d, 1)).squeeze(-1) * d ** -0.5, -1)[:, None]
            ref = (p @ v).view(-1)
            # probabilities rounded to bfloat16 beside a sum of the unrounded ones, the result rounded; 1e-4: exponentials and sums
            assert ((out[t].double() - ref).abs() <= 2.0 ** -8 * (p @ v.abs()).view(-1) + 2.0 ** -8 * ref.abs() + 1e-4).all(), (name, t)
        assert (out[n:] == out[0]).all()


def test_what_has_no_shares():
    from qwen_decoder_b200 import kernels
    ok = lambda **k: kernels.decode_shares_supported(**{**dict(dtype=torch.bfloat16, n_tokens=20, H=8, G=2, d=128, page_size=16, max_keys=99), **k})
    assert ok() and not ok(n_tokens=1) and not ok(n_tokens=1025) and not ok(d=96) and not ok(dtype=torch.float32) and not ok(max_keys=1 << 20)
    assert not ok(page_size=24) and not ok(H=64)


def test_when_shares_by_length_pay():
    from qwen_decoder_b200.engine.batch import uneven_contexts
    assert not uneven_contexts([2048] * 64, 64) and uneven_contexts([2048] * 40, 64) and uneven_contexts([500, 4000, 900], 3)
    assert not uneven_contexts([], 0) and not uneven_contexts([4000], 1) and not uneven_contexts([0, 0], 2)
    assert not uneven_contexts([299, 20, 30], 3) and uneven_contexts([319, 20, 30], 3)


def test_shares_of_equal_contexts():
    from qwen_decoder_b200.parts.attention import decode_splits
    assert [decode_splits(48, k, 592) for k in (1, 160, 300, 319, 320, 330, 2048)] == [1, 1, 1, 1, 2, 3, 12]
    assert decode_splits(700, 4000, 592) == 1 and decode_splits(2, 1 << 20, 592) == 64
