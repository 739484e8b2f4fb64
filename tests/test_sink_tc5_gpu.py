"""The tcgen05 form of the attention with sinks, blocks, gates and strided rows against float64, beside the mma.sync form: portions that
end inside tiles, histories, blocks that end inside tiles, and rows of the cache that hold no numbers."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"


def setup(lengths, starts, H, G, d, page, seed=0):
    g = torch.Generator(device=DEV).manual_seed(sum(lengths) + d + seed)
    rnd = lambda *s: torch.empty(s, device=DEV).normal_(generator=g)
    need = [-(-(s + n) // page) for n, s in zip(lengths, starts)]
    pages = sum(need) + 1                                      # the last one belongs to nobody
    kv = rnd(pages, 2, G, page, d).bfloat16()
    order = torch.randperm(pages - 1, device=DEV, generator=g).to(torch.int32)
    table = torch.full((len(lengths), max(need)), pages - 1, dtype=torch.int32, device=DEV)
    at = 0
    for r, n in enumerate(need):
        table[r, :n] = order[at:at + n]
        at += n
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    return g, rnd, kv, table, cu, torch.tensor(starts, dtype=torch.int32, device=DEV)


def reference(q, kv, table, lengths, starts, H, G, d, page, scale, window, chunk, sinks, gate, gate_elem, out_scale):
    out, t = [], 0
    for r, (n, s) in enumerate(zip(lengths, starts)):
        total = s + n
        rows = kv[table[r].long()].double()                    # [pages, 2, G, page, d]
        k, v = (rows[:, i].transpose(0, 1).reshape(G, -1, d)[:, :total].repeat_interleave(H // G, 0) for i in (0, 1))
        qq = q[t:t + n].double().view(n, H, d).transpose(0, 1)
        pos = torch.arange(s, total, device=DEV)[:, None]
        key = torch.arange(total, device=DEV)[None]
        seen = key <= pos
        if window:
            seen &= key > pos - window
        if chunk:
            seen &= key // chunk == pos // chunk
        sc = (qq @ k.transpose(1, 2) * scale).masked_fill(~seen, float("-inf"))
        if sinks is not None:
            sc = torch.cat([sc, sinks.double().view(H, 1, 1).expand(H, n, 1)], -1)
        w = sc.softmax(-1)[..., :total]
        y = (w @ v.masked_fill(~seen.any(0)[None, :, None], 0.0)).transpose(0, 1).reshape(n, H * d) * out_scale
        if gate is not None:
            z = torch.sigmoid(gate[t:t + n].double())
            y = y * (z if gate_elem else z.repeat_interleave(d, 1))
        out.append(y)
        t += n
    return torch.cat(out)


CASES = [
    ([130], [0], 8, 2, 128, 16, 0, 0, True, "elem"),
    ([300, 65], [0, 200], 4, 2, 64, 16, 0, 100, False, "elem"),
    ([64, 200, 40], [30, 0, 513], 8, 1, 128, 32, 0, 256, True, "head"),
    ([257], [1000], 16, 2, 128, 16, 70, 0, False, None),
    ([90, 333], [7, 129], 7, 7, 64, 16, 200, 150, True, "elem"),
]


@pytest.mark.parametrize("lengths,starts,H,G,d,page,window,chunk,sink,gated", CASES)
@pytest.mark.parametrize("nan", [False, True])
def test_against_float64(lengths, starts, H, G, d, page, window, chunk, sink, gated, nan, monkeypatch):
    from qwen_decoder_b200 import kernels
    g, rnd, kv, table, cu, start = setup(lengths, starts, H, G, d, page)
    T = sum(lengths)
    q = rnd(T, H * d).bfloat16()
    sinks = 2 * rnd(H) if sink else None
    wide = rnd(T, H * d + 4)
    gate = None if gated is None else wide[:, :H * d] if gated == "elem" else wide[:, :H]
    if nan:                                                    # what lies behind a request's keys, and the page that is nobody's
        kv[-1] = float("nan")
        for r, (n, s) in enumerate(zip(lengths, starts)):
            last, used = int(table[r, (s + n - 1) // page]), (s + n - 1) % page + 1
            kv[last, :, :, used:] = float("nan")
    args = (kv, table, cu, start, len(lengths), T, H, G, d, d, page, d ** -0.5, window, sinks)
    extra = dict(chunk=chunk, gate=gate, gate_elem=gated == "elem", out_scale=0.8)
    want = reference(q, kv, table, lengths, starts, H, G, d, page, d ** -0.5, window, chunk, sinks, gate, gated == "elem", 0.8)
    err = []
    for tc5 in (False, True):
        monkeypatch.setattr(kernels, "SINK_TC5", tc5)
        room = torch.full((T, H * d + 8), 7.0, dtype=torch.bfloat16, device=DEV)
        kernels.sink_attention_mma(q, room[:, :H * d], *args, **extra)
        assert bool((room[:, H * d:] == 7.0).all())
        err.append(float((room[:, :H * d].double() - want).norm() / want.norm()))
    assert kernels.prefill_attention_tc5_status() == 0
    # both round the result to bfloat16 and keep weights to 2^-17: no further off than the other form, but for the order of sums
    assert err[1] <= 1.02 * err[0] + 1e-5 and err[1] <= 2.0 ** -8, err


def test_sinks_far_from_the_scores(monkeypatch):
    from qwen_decoder_b200 import kernels
    for value in (-300.0, 300.0, 0.0):
        g, rnd, kv, table, cu, start = setup([140], [0], 4, 1, 64, 16)
        q = rnd(140, 256).bfloat16()
        sinks = torch.full((4,), value, device=DEV)
        out = torch.empty(140, 256, dtype=torch.bfloat16, device=DEV)
        kernels.sink_attention_mma(q, out, kv, table, cu, start, 1, 140, 4, 1, 64, 64, 16, 0.125, 0, sinks)
        want = reference(q, kv, table, [140], [0], 4, 1, 64, 16, 0.125, 0, 0, sinks, None, False, 1.0)
        assert torch.isfinite(out).all()
        assert float((out.double() - want).abs().max()) <= 2.0 ** -7 * max(1e-30, float(want.abs().max()))


# query and kv heads, size, tokens a portion, portions, keys, us on mma.sync, us on tcgen05 (a B200, captured calls)
@pytest.mark.parametrize("H,G,d,n,R,keys,mma,tc5", [
    (16, 2, 128, 2, 1, 2, 6.6, 6.9), (16, 2, 128, 2, 1, 902, 53.8, 15.5), (16, 2, 128, 17, 1, 17, 7.9, 8.1), (16, 2, 128, 1500, 1, 1500, 107.7, 24.3),
    (16, 2, 128, 3, 16, 53, 9.3, 7.3), (8, 8, 64, 2, 1, 2, 5.2, 5.9), (8, 8, 64, 17, 1, 17, 5.8, 5.9), (8, 8, 64, 2, 60, 202, 30.5, 39.2),
    (8, 8, 64, 20, 8, 320, 17.6, 8.6), (16, 16, 128, 3, 16, 53, 9.4, 16.8), (16, 16, 128, 3, 16, 1003, 74.0, 36.4), (16, 16, 128, 2, 60, 202, 82.2, 84.0),
    (32, 4, 64, 2, 60, 202, 21.0, 23.3), (32, 4, 64, 32, 1, 932, 41.7, 14.3), (32, 8, 128, 2, 1, 2, 6.3, 7.1), (32, 8, 128, 17, 1, 17, 8.2, 6.9),
    (32, 8, 128, 2, 60, 202, 45.1, 44.1)])
def test_the_faster_form(H, G, d, n, R, keys, mma, tc5):
    from qwen_decoder_b200 import kernels
    taken = kernels.sink_tc5_faster(n * R, R, H, G, d, keys, 148)
    assert (tc5 if taken else mma) <= 1.06 * min(mma, tc5)
