"""Linear attention of long portions in chunks (``csrc/linear_chunk.cuh``): against the recurrence in float64 and against the token by
token kernels, for lengths that end anywhere in a chunk, several requests, both kinds of heads, strided rows and non-finite tokens."""
import types

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"


def make(lengths, H, G, d, delta, per_token, seed=0, decay=(0.3, 1.0), common=0.0):
    T = sum(lengths)
    g = torch.Generator(device=DEV).manual_seed(seed + T + d)
    rnd = lambda *s: torch.empty(s, device=DEV).normal_(generator=g)
    p = types.SimpleNamespace(H=H, G=G, d=d, lengths=lengths, T=T)
    p.q, p.k = rnd(T, G, d), rnd(T, G, d)
    if common:                                           # keys and queries that share a direction
        way = rnd(1, G, d)
        p.q, p.k = ((1 - common) ** 0.5 * x + common ** 0.5 * way for x in (p.q, p.k))
    if delta:
        p.k /= p.k.norm(dim=-1, keepdim=True)
    p.q *= d ** -0.5
    p.wide = rnd(T, 2 * H * d + 8)                       # values and gate beside one another, rows with room between them
    p.v, p.gate = p.wide[:, :H * d], p.wide[:, H * d:2 * H * d]
    p.beta = torch.rand(T, H, device=DEV, generator=g) if delta else None
    lo, hi = decay
    p.g = lo + (hi - lo) * torch.rand((T, H) if per_token else (H,), device=DEV, generator=g)
    p.norm = 1 + 0.1 * rnd(d)
    p.state = rnd(len(lengths) + 2, H * d * d + 8)
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    req = torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths)).to(DEV, torch.int32)
    slots = torch.arange(len(lengths), 0, -1, device=DEV).to(torch.int32)
    p.ctx = types.SimpleNamespace(num_requests=len(lengths), cu_tokens=cu, state_slots=slots, token_request=req)
    return p


def run(p, monkeypatch, chunks, dtype=torch.float32, write=True, norm=True):
    from qwen_decoder_b200 import kernels
    state = p.state.clone()
    room = torch.empty(p.T, p.H * p.d + 2, dtype=dtype, device=DEV)
    out = room[:, :p.H * p.d]
    asked, real = [], kernels.linear_chunk_scratch
    def scratch(*a):
        asked.append(real(*a))
        return asked[-1] if chunks else 0
    with monkeypatch.context() as m:
        m.setattr(kernels, "linear_chunk_scratch", scratch)
        kernels.linear_scan(p.q, p.k, p.v, p.g, p.beta, p.H, p.d, p.d, state, 4, p.ctx, write, p.gate, p.norm if norm else None, 1e-5, 0.7, out)
    torch.cuda.synchronize()
    return out, state, asked[0]


def reference(p, norm=True):
    H, G, d = p.H, p.G, p.d
    out = torch.empty(p.T, H, d, dtype=torch.float64)
    states = p.state.double().cpu().clone()
    q, k = (x.double().cpu().repeat_interleave(H // G, dim=1) for x in (p.q, p.k))
    v = p.v.double().cpu().view(p.T, H, d)
    g = p.g.double().cpu().expand(p.T, H)
    t = 0
    for r, n in enumerate(p.lengths):
        slot = int(p.ctx.state_slots[r])
        S = states[slot, 4:4 + H * d * d].view(H, d, d).transpose(1, 2).clone()          # [H, keys, values]
        for _ in range(n):
            S = g[t][:, None, None] * S
            x = v[t]
            if p.beta is not None:
                x = p.beta[t].double().cpu()[:, None] * (x - (S.transpose(1, 2) @ k[t][:, :, None])[..., 0])
            S = S + k[t][:, :, None] * x[:, None, :]
            out[t] = (S.transpose(1, 2) @ q[t][:, :, None])[..., 0]
            t += 1
        states[slot, 4:4 + H * d * d] = S.transpose(1, 2).reshape(-1)
    out = out / torch.sqrt((out * out).mean(-1, keepdim=True) + 1e-5)
    if norm:
        out = out * p.norm.double().cpu()
    z = p.gate.double().cpu().view(p.T, H, d)
    return (out * z * torch.sigmoid(z) * 0.7).view(p.T, -1), states


CASES = [([192], 2, 2, 64, False, False), ([300], 4, 2, 64, False, True), ([64, 1, 303, 400], 2, 1, 64, False, True), ([229, 160], 2, 2, 128, False, True),
         ([127, 1, 608], 2, 2, 128, False, False)]


@pytest.mark.parametrize("lengths,H,G,d,delta,per_token", CASES)
def test_against_float64(lengths, H, G, d, delta, per_token, monkeypatch):
    p = make(lengths, H, G, d, delta, per_token)
    want, states = reference(p)
    got, state, floats = run(p, monkeypatch, True)
    old, old_state, _ = run(p, monkeypatch, False)
    assert floats > 0
    err = lambda a, b: float((a.double().cpu() - b).norm() / b.norm())
    # no further from float64 than the kernels that go token by token, but for a unit in the last place of float32
    assert err(got, want) <= max(err(old, want), 2.0 ** -22), (err(got, want), err(old, want))
    assert err(state, states) <= max(err(old_state, states), 2.0 ** -22), (err(state, states), err(old_state, states))
    assert torch.equal(state[0], p.state[0]) and torch.equal(state[:, :4], p.state[:, :4])             # nobody else's


# The delta rule goes four tokens at a time.  Its triangular system a chunk in float32 left 2.7e-7 (outputs) and 1.9e-7 (states) here
# with keys that share a direction; four at a time leave 1.3e-7: sums of 128 products and about five roundings after them, 2^-24 each.
@pytest.mark.parametrize("common", [0.0, 0.9, 0.99])
def test_delta_rule_with_keys_alike(common, monkeypatch):
    p = make([700], 4, 2, 128, True, True, seed=2, decay=(0.9, 1.0), common=common)
    want, states = reference(p)
    got, state, floats = run(p, monkeypatch, True)
    assert floats == 0
    err = lambda a, b: float((a.double().cpu() - b).norm() / b.norm())
    slots = p.ctx.state_slots.long().cpu()
    assert err(got, want) <= 3 * 2.0 ** -24 and err(state.cpu()[slots], states[slots]) <= 3 * 2.0 ** -24, (
        err(got, want), err(state.cpu()[slots], states[slots]))


# outputs and states no further from float64 than token by token, but for two roundings to float32, 2^-24 each
@pytest.mark.parametrize("decay", [(0.3, 1.0), (0.9, 1.0), (0.99, 1.0)])
@pytest.mark.parametrize("common", [0.0, 0.9, 0.99])
@pytest.mark.parametrize("d", [64, 128])
def test_no_less_precise(d, common, decay, monkeypatch):
    p = make([700], 4, 2, d, False, True, seed=2, decay=decay, common=common)
    want, states = reference(p)
    err = lambda a, b: float((a.double().cpu() - b).norm() / b.norm())
    slots, errors = p.ctx.state_slots.long().cpu(), []
    for chunks in (True, False):
        out, state, floats = run(p, monkeypatch, chunks)
        errors.append((err(out, want), err(state.cpu()[slots], states[slots])))
        assert floats > 0
    assert all(new <= max(before, 2.0 ** -23) for new, before in zip(*errors)), errors


@pytest.mark.parametrize("d,delta", [(64, False), (128, False)])
def test_options(d, delta, monkeypatch):
    p = make([980, 100], 2, 1, d, delta, True, seed=5)
    want, _ = reference(p, norm=False)
    got, state, _ = run(p, monkeypatch, True, dtype=torch.bfloat16, write=False, norm=False)
    assert torch.equal(state, p.state)
    assert float((got.double().cpu() - want).norm() / want.norm()) <= 2.0 ** -8
    few = make([100, 100], 2, 1, d, delta, True)
    assert run(few, monkeypatch, True)[2] == 0                                             # short portions go token by token


@pytest.mark.parametrize("d,delta", [(64, False), (128, False)])
@pytest.mark.parametrize("what,value", [(w, x) for w in "vkg" for x in (float("inf"), float("nan"), 3.4e38) if (w, x) != ("g", 3.4e38)])
def test_tokens_before_a_bad_one(d, delta, what, value, monkeypatch):
    p = make([960, 70], 2, 2, d, delta, True, seed=9, decay=(0.9, 1.0))
    good, _, _ = run(p, monkeypatch, True)
    at = 64 + 37
    if what == "v":
        p.v[at, 3] = value
    elif what == "k":
        p.k[at, 0, 5] = value
    else:
        p.g[at, 0] = value
    got, state, _ = run(p, monkeypatch, True)
    # tokens before it, and the other request: another order of sums at most
    for a in (slice(0, at), slice(960, 1030)):
        assert torch.isfinite(got[a]).all()
        assert float((got[a] - good[a]).norm() / good[a].norm()) <= 1e-5


def test_decays_of_all_sizes(monkeypatch):
    """Decays whose products leave float32 within a chunk."""
    for delta, d in ((False, 64), (False, 128)):
        p = make([530], 2, 2, d, delta, True, seed=3, decay=(0.0, 0.3))
        p.g[40:60] = 0.0
        want, states = reference(p)
        got, state, _ = run(p, monkeypatch, True)
        assert float((got.double().cpu() - want).norm() / want.norm()) <= 1e-5
        assert float((state.double().cpu() - states).norm() / states.norm()) <= 1e-6


@pytest.mark.parametrize("d,lengths", [(64, [700]), (128, [130, 64, 600, 3]), (64, [64, 1000])])
@pytest.mark.parametrize("chunks", [1, 3, 7])
@pytest.mark.parametrize("write", [True, False])
def test_passes(d, lengths, chunks, write, monkeypatch):
    """Less scratch than all chunks take: the same bits from several passes, wherever they cut the requests."""
    from qwen_decoder_b200 import kernels
    p = make(lengths, 4, 2, d, False, True, seed=1)
    want, state, floats = run(p, monkeypatch, True, write=write)
    less = chunks * 4 * (68 + d * d) + 2 * 4 * d * d
    assert 0 < less < floats
    monkeypatch.setattr(kernels, "linear_chunk_scratch", lambda *a: less)
    before = kernels.launches()
    got, state2, _ = run(p, monkeypatch, True, write=write)
    assert kernels.launches() - before == 3 * -(-(p.T // 64 + len(lengths)) // chunks)
    assert torch.equal(got, want) and torch.equal(state2, state)
    assert write or torch.equal(state2, p.state)


def test_scratch_has_a_limit():
    from qwen_decoder_b200 import kernels
    for T, R, H, d in ((1500, 1, 32, 64), (32768, 1, 32, 128), (1 << 20, 3, 4, 128), (4000000, 1, 8, 64)):
        floats = kernels.linear_chunk_scratch(T, R, H, H, d, d, d, False, 0)
        assert 0 < floats <= 1 << 24
    assert kernels.linear_chunk_scratch(1 << 20, 1, 1024, 1024, 128, 128, 128, False, 0) == 0          # not two states and a chunk


# heads, size of one, portions, us in chunks, us token by token (a B200, captured calls): the faster form, or one 5 % from it
@pytest.mark.parametrize("H,d,lengths,chunks,tokens", [
    (32, 64, [192], 19.1, 23.0), (32, 64, [1500], 67.4, 154.9), (32, 64, [200] * 3, 36.8, 41.7), (32, 64, [192] * 8, 74.5, 62.1),
    (32, 64, [400] * 8, 153.6, 127.1), (16, 64, [400] * 8, 79.6, 81.6), (16, 64, [600] * 16, 233.3, 190.0), (64, 64, [200] * 3, 67.9, 53.4),
    (128, 64, [1500], 255.7, 301.6), (32, 64, [3, 5, 600], 38.4, 109.6), (4, 64, [600] * 16, 62.0, 91.7),
    (32, 128, [200] * 3, 84.5, 73.8), (32, 128, [600], 78.1, 111.8), (64, 128, [192] * 8, 417.8, 310.1), (16, 128, [600] * 16, 632.6, 487.2),
    (128, 128, [400], 196.8, 182.1), (128, 128, [1500], 726.1, 673.9), (64, 128, [1500], 340.1, 405.0), (8, 128, [400] * 8, 103.2, 109.1)])
def test_the_faster_form(H, d, lengths, chunks, tokens):
    from qwen_decoder_b200 import kernels
    taken = kernels.linear_chunk_scratch(sum(lengths), len(lengths), H, H, d, d, d, False, 0, max(lengths)) > 0
    assert (chunks if taken else tokens) <= 1.05 * min(chunks, tokens)
