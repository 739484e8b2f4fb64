"""``linear_prep`` where a thread walks a channel's tokens against the plain statement of the same preparation: portions of
several requests that begin inside a CTA's tokens, kept inputs, every number of taps with a form of its own."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"


@pytest.mark.parametrize("taps", [0, 2, 3, 4, 5])
@pytest.mark.parametrize("d,G,dv,H", [(128, 2, 128, 4), (64, 3, 40, 3), (30, 2, 64, 2), (100, 1, 128, 2)])
def test_linear_prep_of_portions(taps, d, G, dv, H):
    from qwen_decoder_b200 import kernels
    g = torch.Generator().manual_seed(taps * 100 + d)
    lens, slots = [1, 150, 17, 2, 31], [3, 0, 4, 1, 2]
    T, C, R = sum(lens), 2 * G * d + H * dv, len(lens)
    u = torch.randn(T, C + H, generator=g)
    w = torch.randn(C, max(taps, 1), generator=g) if taps else None
    keep = max(taps - 1, 0)
    state = torch.randn(R + 1, 5 + keep * C + 3, generator=g)
    cu = torch.tensor([0] + lens).cumsum(0)
    want = torch.zeros(T, C, dtype=torch.float64)
    for r, n in enumerate(lens):
        x = u[cu[r]:cu[r] + n, :C].double()
        if taps:
            x = torch.cat([state[slots[r], 5:5 + keep * C].view(keep, C).double(), x])
            x = sum(x[j:j + n] * w[:, j].double() for j in range(taps))
            x = x * torch.sigmoid(x)
        want[cu[r]:cu[r] + n] = x
    unit = lambda y: y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)
    q, k, v = want[:, :G * d].view(T, G, d), want[:, G * d:2 * G * d].view(T, G, d), want[:, 2 * G * d:]
    q, k = unit(q) * 0.25, unit(k)

    class Ctx:
        token_request = torch.repeat_interleave(torch.arange(R), torch.tensor(lens)).to(torch.int32).to(DEV)
        cu_tokens = cu.to(torch.int32).to(DEV)
        state_slots = torch.tensor(slots, dtype=torch.int32, device=DEV)
        num_requests, num_tokens = R, T
        positions = torch.zeros(T, dtype=torch.int32, device=DEV)

    st = state.to(DEV)
    got = kernels.linear_prep(u.to(DEV), H, G, d, dv, w.to(DEV) if taps else None, st, 5, Ctx, True, 1e-6, 0, 0, None, None,
                              0.25, 1.0, -1, -1, None, None)
    dp = kernels.linear_pad(d)
    for name, have, need in (("q", got[0], q), ("k", got[1], k)):
        have = have.view(T, G, dp).double().cpu()
        assert float((have[..., :d] - need).abs().max()) < 2e-6, name
        assert bool((have[..., d:] == 0).all()), name
    if taps:
        assert float((got[2].view(T, H * dv).double().cpu() - v).abs().max()) < 1e-5 * float(v.abs().max())


@pytest.mark.parametrize("pairing", [0, 1])
@pytest.mark.parametrize("taps,d,G,dv,H,dims", [(4, 128, 2, 64, 4, 128), (0, 64, 3, 40, 3, 32), (3, 30, 2, 64, 2, 30), (2, 100, 1, 128, 2, 24), (5, 64, 2, 64, 2, 64)])
def test_linear_prep_rotation_and_gates(pairing, taps, d, G, dv, H, dims):
    """What the test above leaves out, at positions of their own for every token: rotation of a whole head and of its first part in
    both pairings, k's factors, beta and the decay, and the kept inputs moved on."""
    from qwen_decoder_b200 import kernels
    g = torch.Generator().manual_seed(taps * 100 + d + pairing)
    lens, slots = [1, 150, 17, 2, 31], [3, 0, 4, 1, 2]
    T, C, R = sum(lens), 2 * G * d + H * dv, len(lens)
    u = torch.randn(T, C + 2 * H + 1, generator=g)
    w = torch.randn(C, max(taps, 1), generator=g) if taps else None
    keep = max(taps - 1, 0)
    state = torch.randn(R + 1, 5 + keep * C + 3, generator=g)
    A_log, dt_bias, k_mul = torch.randn(H, generator=g), torch.randn(H, generator=g), torch.rand(T, G, generator=g) + 0.5
    ang = torch.rand(4 * T, dims // 2, generator=g, dtype=torch.float64) * 6.0
    pos = torch.randperm(4 * T, generator=g)[:T]
    cu = torch.tensor([0] + lens).cumsum(0)
    want, after = torch.zeros(T, C, dtype=torch.float64), state.double().clone()
    for r, n in enumerate(lens):
        x = u[cu[r]:cu[r] + n, :C].double()
        if taps:
            x = torch.cat([state[slots[r], 5:5 + keep * C].view(keep, C).double(), x])
            after[slots[r], 5:5 + keep * C] = x[n:].reshape(-1)
            x = sum(x[j:j + n] * w[:, j].double() for j in range(taps))
            x = x * torch.sigmoid(x)
        want[cu[r]:cu[r] + n] = x

    def turned(y):
        half = dims // 2
        a, b = (torch.arange(0, dims, 2), torch.arange(1, dims, 2)) if pairing == 0 else (torch.arange(half), torch.arange(half, dims))
        c, s = (f(ang.float().double()[pos])[:, None] for f in (torch.cos, torch.sin))
        out = y.clone()
        out[..., a], out[..., b] = y[..., a] * c - y[..., b] * s, y[..., b] * c + y[..., a] * s
        return out

    q, k, v = want[:, :G * d].view(T, G, d), want[:, G * d:2 * G * d].view(T, G, d), want[:, 2 * G * d:]
    q, k = turned(q) * 0.25, turned(k) * 0.5 * k_mul.double()[..., None]

    class Ctx:
        token_request = torch.repeat_interleave(torch.arange(R), torch.tensor(lens)).to(torch.int32).to(DEV)
        cu_tokens = cu.to(torch.int32).to(DEV)
        state_slots = torch.tensor(slots, dtype=torch.int32, device=DEV)
        num_requests, num_tokens = R, T
        positions = pos.to(torch.int32).to(DEV)

    st = state.to(DEV)
    cos, sin = (f(ang.float()).to(DEV).contiguous() for f in (torch.cos, torch.sin))
    got = kernels.linear_prep(u.to(DEV), H, G, d, dv, w.to(DEV) if taps else None, st, 5, Ctx, True, None, dims, pairing, cos, sin,
                              0.25, 0.5, C, C + H + 1, A_log.to(DEV), dt_bias.to(DEV), k_mul.to(DEV))
    dp = kernels.linear_pad(d)
    for name, have, need in (("q", got[0], q), ("k", got[1], k)):
        have = have.view(T, G, dp).double().cpu()
        assert float((have[..., :d] - need).abs().max()) < 2e-6 * max(1.0, float(need.abs().max())), name
        assert bool((have[..., d:] == 0).all()), name
    beta = torch.sigmoid(u[:, C:C + H].double())
    decay = torch.exp(-torch.exp(A_log.double()) * torch.nn.functional.softplus(u[:, C + H + 1:C + 2 * H + 1].double() + dt_bias.double()))
    assert float((got[3].double().cpu() - beta).abs().max()) < 1e-6
    assert float((got[4].double().cpu() - decay).abs().max()) < 2e-6
    assert torch.equal(st.cpu(), after.float())
    if taps:
        assert float((got[2].view(T, H * dv).double().cpu() - v).abs().max()) < 1e-5 * float(v.abs().max())
