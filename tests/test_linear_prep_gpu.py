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
