"""float32 rotation with cache write, and the gate, by pieces of 16 bytes: the forms of pairs, odd sizes and rows that start off them."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"


# d, rotated width: whole heads, parts of them, nothing, and widths that only the general kernel takes (18; 12 half-split; 6)
@pytest.mark.parametrize("pairing", [0, 1])
@pytest.mark.parametrize("d,rot", [(128, 128), (64, 32), (20, 16), (20, 12), (36, 4), (12, 0), (18, 18), (20, 6)])
@pytest.mark.parametrize("T,write", [(1, True), (7, True), (3, False)])
def test_rope_f32(T, write, d, rot, pairing):
    from qwen_decoder_b200 import kernels
    H, G, page, pages = 6, 2, 4, 5
    g = torch.Generator(device=DEV).manual_seed(d + rot)
    qkv = torch.empty(T, (H + 2 * G) * d, device=DEV).normal_(generator=g)
    kv = torch.zeros(pages, 2, G, page, d, device=DEV)
    pos = torch.randint(0, 50, (T,), device=DEV, generator=g).to(torch.int32)
    slots = torch.randperm(pages * page, device=DEV, generator=g)[:T].to(torch.int32)
    angle = torch.rand(50, max(1, rot // 2), device=DEV, generator=g) * 6
    cos, sin = (angle.cos(), angle.sin()) if rot else (None, None)
    want = qkv.double().view(T, H + 2 * G, d).clone()
    if rot:
        x = want[:, :H + G, :rot]
        a, b = (x[..., 0::2], x[..., 1::2]) if pairing == 0 else (x[..., :rot // 2], x[..., rot // 2:])
        c, s = cos[pos.long()].double()[:, None], sin[pos.long()].double()[:, None]
        u, v = a * c - b * s, a * s + b * c
        want[:, :H + G, :rot] = torch.stack([u, v], -1).flatten(-2) if pairing == 0 else torch.cat([u, v], -1)
    kernels.rope_kv_write(qkv, H, G, d, rot, pairing, cos, sin, pos, kv if write else None, slots if write else None, page, write)
    tol = dict(rtol=0, atol=4e-6)                   # three roundings of numbers up to 8, 2^-24 each
    torch.testing.assert_close(qkv.view(T, -1, d)[:, :H].double(), want[:, :H], **tol)
    if write:
        at = kv[slots.long() // page, :, :, slots.long() % page].double()        # [T, K|V, heads, d]
        torch.testing.assert_close(at[:, 0], want[:, H:H + G], **tol)
        torch.testing.assert_close(at[:, 1], want[:, H + G:], **tol)


@pytest.mark.parametrize("T,F", [(1, 4), (3, 1000), (5, 6), (203, 11008)])
@pytest.mark.parametrize("act", [0, 2])
def test_gate_f32(T, F, act):
    from qwen_decoder_b200 import kernels
    x = torch.empty(T, 2 * F, device=DEV).normal_(generator=torch.Generator(device=DEV).manual_seed(F)) * 3
    out = torch.empty(T, F, device=DEV)
    kernels.swiglu(x, out, act)
    g, u = x.double().chunk(2, 1)
    want = (g * torch.sigmoid(g) if act == 0 else torch.nn.functional.gelu(g, approximate="tanh")) * u
    # expf and the quotient: a few units in the last place of the exponential's argument, which reaches 60 for gelu
    assert float((out.double() - want).norm() / want.norm()) <= 1e-6
