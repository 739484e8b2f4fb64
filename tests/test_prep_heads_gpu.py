"""What stands before attention and before the recurrence, a warp or a part of one per head (``qkv_prep``, ``linear_prep`` without a
convolution), against the general kernels: the same rows one element off 16-byte pieces take those."""
import types

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"


def rows(T, C, g):
    """The same numbers in rows of whole 16-byte pieces and in rows that are not."""
    a = torch.empty(T, -(-C // 4) * 4 + 4, device=DEV).normal_(generator=g)
    b = torch.empty(T, a.shape[1] + 1, device=DEV)
    b[:, :C] = a[:, :C]
    return a[:, :C], b[:, :C]


def context(T, g, pages, page):
    return types.SimpleNamespace(num_requests=1, token_request=torch.zeros(T, dtype=torch.int32, device=DEV),
                                 cu_tokens=torch.tensor([0, T], dtype=torch.int32, device=DEV), state_slots=torch.zeros(1, dtype=torch.int32, device=DEV),
                                 positions=torch.randint(0, 90, (T,), device=DEV, generator=g).to(torch.int32))


def table(dims, g):
    angle = 6 * torch.rand(90, max(4, dims // 2), device=DEV, generator=g)
    return (angle.cos().contiguous(), angle.sin().contiguous()) if dims else (None, None)


def close(a, b):
    # one rounding more or less of a product, and of the store in bfloat16
    tol = 2.0 ** -8 if a.dtype == torch.bfloat16 else 2e-6
    torch.testing.assert_close(a.float(), b.float(), rtol=tol, atol=2e-6)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,G,d,vd,dims", [(3, 1, 128, 128, 128), (4, 2, 64, 40, 64), (2, 2, 20, 12, 16), (5, 1, 100, 128, 40), (2, 1, 32, 32, 0), (2, 0, 64, 64, 8)])
@pytest.mark.parametrize("pairing", [0, 1])
@pytest.mark.parametrize("norm,after", [("none", False), ("head", False), ("head", True)])
def test_qkv_prep(H, G, d, vd, dims, pairing, norm, after, dtype):
    from qwen_decoder_b200 import kernels
    T, page, pages = 13, 4, 6
    g = torch.Generator(device=DEV).manual_seed(d + H)
    C = H * d + G * (d + vd)
    ctx = context(T, g, pages, page)
    slots = torch.randperm(page * pages, device=DEV, generator=g)[:T].to(torch.int32)
    cos, sin = table(dims, g)
    got = []
    for u in rows(T, C, g):
        q = torch.empty(T, H * d, dtype=dtype, device=DEV)
        kv = torch.zeros(pages, max(G, 1) * page * (d + vd), dtype=dtype, device=DEV)
        kernels.qkv_prep(u, H, G, d, vd, None, None, 0, ctx, False, norm, after, None, None, 1e-5, dims, pairing, cos, sin, q, kv, slots, page, G > 0)
        got.append((q, kv))
    close(got[0][0], got[1][0])
    close(got[0][1], got[1][1])


@pytest.mark.parametrize("G,d,dims", [(3, 32, 32), (2, 64, 24), (5, 64, 64), (2, 128, 128), (1, 128, 0)])
@pytest.mark.parametrize("pairing", [0, 1])
@pytest.mark.parametrize("unit,factor", [(None, False), (1e-6, True)])
@pytest.mark.parametrize("T", [1, 45])
def test_linear_prep(G, d, dims, pairing, unit, factor, T):
    from qwen_decoder_b200 import kernels
    H, dv = 2 * G, 8
    g = torch.Generator(device=DEV).manual_seed(d + G)
    ctx = context(T, g, 1, 1)
    cos, sin = table(dims, g)
    mul = torch.rand(T, G, device=DEV, generator=g) if factor else None
    got = []
    for u in rows(T, 2 * G * d + H * dv, g):
        q, k, v, beta, decay = kernels.linear_prep(u, H, G, d, dv, None, None, 0, ctx, False, unit, dims, pairing, cos, sin, 0.3, 0.7, -1, -1, None, None, mul)
        got.append((q, k))
    close(got[0][0], got[1][0])
    close(got[0][1], got[1][1])
