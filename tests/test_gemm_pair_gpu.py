"""Products on pairs of multiprocessors (``csrc/gemm_pair.cu``) at the edges of their tiles, against float64."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"
# (tokens, features, k): one token more and less than a CTA's and a pair's rows, features and k that end inside a tile or a block
SIZES = [(17, 64, 64), (24, 1000, 712), (127, 96, 128), (128, 2049, 200), (129, 512, 2056), (256, 130, 64), (257, 264, 1024), (700, 2050, 320)]


def operands(T, N, K, pad=8):
    g = torch.Generator(device=DEV).manual_seed(T + N + K)
    x = torch.empty(T, K + pad, device=DEV).normal_(generator=g).bfloat16()[:, :K]           # rows with room between them
    w = (torch.empty(N, K, device=DEV).normal_(generator=g) * K ** -0.5).bfloat16()
    return x, w, torch.empty(N, device=DEV).normal_(generator=g)


def check(got, want, tol, each=None):
    """The whole within ``tol``; each element of a bfloat16 result within its rounding and ``each``, what the float32 sums may be off."""
    from qwen_decoder_b200 import kernels
    assert kernels.library("gemm_pair").qd_gemm_pair_status() == 0
    off = (got.double() - want).abs()
    assert float(off.norm() / want.norm()) <= tol
    if got.dtype == torch.bfloat16:
        assert (off <= 2.0 ** -8 * want.abs() + each).all()


def sums_off(x, w):
    """Of a float32 sum in the tensor cores: K / 16 additions, each cut off at 2^-23 of what is added up at most."""
    return (x.shape[1] / 16 + 1) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)


def gated_off(g, u, off_g, off_u):
    """Of act(g) u: both activations' slopes are below 1.2 and their results below |g|; 2^-20: the fast exponential and quotient."""
    return 1.2 * off_g * u.abs() + (g.abs() + off_g) * off_u + 2.0 ** -20 * (g * u).abs()


# float32 sums of K exact products, cut off at every addition: K / 16 additions of 2^-23 at most
# bfloat16 results: rounding once, 2^-9 at most
@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("T,N,K", SIZES)
@pytest.mark.parametrize("bn", [32, 160, 256])
def test_sums(T, N, K, cg, bn):
    from qwen_decoder_b200 import kernels
    x, w, b = operands(T, N, K)
    want = x.double() @ w.double().T
    for dtype, tol in ((torch.float32, K / 16 * 2.0 ** -23 + 1e-7), (torch.bfloat16, 2.0 ** -9)):
        out = torch.full((T, N), float("nan"), dtype=dtype, device=DEV)
        kernels.gemm_pair(x, w, b, out, cg, bn)
        check(out, want + b.double(), tol, sums_off(x, w) + 2.0 ** -23 * b.abs())
    splits = min(3, -(-K // 64))
    part = torch.full((splits, T, N), float("nan"), device=DEV)
    kernels.gemm_pair(x, w, None, part, cg, bn, splits, kernels.EPI_PARTIAL)
    check(part.double().sum(0), want, K / 16 * 2.0 ** -23 + 1e-7)


@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("T,N,K", [s for s in SIZES if s[1] % 2 == 0])
@pytest.mark.parametrize("bn,act,with_bias", [(32, 0, True), (224, 2, True), (256, 0, False)])
def test_gated(T, N, K, cg, bn, act, with_bias):
    from qwen_decoder_b200 import kernels
    x, w, b = operands(T, N, K)
    g, u = (x.double() @ w.double().T + (b.double() if with_bias else 0.0)).chunk(2, 1)
    want = (g * torch.sigmoid(g) if act == 0 else torch.nn.functional.gelu(g, approximate="tanh")) * u
    out = torch.full((T, N // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.gemm_pair(x, w, b if with_bias else None, out, cg, bn, 1, kernels.EPI_SWIGLU + 256 * act)
    off_g, off_u = (sums_off(x, w) + 2.0 ** -23 * b.abs()).chunk(2, 1)
    check(out, want, 2.0 ** -9, gated_off(g, u, off_g, off_u))


def test_gate_far_from_zero():
    """silu of large arguments of both signs: its exponential overflows on one side and vanishes on the other."""
    from qwen_decoder_b200 import kernels
    T, F, K = 32, 64, 64
    x = torch.zeros(T, K, dtype=torch.bfloat16, device=DEV)
    x[:, 0] = torch.tensor([-3e38, -200.0, -100.0, -88.0, 88.0, 100.0, 3e38, 0.0], device=DEV).repeat(4)
    w = torch.zeros(2 * F, K, dtype=torch.bfloat16, device=DEV)
    w[:, 0] = 1.0
    w[F:, 0] = 0.5 ** 10
    out = torch.empty(T, F, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_pair(x, w, None, out, 1, 128, 1, kernels.EPI_SWIGLU)
    g, u = (x.float() @ w.float().T).chunk(2, 1)
    want = g.double() * torch.sigmoid(g.double()) * u.double()
    assert torch.isfinite(out[torch.isfinite(want.float())]).all()
    # (below float32's normal numbers the fast quotient may give zero)
    torch.testing.assert_close(out.double()[want.abs() < 3e38], want[want.abs() < 3e38], rtol=2.0 ** -8, atol=1e-35)


@pytest.mark.parametrize("act", [0, 2])
def test_gates_that_are_no_finite_numbers(act):
    """Minus infinity goes to the limit, zero; infinity and what is no number stay, as in the activation's own kernel."""
    from qwen_decoder_b200 import kernels
    T, F, K = 20, 64, 64
    x, w, b = operands(T, 2 * F, K)
    b[:16], b[16:32], b[32:40] = float("-inf"), float("inf"), float("nan")
    b[F + 8:F + 24], w[F + 8:F + 24] = 0.0, 0.0          # other factors of zero
    out, own = (torch.empty(T, F, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    kernels.gemm_pair(x, w, b, out, 1, 128, 1, kernels.EPI_SWIGLU + 256 * act)
    kernels.swiglu((x.double() @ w.double().T + b.double()).bfloat16(), own, act)
    assert bool((out[:, :16] == 0).all())
    assert bool(out[:, 16:24].isnan().all() and out[:, 24:32].isinf().all() and out[:, 32:40].isnan().all())
    assert torch.equal(out[:, 24:32], own[:, 24:32]) and bool(own[:, 16:24].isnan().all() and own[:, 32:40].isnan().all())


def test_refusals():
    from qwen_decoder_b200 import kernels
    x, w, _ = operands(20, 64, 64, pad=0)
    out = torch.empty(20, 64, dtype=torch.bfloat16, device=DEV)
    for cg, bn in ((3, 64), (1, 48), (1, 288), (2, 0)):
        with pytest.raises(kernels.KernelError):
            kernels.gemm_pair(x, w, None, out, cg, bn)
    with pytest.raises(kernels.KernelError):                          # rows that start off 16 bytes
        kernels.gemm_pair(torch.empty(20 * 64 + 4, dtype=torch.bfloat16, device=DEV)[4:].view(20, 64), w, None, out, 1, 64)


def test_wait_that_runs_out_is_reported():
    from qwen_decoder_b200 import kernels
    kernels.library("gemm_pair")
    kernels.check_status()
    kernels.wait_probe("gemm_pair", 4096)
    with pytest.raises(kernels.KernelError, match="gemm_pair"):
        kernels.check_status()
    kernels.check_status()


@pytest.mark.parametrize("T,N,K,epi", [(17, 4096, 512, 2), (40, 1024, 4096, 1), (130, 1024, 4096, 1), (200, 2048, 1024, 2), (1030, 8192, 1024, 2),
                                       (24, 16384, 256, 0)])
def test_plans(T, N, K, epi):
    """What the plan says is taken, and agrees with the general product."""
    from qwen_decoder_b200 import kernels
    x, w, _ = operands(T, N, K, pad=0)
    plan = kernels.gemm_pair_plan(x, w, epi)
    assert plan is not None
    want = x.double() @ w.double().T
    if epi == kernels.EPI_PARTIAL:
        assert plan[2] > 1
        part = torch.full((plan[2], T, N), float("nan"), device=DEV)
        kernels.gemm_pair(x, w, None, part, *plan, epi=epi)
        check(part.double().sum(0), want, K / 16 * 2.0 ** -23 + 1e-7)
        return
    out = torch.full((T, N if epi == 0 else N // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.gemm_pair(x, w, None, out, *plan, epi=epi)
    each = sums_off(x, w)
    if epi:
        g, u = want.chunk(2, 1)
        want, each = g * torch.sigmoid(g) * u, gated_off(g, u, *each.chunk(2, 1))
    check(out, want, 2.0 ** -9, each)
