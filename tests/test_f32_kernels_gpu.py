"""The float32 kernels for rows of whole 16-byte pieces, at the edges of their tiles, against float64."""
import math

import pytest
import torch

from test_kernels_gpu import DEV, _paged_setup, close
import plain_model

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]


@pytest.mark.parametrize("T", [1, 2, 3, 5, 8, 9, 17, 25, 33, 41, 64, 65, 97, 128, 129, 203, 260])
@pytest.mark.parametrize("N,K,splits", [(8, 4, 1), (129, 36, 1), (260, 516, 3), (1000, 2048, None), (8200, 132, None)])
def test_gemm_f32(T, N, K, splits):
    from qwen_decoder_b200 import kernels
    if splits and T <= kernels.F32_FEW_TOKENS:
        splits = 1
    g = torch.Generator(device=DEV).manual_seed(T * N + K)
    x = torch.empty(T, K + 8, device=DEV).normal_(generator=g)[:, 4:4 + K]          # rows of a wider buffer
    w = torch.empty(N, K, device=DEV).normal_(0.0, 0.05, generator=g)
    for bias in (None, torch.empty(N, device=DEV).normal_(generator=g)):
        out = torch.empty(T, N + 3, dtype=torch.float32, device=DEV)
        out.fill_(7.0)
        kernels.gemm_f32(x, w, bias, out[:, :N], splits=splits)
        close(out[:, :N], x.double() @ w.double().t() + (bias.double() if bias is not None else 0.0), torch.float32)
        assert bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("T", [1, 32, 33, 100, 128, 203, 224, 225, 449])
@pytest.mark.parametrize("N,K,splits", [(8, 4, 1), (130, 68, 1), (260, 516, 2), (1000, 2048, None), (256, 1152, 1)])
def test_gemm_f32_split(T, N, K, splits):
    """The tensor cores on operands cut into three pieces: edges of tiles of 128 features and of 224 tokens, a last block of k
    that is not whole, shares of K, an accumulator moved several times (K = 2048 and 1152 in one share)."""
    from qwen_decoder_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(T * N + K)
    x = torch.empty(T, K + 8, device=DEV).normal_(generator=g)[:, 4:4 + K]
    x[T // 2, K // 2] *= 1e4                                 # one element far above the others
    w = torch.empty(N, K, device=DEV).normal_(0.0, 0.05, generator=g)
    for bias in (None, torch.empty(N, device=DEV).normal_(generator=g)):
        out = torch.empty(T, N + 4, dtype=torch.float32, device=DEV)
        out.fill_(7.0)
        kernels.gemm_f32_split(x, w, bias, out[:, :N], splits=splits)
        want = x.double() @ w.double().t() + (bias.double() if bias is not None else 0.0)
        # row by row: at most 16 MMAs a chunk of the large products at 2^-24 of the largest partial sum each, and roundings
        rows = want.abs().amax(dim=1, keepdim=True).clamp(min=1e-3)
        assert float(((out[:, :N].double() - want).abs() / rows).max()) < 3e-6
        assert bool((out[:, N:] == 7.0).all())


def test_gemm_f32_dispatch():
    """What the kernel for whole pieces refuses (a row that is none, a start off the boundary) takes the general one."""
    from qwen_decoder_b200 import kernels
    from qwen_decoder_b200.parts import matmul_backend
    g = torch.Generator(device=DEV).manual_seed(5)
    for T, N, K, shift in ((3, 400, 510, 0), (20, 400, 512, 1), (20, 400, 512, 0), (20, 40, 32, 0), (40, 1100, 1000, 0)):
        wide = torch.empty(T, K + 4, device=DEV).normal_(generator=g)
        x = wide[:, shift:shift + K]
        w = torch.empty(N, K, device=DEV).normal_(generator=g)
        assert kernels.gemm_f32_supported(x, w) == (K % 4 == 0 and shift == 0)
        out = torch.empty(T, N, dtype=torch.float32, device=DEV)
        matmul_backend.linear(x, w, None, out)
        close(out, x.double() @ w.double().t(), torch.float32)


@pytest.mark.parametrize("cfg", [(16, 2, 128, 16, None), (7, 1, 64, 32, None), (3, 3, 4, 8, 37), (24, 2, 100, 16, 50), (4, 2, 16, 1, None)])
@pytest.mark.parametrize("splits", [1, 3, 64])
def test_attention_f32(cfg, splits):
    from qwen_decoder_b200 import kernels
    H, G, d, page_size, window = cfg
    lens = [133, 1, 33]
    kv, bt, ks, vs = _paged_setup(torch.float32, lens, G, d, page_size, seed=8)
    items = [(0, p) for p in (0, 3, 31, 32, 95, 132)] + [(1, 0)] + [(2, p) for p in (4, 32)]
    q = torch.randn(len(items), (H + 2 * G) * d, generator=torch.Generator().manual_seed(9))     # q, k and v side by side
    q[2] *= 4.0
    out = torch.empty(len(items), H * d, dtype=torch.float32, device=DEV)
    tr, pos = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in zip(*items))
    for _ in range(2):                                       # the second launch finds the tickets as the first left them
        kernels.attention_f32(q.to(DEV), q.shape[1], out, kv.to(DEV), bt.to(DEV), tr, pos, len(items), H, G, d, page_size,
                              1.0 / math.sqrt(d), window or 0, splits)
    for i, (r, p) in enumerate(items):
        n = p + 1
        qq = torch.zeros(n, H * d, dtype=torch.float64)
        qq[p] = q[i, :H * d].double()
        want = plain_model.attention(qq, ks[r][:n].double().reshape(n, G * d), vs[r][:n].double().reshape(n, G * d), H, G, d, window)[p]
        close(out[i], want, torch.float32, scale=float(vs[r][:n].abs().max()))


def _product(x, w, bias=None):
    from qwen_decoder_b200 import kernels
    out = torch.empty(x.shape[0], w.shape[0], dtype=torch.float32, device=DEV)
    kernels.gemm_f32(x, w, bias, out)
    return out


@pytest.mark.parametrize("N,K", [(1000, 2048), (2560, 512), (256, 5504), (20000, 132), (515, 516)])
def test_gemm_f32_rows_alone(N, K):
    """A row's result has the same bits whatever the number of rows and wherever the row lies among them: every form for few tokens,
    tiles of 2, 3 and 4 slots, a second tile, a second segment."""
    g = torch.Generator(device=DEV).manual_seed(N + K)
    x = torch.empty(500, K, device=DEV).normal_(generator=g)
    w = torch.empty(N, K, device=DEV).normal_(0.0, 0.05, generator=g)
    b = torch.empty(N, device=DEV).normal_(generator=g)
    want = _product(x, w, b)
    for first, n in [(0, 1), (499, 1), (3, 16), (5, 17), (100, 33), (7, 48), (1, 64), (2, 65), (250, 129), (11, 203), (0, 224), (40, 225), (13, 449)]:
        assert torch.equal(_product(x[first:first + n], w, b), want[first:first + n]), (first, n)


@pytest.mark.parametrize("kind", ["one", "few", "positive", "low_bits", "normal"])
@pytest.mark.parametrize("K", [256, 512, 2048])
@pytest.mark.parametrize("T", [4, 100])
def test_gemm_f32_error(kind, K, T):
    """No further from float64 than one float32 FMA chain over k: on rows of which one term carries the result (the chain rounds it
    once), where no error cancels, and where the lower bits of both operands are all ones.  (Beside the chain's error: the roundings
    of the smaller sums, 2^-8 of half a unit.)  Three terms: at most two additions that are cut off, less than a unit (2^-23) each,
    and one rounding of half a unit, of the terms' magnitude."""
    from qwen_decoder_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(K)
    N = 1024
    x, w = torch.empty(T, K, device=DEV).normal_(generator=g), torch.empty(N, K, device=DEV).normal_(generator=g)
    if kind in ("one", "few"):
        n = 1 if kind == "one" else 3
        keep = torch.rand(T, K, device=DEV, generator=g).topk(n, dim=1).indices
        x = torch.zeros_like(x).scatter_(1, keep, x.gather(1, keep))
    elif kind == "positive":
        x, w = x.abs(), w.abs()
    elif kind == "low_bits":
        x, w = (t.abs().view(torch.int32).bitwise_or(0xFFFF).view(torch.float32) for t in (x, w))
    want = x.double() @ w.double().t()
    scale = x.double().abs() @ w.double().abs().t()
    off = ((_product(x, w).double() - want).abs() / scale)
    if kind == "few":
        assert float(off.max()) <= 2.5 * 2.0 ** -23
        return
    chain = torch.empty(T, N, dtype=torch.float32, device=DEV)
    kernels.gemm_generic(x, w, None, chain)
    ref = (chain.double() - want).abs() / scale
    assert float(off.max()) <= float(ref.max()) * (1 + 2.0 ** -7), (float(off.max()), float(ref.max()))
    assert float(off.pow(2).mean()) <= float(ref.pow(2).mean()) * (1 + 2.0 ** -6)


@pytest.mark.parametrize("T", [1, 5, 40, 64, 203, 300])
@pytest.mark.parametrize("N,K", [(256, 516), (1000, 1024)])
def test_gemm_f32_ends_of_the_range(T, N, K):
    """Infinities, NaN, numbers that bfloat16 would round to infinity and numbers below its range: what the FMA chain gives, bit for
    bit (NaN for NaN), in the rows and columns that have them; the other results stay as they are."""
    from qwen_decoder_b200 import kernels
    inf, big, tiny = float("inf"), 3.4e38, 3e-37
    g = torch.Generator(device=DEV).manual_seed(T)
    x, w = torch.empty(T, K, device=DEV).normal_(generator=g), torch.empty(N, K, device=DEV).normal_(0.0, 0.05, generator=g)
    b = torch.empty(N, device=DEV).normal_(generator=g)
    w[:, 9] = 0.0
    w[5, 9], w[6, 100], w[7, 3] = 2.0, -inf, float("nan")
    plain = _product(x, w, b)
    rows = {0: (inf, 2), T // 2: (-inf, 9), T - 1: (big, 9)}
    for r, (v, k) in rows.items():
        x[r, k] = v
    for bias in (b, None):
        got, chain = _product(x, w, bias), torch.empty(T, N, dtype=torch.float32, device=DEV)
        kernels.gemm_generic(x, w, bias, chain)
        odd = ~chain.isfinite()
        assert bool(odd.any()) and torch.equal(got.isnan(), chain.isnan())
        assert torch.equal(got[odd].nan_to_num(0.0, inf, -inf), chain[odd].nan_to_num(0.0, inf, -inf))
        assert float((got - chain)[~odd].abs().max()) < 1e-5 * float(chain[~odd].abs().max())
    if T > 3:
        others = [r for r in range(T) if r not in rows]
        assert torch.equal(_product(x, w, b)[others].nan_to_num(7.0), plain[others].nan_to_num(7.0))
    x = torch.empty(T, K, device=DEV).normal_(generator=g) * tiny
    chain = torch.empty(T, N, dtype=torch.float32, device=DEV)
    w[6:8] = 0.01
    kernels.gemm_generic(x, w, None, chain)
    assert torch.equal(_product(x, w), chain)


def _attend(q, out, kv, bt, tr, pos, cfg, splits):
    from qwen_decoder_b200 import kernels
    H, G, d, page_size, window = cfg
    kernels.attention_f32(q, q.shape[1], out, kv, bt, tr, pos, q.shape[0], H, G, d, page_size, 1.0 / math.sqrt(d), window or 0, splits)


@pytest.mark.parametrize("cfg", [(16, 2, 128, 16, None), (7, 1, 64, 32, None), (6, 3, 20, 8, 1100), (24, 2, 100, 16, 50)])
def test_attention_f32_token_alone(cfg):
    """A token's result has the same bits alone and among others, whatever the CTAs of its cluster: contexts of one run, one wave,
    eight waves, runs of 8, 16 and 24 keys."""
    H, G, d, page_size, window = cfg
    lens = [2300, 1, 700]
    kv, bt, ks, vs = _paged_setup(torch.float32, lens, G, d, page_size, seed=3)
    items = [(0, p) for p in (0, 7, 8, 127, 128, 1023, 1024, 1500, 2047, 2048, 2299)] + [(1, 0)] + [(2, p) for p in (4, 255, 256, 699)]
    tr, pos = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in zip(*items))
    q = torch.empty(len(items), H * d, device=DEV).normal_(generator=torch.Generator(device=DEV).manual_seed(4))
    kv, bt = kv.to(DEV), bt.to(DEV)
    want = torch.empty(len(items), H * d, device=DEV)
    _attend(q, want, kv, bt, tr, pos, cfg, 8)
    for splits in (1, 2, 4):
        out = torch.empty_like(want)
        _attend(q, out, kv, bt, tr, pos, cfg, splits)
        assert torch.equal(out, want), splits
    for i in range(len(items)):
        out = torch.empty(1, H * d, device=DEV)
        _attend(q[i:i + 1], out, kv, bt, tr[i:i + 1].contiguous(), pos[i:i + 1].contiguous(), cfg, 1 << i % 4)
        assert torch.equal(out[0], want[i]), items[i]
    for i, (r, p) in enumerate(items):
        n = p + 1
        qq = torch.zeros(n, H * d, dtype=torch.float64)
        qq[p] = q[i].cpu().double()
        ref = plain_model.attention(qq, ks[r][:n].double().reshape(n, G * d), vs[r][:n].double().reshape(n, G * d), H, G, d, window)[p]
        close(want[i], ref, torch.float32, scale=float(vs[r][:n].abs().max()))


def test_attention_f32_more_tokens_than_a_grid():
    """65,537 tokens of one head of 4 in one step, as the general kernel takes them."""
    from qwen_decoder_b200 import kernels
    T, page_size, cfg = 65537, 16, (1, 1, 4, 16, 24)
    kv, bt, _, _ = _paged_setup(torch.float32, [64], 1, 4, page_size, seed=5)
    kv, bt = kv.to(DEV), bt.to(DEV)
    q = torch.empty(T, 4, device=DEV).normal_(generator=torch.Generator(device=DEV).manual_seed(6))
    pos = (torch.arange(T, device=DEV) % 64).to(torch.int32)
    tr = torch.zeros(T, dtype=torch.int32, device=DEV)
    out, want = torch.empty(T, 4, device=DEV), torch.empty(T, 4, device=DEV)
    _attend(q, out, kv, bt, tr, pos, cfg, 1)
    kernels.paged_attention_generic(q, 4, want, kv, bt, tr, pos, T, 1, 1, 4, page_size, 0.5, 24)
    assert float((out - want).abs().max()) < 2e-6 * float(want.abs().max())


def test_f32_step_token_alone(tmp_path):
    """Logits of the float32 engine, with matrices that ``gemm_f32`` takes, bit for bit: a prompt in one step, cut in several ways
    (down to single tokens, replayed as a captured step), beside other requests."""
    from qwen_decoder_b200.config import Qwen2Config
    from qwen_decoder_b200.engine import ModelRunner, StepEntry
    from qwen_decoder_b200.weights import write_random_model
    cfg = {"architectures": ["Qwen2ForCausalLM"], "hidden_size": 512, "intermediate_size": 1280, "num_hidden_layers": 2,
           "num_attention_heads": 8, "num_key_value_heads": 2, "vocab_size": 1000, "max_position_embeddings": 512,
           "rope_theta": 10000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": False}
    folder = write_random_model(Qwen2Config.from_dict(cfg), str(tmp_path), 4, dtype=torch.float32, std=0.08)
    runner = ModelRunner.from_folder(folder, dtype="float32", device=DEV, num_pages=64)
    g = torch.Generator().manual_seed(7)
    tokens = torch.randint(0, 1000, (150,), generator=g).tolist()

    def run(cuts, beside=()):
        rc, others, at, got = runner.open("it"), [runner.open(f"o{i}") for i in range(len(beside))], 0, []
        for n in cuts:
            entries = [StepEntry(rc, tokens[at:at + n], list(range(n)))]
            entries += [StepEntry(o, torch.randint(0, 1000, (k,), generator=g).tolist(), [k - 1]) for o, k in zip(others, beside)]
            got.append(runner.step(entries)[:n].clone())
            at += n
        for r in [rc] + others:
            runner.close(r)
        return torch.cat(got)

    want = run([150])
    assert bool(want.isfinite().all())
    for cuts, beside in [([1, 16, 17, 48, 68], ()), ([75, 75], (3, 20)), ([149, 1], (1, 1, 64)), ([140] + [1] * 10, ()), ([140] + [1] * 10, (1,) * 7)]:
        assert torch.equal(run(cuts, beside), want), (cuts, beside)


def test_gemm_f32_wait_that_runs_out_is_reported_once():
    """The library's own bounded wait, on an mbarrier nobody arrives at, with a limit of a few thousand polls; products go on."""
    from qwen_decoder_b200 import kernels
    kernels.check_status()
    kernels.wait_probe("gemm_f32", 4096)
    torch.cuda.synchronize()
    with pytest.raises(kernels.KernelError, match="gemm_f32"):
        kernels.check_status()
    kernels.check_status()
    x, w = torch.ones(3, 512, device=DEV), torch.ones(300, 512, device=DEV)
    assert bool((_product(x, w) == 512.0).all())
