"""Where the k-th largest logit is found on a short list: ties at the threshold, lists that overflow, k at and above the number of
threads, vocabularies smaller than the threads, infinities; against the same rule in numpy."""
import numpy as np
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("guard_regions")]
DEV = "cuda:0"


def fits(row, k, temp, draw, got):
    if temp == 0:
        return got == int(np.argmax(row))
    keep = np.ones(len(row), bool)
    if 0 < k < len(row):
        keep = row >= np.sort(row)[::-1][k - 1]
    p = np.where(keep, np.exp((row.astype(np.float64) - row.max()) / temp), 0.0)
    c = np.cumsum(p) / p.sum()
    # the running sum is 1,024 float32 additions over segments: off by at most 1024 * 2^-24
    return keep[got] and c[got] >= draw - 1e-4 and c[got] - p[got] / p.sum() <= draw + 1e-4


@pytest.mark.parametrize("V", [5, 300, 1023, 1024, 1025, 4096, 151936])
@pytest.mark.parametrize("kind", ["normal", "ties", "equal", "infinite"])
def test_sample_selection(V, kind):
    from qwen_decoder_b200 import kernels
    rng = np.random.default_rng(V)
    ks = [0, 1, 2, 40, 1000, 1024, 1025, 3000, V - 1, V]
    logits = rng.normal(0.0, 3.0, (len(ks), V)).astype(np.float32)
    if kind == "ties":
        logits = np.round(logits)
    elif kind == "equal":
        logits[:] = 1.5
    elif kind == "infinite":
        logits[:, rng.integers(0, V, max(1, V // 3))] = -np.inf
        logits[:, 0] = 0.25
    temps = np.full(len(ks), 0.7, np.float32)
    temps[0] = 0.0
    draws = rng.random(len(ks)).astype(np.float32)
    out = torch.empty(len(ks), dtype=torch.int32, device=DEV)
    t = lambda a, dt: torch.tensor(a, dtype=dt, device=DEV)
    kernels.sample(torch.from_numpy(logits).to(DEV), t(temps, torch.float32), t(ks, torch.int32), t(draws, torch.float32), out)
    for r, got in enumerate(out.tolist()):
        assert 0 <= got < V and fits(logits[r], ks[r], float(temps[r]), float(draws[r]), got), (r, ks[r], got)


def test_zeros_of_both_signs_tie():
    """k = 2 with the largest value 0 at five places, two of them +0: the threshold is +0, -0 reaches it too, so each of the five is
    drawn a fifth of the time."""
    from qwen_decoder_b200 import kernels
    V, n = 2000, 64
    row = np.full(V, -30.0, np.float32)
    row[[777, 1500]], row[[5, 40, 41]] = 0.0, -0.0
    draws = ((np.arange(n) + 0.5) / n).astype(np.float32)
    out = torch.empty(n, dtype=torch.int32, device=DEV)
    kernels.sample(torch.from_numpy(np.tile(row, (n, 1))).to(DEV), torch.full((n,), 0.7, device=DEV),
                   torch.full((n,), 2, dtype=torch.int32, device=DEV), torch.from_numpy(draws).to(DEV), out)
    want = [[5, 40, 41, 777, 1500][int(d * 5)] for d in draws]       # five equal shares, no draw within 1e-3 of a border
    assert all(abs(d * 5 - round(d * 5)) > 1e-3 for d in draws)
    assert out.tolist() == want
