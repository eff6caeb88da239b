"""The sampling kernel's step counter (blocks of one cluster up to 8 sequences, a second kernel beyond) and its draw at the edges
of the vocabulary."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gruboros_b200.ops import kernels as K
from tests.test_decode_gpu import filtered_probs


@pytest.mark.parametrize("B", [1, 2, 5, 8, 9])
def test_counter_and_history_advance_together(B):
    g = torch.Generator(device="cuda").manual_seed(B)
    counter = torch.tensor([0, 7], dtype=torch.int64, device="cuda")
    hist = torch.full((B, 6), -1, dtype=torch.int64, device="cuda")
    tok = torch.zeros(B, dtype=torch.uint8, device="cuda")
    want = []
    for t in range(6):
        logits = torch.randn(B, 256, device="cuda", generator=g)
        K.sample(logits, tok, temperature=0.0, counter=counter, history=hist)
        want.append(logits.argmax(-1))
    assert torch.equal(hist, torch.stack(want, dim=1)) and counter.tolist() == [6, 7]


@pytest.mark.parametrize("V", [1, 2, 31, 33, 128, 255, 256])
def test_draw_is_the_inverse_cdf(V):
    g = torch.Generator(device="cuda").manual_seed(V)
    B = 64
    logits = torch.randn(B, V, device="cuda", generator=g) * 2
    logits[0, V // 2] = float("-inf") if V > 1 else 0.0
    logits[1] = 1.0                                                 # ties: lower index first
    u = torch.rand(B, device="cuda", generator=g)
    u[2], u[3] = 0.0, 1.0 - 2.0 ** -24
    tok = torch.zeros(B, dtype=torch.uint8, device="cuda")
    probs = torch.empty(B, V, device="cuda")
    K.sample(logits, tok, temperature=0.9, top_k=20, top_p=0.8, u=u, probs_out=probs)
    keep = torch.arange(B, device="cuda") != 1                      # torch.sort leaves the order of ties open
    want = filtered_probs(logits, 0.9, 20, 0.8)
    close = (probs.double() - want).abs().amax(-1) < 1e-5
    assert bool(close[keep].float().mean() > 0.95)                  # an entry at the threshold may fall either way in fp32
    cdf = probs.double().cumsum(-1)
    for b in range(B):
        t = int(tok[b])
        assert probs[b, t] > 0
        assert (float(cdf[b, t - 1]) if t else 0.0) - 1e-5 <= float(u[b]) <= float(cdf[b, t]) + 1e-5     # 256 fp32 sums below 1: 256 * 2^-25
