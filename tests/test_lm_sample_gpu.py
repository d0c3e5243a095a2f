"""The sampling head on its two layouts (up to 32 rows, more rows): tokens and log-probabilities of the same noise against fp64 logits, ties,
vocabularies around a tile, greedy and noisy rows side by side.

The noise is the kernel's own, so noisy rows are checked through the layouts: the first rows of a batch of 33 draw what a batch of up to 32 draws
(noise is keyed by row, column and step). A log-probability of magnitude m carries fp32 rounding of the shifted logits, a few 1e-6, and of
the product's sums, 1e-5 at 512 terms of size one."""
import pytest
import torch

from areal_b200.ops import _lib
from areal_b200.ops.lm_head import lm_head_sample, new_sampling_rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 7, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("V", [5, 127, 128, 129, 3000, 40000])
@pytest.mark.parametrize("cap", [0.0, 2.0])
def test_layouts_agree(B, V, cap):
    torch.manual_seed(B + V)
    x = torch.randn(33, 512, device="cuda").bfloat16()
    w = (0.05 * torch.randn(V, 512, device="cuda")).bfloat16()
    t = torch.empty(33, device="cuda").uniform_(0.5, 1.5)
    t[::3] = 0.0
    for seed in range(3):
        tok, lp = lm_head_sample(x[:B], w, t[:B].contiguous(), new_sampling_rng(seed, "cuda"), cap)
        tok2, lp2 = lm_head_sample(x, w, t, new_sampling_rng(seed, "cuda"), cap)
        z = x[:B].double() @ w.double().t()
        z = cap * torch.tanh(z / cap) if cap else z
        z = z / torch.where(t[:B] > 0, t[:B], torch.ones_like(t[:B])).double()[:, None]
        assert torch.equal(tok, tok2[:B])
        assert float((lp - lp2[:B]).abs().max()) < 5e-5
        assert float((lp.double() - z.log_softmax(-1).gather(1, tok[:, None].long())[:, 0]).abs().max()) < 5e-5
        greedy = t[:B] <= 0
        assert torch.equal(tok[greedy].long(), z.argmax(-1)[greedy])
    assert _lib.read_status() == 0


@pytest.mark.parametrize("B", [3, 40])
def test_ties_take_the_smallest_token(B):
    x = torch.ones(B, 64, device="cuda").bfloat16()
    w = torch.zeros(1000, 64, device="cuda").bfloat16()
    w[[130, 131, 517, 900]] = 1.0
    tok, lp = lm_head_sample(x, w, torch.zeros(B, device="cuda"), new_sampling_rng(0, "cuda"))
    assert bool((tok == 130).all()) and float((lp + torch.log(torch.tensor(4.0))).abs().max()) < 1e-5
