"""Products on pairs of SMs (256 x 256 tiles): sizes around a tile and around half of one, every operand major, both output types
and accumulation; the LM head's products on them.

Bound: as for any product here: exact bf16 operands, fp32 sums (1e-3 of a typical result leaves room for K up to 4096), one rounding
to bf16 (2^-8 of the value covers half a step)."""
import pytest
import torch

from areal_b200.ops import _lib
from areal_b200.ops.gemm import gemm
from areal_b200.ops.lm_head import lm_head_logprobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (128, 256, 64), (129, 264, 72), (255, 8, 1000), (256, 256, 448), (257, 520, 128), (640, 1000, 392),
                                   (4000, 2056, 200)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_tiles(M, N, K, a_mn, b_mn):
    torch.manual_seed(M + N + K)
    a, b = (torch.randn(r, K, device="cuda").bfloat16() for r in (M, N))
    want = a.double() @ b.double().t()
    scale = want.square().mean().sqrt()
    A = a.t().contiguous() if a_mn else a
    B = b.t().contiguous() if b_mn else b
    kw = dict(a_mn=a_mn, b_mn=b_mn, bn=512)
    bias = torch.randn(N, device="cuda").bfloat16()
    got = gemm(A, B, bias=bias, **kw)
    err = (got.double() - want - bias.double()).abs()
    assert bool((err <= 2.0 ** -8 * (want + bias.double()).abs() + 1e-3 * scale).all())
    out = torch.randn(M, N, device="cuda")
    before = out.double()
    for n in (1, 2):
        gemm(A, B, out=out, accumulate=True, **kw)
        assert float((out.double() - before - n * want).abs().max()) <= 1e-5 * K ** 0.5 * float(scale.clamp(min=1.0)) + 1e-5
    assert torch.equal(gemm(A, B, **kw), gemm(A, B, **kw))
    assert _lib.read_status() == 0


@pytest.mark.parametrize("T", [1, 128, 129, 256, 385])
@pytest.mark.parametrize("V", [250, 1000, 5000])
def test_lm_head(T, V):
    torch.manual_seed(T + V)
    x = torch.randn(T, 256, device="cuda").bfloat16().requires_grad_()
    w = (0.1 * torch.randn(V, 256, device="cuda")).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device="cuda")
    logp, ent = lm_head_logprobs(x, w, labels)
    g = torch.randn(T, device="cuda")
    (logp * g).sum().backward()
    xd, wd = (t.detach().double().requires_grad_() for t in (x, w))
    z = (xd @ wd.t()).log_softmax(-1)
    want = z.gather(1, labels[:, None])[:, 0]
    (want * g).sum().backward()
    assert float((logp.detach() - want.detach()).abs().max()) < 1e-4
    assert float((ent.detach() + (z.exp() * z).sum(-1).detach()).abs().max()) < 1e-4
    for a, b in ((x.grad, xd.grad), (w.grad, wd.grad)):  # the logits' gradient is held in bf16
        assert float((a.double() - b).norm()) <= 1e-2 * float(b.norm())
    assert _lib.read_status() == 0
