"""Attention backward at the edges of its 128-row blocks: sequences one off a block, whole blocks between partial ones, groups of one to seven
query heads, keys and values as strided views; and the same bits for dK and dV on every run (dQ is summed in arrival order).

Bound: P and dS are rounded to bf16 (half a step, 2^-9, each) and summed in fp32, the results are rounded once more: three independent roundings
of 2^-9 / sqrt(3) rms make 0.2% of a result that does not cancel; 1% leaves room for the cancellation in dS."""
import pytest
import torch

from areal_b200.ops import _lib
from areal_b200.ops.attention import VarlenMeta, attention_ref, varlen_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1], [127], [129], [256], [640, 3, 385], [130] * 9])
@pytest.mark.parametrize("heads", [(1, 1), (7, 1), (8, 4)])
def test_backward_blocks(lens, heads):
    Hq, Hkv = heads
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + Hq)
    new = lambda *s: torch.empty(s, device="cuda").normal_(generator=g).bfloat16()
    T, cu = sum(lens), [0]
    for n in lens:
        cu.append(cu[-1] + n)
    q, do, kv = new(T, Hq, 128).requires_grad_(), new(T, Hq, 128), new(T, 2 * Hkv * 128).requires_grad_()
    meta = VarlenMeta(cu, "cuda")
    split = lambda t: (t[:, :Hkv * 128].unflatten(1, (Hkv, 128)), t[:, Hkv * 128:].unflatten(1, (Hkv, 128)))
    got = []
    for _ in range(3):
        q.grad = kv.grad = None
        varlen_attention(q, *split(kv), meta).backward(do)
        got.append((q.grad.clone(), kv.grad.clone()))
    assert _lib.read_status() == 0
    assert all(torch.equal(a[1], got[0][1]) for a in got)
    qd, kvd = (t.detach().float().requires_grad_() for t in (q, kv))
    attention_ref(qd, *split(kvd), cu).backward(do.float())
    for a, b in ((got[0][0], qd.grad), (got[0][1][:, :Hkv * 128], kvd.grad[:, :Hkv * 128]), (got[0][1][:, Hkv * 128:], kvd.grad[:, Hkv * 128:])):
        # a sequence of one token has no gradient with respect to its score: dQ and dK are rounding noise around zero
        scale = max(float(b.norm()), 1e-2 * float(do.float().norm()))
        assert float((a.float() - b).norm()) <= 1e-2 * scale
