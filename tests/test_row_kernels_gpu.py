"""Row kernels (RMSNorm, q/k norm + rotation, SwiGLU) at the edges of their layouts: rows that fill no thread group, the
widths where a thread starts to own two vectors, odd row and head counts, operands that start off a 16-byte boundary.

Bounds: results are bf16, so they may be half a step (2^-9) off besides the fp32 error; a column sum of T products of
numbers around one carries the bf16 rounding of its result only, the terms are summed in fp32."""
import pytest
import torch

from areal_b200.ops import fused

pytestmark = pytest.mark.gpu
STEP = 2.0 ** -8


def _close(a, b, scale=None):
    b = b.double()
    scale = b.square().mean().sqrt() if scale is None else scale
    err = (a.double() - b).abs()
    assert (err <= STEP * b.abs() + 2e-3 * scale).all(), float((err / (STEP * b.abs() + 2e-3 * scale)).max())


def _bf(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


@pytest.mark.parametrize("H", [8, 256, 264, 2048, 2056, 4096, 4104, 8192])
@pytest.mark.parametrize("T", [1, 2, 5, 1300])
def test_rmsnorm_rows(T, H):
    torch.manual_seed(H + T)
    x, r, dy, dh = (_bf(T, H) for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16()
    a = [t.clone().requires_grad_() for t in (x, r, w)]
    y, h = fused.rmsnorm(a[0], a[2], 1e-6, a[1])
    torch.autograd.backward([y, h], [dy, dh])
    hd = h.detach().double().requires_grad_()  # the kernel's own residual: the norm works on what is stored
    wd = w.double().requires_grad_()
    yd = hd * torch.rsqrt(hd.square().mean(-1, keepdim=True) + 1e-6) * wd
    torch.autograd.backward([yd, hd], [dy.double(), dh.double()])
    _close(h.detach(), x.double() + r.double())
    _close(y.detach(), yd.detach())
    _close(a[0].grad, hd.grad)
    assert torch.equal(a[0].grad, a[1].grad)
    _close(a[2].grad, wd.grad)
    plain = fused.rmsnorm(h.detach(), w, 1e-6)
    assert torch.equal(plain, y.detach())


@pytest.mark.parametrize("heads", [(1, 1), (3, 1), (5, 2), (16, 8), (28, 4)])
@pytest.mark.parametrize("T", [1, 77, 1001])
@pytest.mark.parametrize("norm", [True, False])
def test_rotation_heads(T, heads, norm):
    Hq, Hkv = heads
    torch.manual_seed(T + Hq)
    # every operand starts 2 bytes past a 16-byte boundary
    off = lambda *s: torch.cat([torch.zeros(1, device="cuda").bfloat16(), _bf(*s).flatten()])[1:].view(*s)
    qkv = off(T, (Hq + 2 * Hkv) * 128).requires_grad_()
    qw, kw = ((1 + 0.1 * off(128)).requires_grad_() for _ in range(2)) if norm else (None, None)
    cos, sin = fused.rope_tables(300, 128, 1e6, "cuda")
    pos = torch.randint(0, 300, (T,), device="cuda", dtype=torch.int32)
    out = fused.qknorm_rope(qkv, qw, kw, cos, sin, pos, Hq, Hkv, 128)
    g = [off(*o.shape) for o in out]
    torch.autograd.backward(list(out), g)
    ref = [t.detach().double().requires_grad_() if t is not None else None for t in (qkv, qw, kw)]
    q, k, v = (t.unflatten(1, (-1, 128)) for t in ref[0].split([Hq * 128, Hkv * 128, Hkv * 128], 1))
    rms = lambda t, w: t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-6) * w if norm else t
    c, s = (t[pos.long()].double()[:, None] for t in (cos, sin))
    rot = lambda t: torch.cat((t[..., :64] * c - t[..., 64:] * s, t[..., 64:] * c + t[..., :64] * s), -1)
    want = (rot(rms(q, ref[1])), rot(rms(k, ref[2])), v)
    torch.autograd.backward(list(want), [t.double() for t in g])
    for a, b, n in zip(out[:2], want, (rms(q, ref[1]), rms(k, ref[2]))):
        # the normalised values are rounded to bf16 ahead of the rotation, half a step each of the two that meet in a result
        _close(a.detach(), b.detach(), 2 * float(n.detach().abs().max()) if norm else None)
    assert torch.equal(out[2], v.detach().bfloat16())
    _close(qkv.grad, ref[0].grad)
    if norm:
        _close(qw.grad, ref[1].grad)
        _close(kw.grad, ref[2].grad)


@pytest.mark.parametrize("T,inter", [(1, 8), (3, 264), (2, 2048), (257, 2056), (70001, 8)])
def test_swiglu_rows(T, inter):
    torch.manual_seed(T)
    gu = _bf(T, 2 * inter).requires_grad_()
    y, dy = fused.swiglu(gu), _bf(T, inter)
    y.backward(dy)
    d = gu.detach().double().requires_grad_()
    want = torch.nn.functional.silu(d[:, :inter]) * d[:, inter:]
    want.backward(dy.double())
    _close(y.detach(), want.detach())
    _close(gu.grad, d.grad)
    # far out, gates are closed or open: no infinities or NaN of the exponential's making
    far = torch.tensor([[-300.0, -88.5, -87.0, -20.0, 20.0, 87.0, 88.5, 300.0] + [1.0] * 8], device="cuda").bfloat16()
    got = fused.swiglu(far)
    _close(got, torch.nn.functional.silu(far[:, :8].double()), 1e-3)
