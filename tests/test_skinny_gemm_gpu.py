"""Decode-sized products: split over K with the weight on the tile's wide side, their reductions (plain, norm, SwiGLU), and the launch
as programmatic dependents.

Bound: operands are exact bf16, products are summed in fp32 (K terms: relative error below K * 2^-24 of the sum of magnitudes, which is
sqrt(K) of a typical sum: 2e-4 at K = 4096) and rounded once to bf16 (2^-9)."""
import pytest
import torch

from areal_b200.ops import _lib, fused
from areal_b200.ops.gemm import _splitk_plan, gemm, linear, linear_rmsnorm, linear_swiglu

pytestmark = pytest.mark.gpu


def _bf(*s, std=1.0):
    return (std * torch.randn(*s, device="cuda")).bfloat16()


def _close(a, b):
    err = (a.double() - b).abs()
    assert bool((err <= 2.0 ** -8 * b.abs() + 1e-3 * b.square().mean().sqrt()).all())


@pytest.mark.parametrize("M", [1, 2, 31, 32, 33, 64, 65, 128, 129, 256, 257, 512])
@pytest.mark.parametrize("N,K", [(4, 1024), (132, 1032), (2048, 2048), (1536, 4096), (6148, 1288)])
def test_products(M, N, K):
    torch.manual_seed(M + N)
    x, w, bias = _bf(M, K), _bf(N, K, std=0.05), _bf(N)
    assert _splitk_plan(M, N, K) >= 2 or N > 4000
    want = x.double() @ w.double().t() + bias.double()
    _close(gemm(x, w, bias=bias), want)
    assert torch.equal(gemm(x, w, bias=bias, chained=True), gemm(x, w, bias=bias))
    if N % 16 == 0:
        assert torch.equal(linear_swiglu(x, w), fused.swiglu(gemm(x, w)))
    assert _lib.read_status() == 0


@pytest.mark.parametrize("M", [1, 17, 100, 200])
def test_dependent_launches(M):
    """A decode block over and over with its kernels launched as dependents: the bits of the ordinary launches, whatever overlaps."""
    torch.manual_seed(M)
    H, I = 2048, 6144
    wa, wg, wd, norm = _bf(H, H, std=0.02), _bf(2 * I, H, std=0.02), _bf(H, I, std=0.02), _bf(H)

    def steps(chained):
        y, res, out = x, r, []
        for _ in range(12):
            y = gemm(y, wa, chained=chained)
            y, res = linear_rmsnorm(y, wa, norm, 1e-6, res, chained=chained)
            y, res = linear_rmsnorm(linear_swiglu(y, wg, chained=chained), wd, norm, 1e-6, res, chained=chained)
            out.append((y, res))
        return out

    for _ in range(4):
        x, r = _bf(M, H), _bf(M, H)
        for (a, b), (c, d) in zip(steps(True), steps(False)):
            assert torch.equal(a, c) and torch.equal(b, d)
    assert _lib.read_status() == 0
