"""Sampling kernel against an fp64 statement: rows where the candidates of a filter fit into shared memory and rows where
they do not, sizes around the warps' segments, unaligned rows, masked, infinite and NaN logits.

A draw may differ from the statement only where the uniform falls within rounding of a boundary: the kernel's fp32 sums are
good to about 1e-6 of the mass, so a token is accepted if its interval of the distribution, widened by 1e-5, holds the uniform."""
import math

import pytest
import torch

from areal_b200.ops import rollout_ops

pytestmark = pytest.mark.gpu


def _check(x, temp, top_k, top_p, u):
    tok, lp = rollout_ops.sample(x, temp, top_k, top_p, u)
    for b in range(x.shape[0]):
        t = int(tok[b])
        y = x[b].double() / (temp[b].double() if temp[b] > 0 else 1.0)
        z = y.log_softmax(-1)
        assert abs(float(lp[b]) - float(z[t])) <= 2e-5 * max(1.0, abs(float(y.max())))
        if temp[b] <= 0:
            assert t == int(y.argmax())
            continue
        p = z.exp()
        keep, unsure = (torch.full_like(p, v, dtype=torch.bool) for v in (True, False))
        k, q = int(top_k[b]) if top_k is not None else 0, float(top_p[b]) if top_p is not None else 1.0
        order = z.sort(descending=True).values
        if 0 < k < len(z):
            keep &= z >= order[k - 1] - 2e-6
            unsure |= (z - order[k - 1]).abs() < 4e-6
        if q < 1:
            n = min(int((order.exp().cumsum(0) < q - 1e-6).sum()), len(z) - 1)
            keep &= z >= order[n] - 2e-6
            unsure |= (z - order[n]).abs() < 4e-6
        assert bool(keep[t])
        cdf = (p * keep).cumsum(0)
        total, lo, hi = float(cdf[-1]), float(cdf[t] - p[t]), float(cdf[t])
        # a threshold is found to 1e-6 of the logarithm: what may or may not be kept widens the interval too
        edge = float(p[unsure].sum()) + 1e-5 * total
        assert lo - edge <= float(u[b]) * total <= hi + edge, (b, t, lo, float(u[b]) * total, hi)


def _rows(B, V, spread, pitch=None, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.empty(B, pitch or V, device="cuda").normal_(0, spread, generator=g)[:, :V]
    u = torch.empty(B, device="cuda").uniform_(0.001, 0.999, generator=g)
    temp = torch.empty(B, device="cuda").uniform_(0.5, 1.5, generator=g)
    return x, temp, u


@pytest.mark.parametrize("V,pitch", [(1, None), (5, None), (127, None), (128, 131), (2047, 2048), (2049, None), (32000, 32001), (151936, None)])
@pytest.mark.parametrize("spread", [0.01, 1.0, 4.0])
def test_filters(V, pitch, spread):
    x, temp, u = _rows(6, V, spread, pitch, V)
    i32 = lambda n: torch.full((6,), n, dtype=torch.int32, device="cuda")
    temp[5] = 0.0
    for top_k, top_p in ((None, None), (None, 0.9), (i32(1), None), (i32(20), None), (i32(513), None), (i32(50), 0.5), (i32(7000), 0.999), (i32(V), 0.0)):
        _check(x, temp, top_k, None if top_p is None else torch.full_like(temp, top_p), u)


def test_ties_and_masks():
    x, temp, u = _rows(4, 9000, 1.0)
    x[0] = 1.5  # all equal: every token is a candidate and none is above another
    x[1, 100:] = -math.inf
    x[2, 10:] = torch.finfo(torch.float32).min
    x[3, 5:8990] = -math.inf
    for top_k, top_p in ((None, None), (None, 0.7), (torch.full((4,), 3, dtype=torch.int32, device="cuda"), None)):
        tok, lp = rollout_ops.sample(x, temp, top_k, None if top_p is None else torch.full_like(temp, top_p), u)
        assert torch.isfinite(lp).all() and (x.gather(1, tok[:, None].long()) > -1e30).all()
        assert torch.equal(tok, rollout_ops.sample(x, temp, top_k, None if top_p is None else torch.full_like(temp, top_p), u)[0])


def test_rows_without_a_distribution():
    x, temp, u = _rows(5, 4000, 1.0)
    x[0], x[1], x[2, 7], x[3, 9] = -math.inf, math.nan, math.inf, math.nan
    for t in (temp, torch.zeros_like(temp)):
        for top_k, top_p in ((None, None), (None, 0.7), (torch.full((5,), 3, dtype=torch.int32, device="cuda"), 0.5)):
            tok, lp = rollout_ops.sample(x, t, top_k, None if top_p is None else torch.full_like(t, top_p), u)
            assert ((tok >= 0) & (tok < 4000)).all()
            assert torch.isnan(lp[:4]).all() and torch.isfinite(lp[4])
            assert int(tok[2]) == 7
