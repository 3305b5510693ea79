"""Split-precision products that read FP32 operands as they lie against 64 bits, and against the form that goes through FP16 parts."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _far(y, ref):
    return float((y.double() - ref).norm() / ref.norm())


# Tiles of 256 rows x 256 outputs on 74 pairs: a ragged last tile, one block of a pair empty, more units than pairs.  FP32 sums of K
# products: the bound is what the form with parts shows, within the spread of its own inputs (a tenth).
@pytest.mark.parametrize("rows,n,k,mats", [(4097, 256, 512, 1), (2300, 512, 256, 2), (20000, 512, 512, 2), (1100, 1024, 640, 1)])
def test_rows(rows, n, k, mats):
    import fast_mimi_b200 as fm
    ops = fm.ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, k, device="cuda", generator=g) * 3
    x[1] = 0.0
    x[2] *= 1e-6
    w = ops.split_half(torch.randn(n, k, device="cuda", generator=g) * k ** -0.5)
    parts = lambda: pytest.fail("too few rows for the direct form")
    got = ops._linear_rows(x, parts, w, (rows,), None, mats=mats)
    old = ops._linear_parts(ops.split_half(x), w, (rows,), None, mats=mats)
    ref = (x.double() @ (w[0].double() + w[1].double()).T).view(rows, mats, n // mats).permute(1, 0, 2)
    assert got.shape == (mats, rows, n // mats) and _far(got, ref) <= 1.1 * _far(old, ref) and _far(got, ref) < 2e-6


@pytest.mark.parametrize("B,T,C,kernel,stride", [(40, 125, 512, 4, 2), (3, 2001, 512, 4, 2), (9, 777, 128, 3, 1), (2500, 1, 512, 4, 2), (30, 333, 64, 6, 4)])
def test_convolution(B, T, C, kernel, stride):
    import fast_mimi_b200 as fm
    ops = fm.ops
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(B, T, C, device="cuda", generator=g)
    w = ops.split_half(torch.randn(512, kernel * C, device="cuda", generator=g) * (kernel * C) ** -0.5)
    t_out = -(-T // stride)
    direct = fm._native.load().fm_split_direct(B * t_out, 512, kernel * C)
    got = ops.downsample_conv(x, w, kernel=kernel, stride=stride)
    at = (torch.arange(t_out, device="cuda")[:, None] * stride - (kernel - stride) + torch.arange(kernel, device="cuda")).clamp(0, T - 1)
    rows = x[:, at].reshape(B * t_out, -1)
    ref = (rows.double() @ (w[0].double() + w[1].double()).T).view(B, t_out, 512)
    assert direct == int(B * t_out >= 2048 and kernel * C % 128 == 0)
    assert got.shape == ref.shape and _far(got, ref) < 3e-6
