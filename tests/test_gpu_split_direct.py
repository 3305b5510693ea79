"""Split-precision products that read FP32 operands as they lie against 64 bits, and against the form that goes through FP16 parts."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _far(y, ref):
    return float((y.double() - ref).norm() / ref.norm())


# Tiles of 256 rows x 256 outputs on 74 pairs: a ragged last tile, one block of a pair empty, more units than pairs (four slices of K: as
# many rows as more than a wave of few-row tiles).  FP32 sums of K
# products: the bound is what the form with parts shows, within the spread of its own inputs (a tenth).
@pytest.mark.parametrize("rows,n,k,mats", [(4097, 256, 512, 1), (4800, 512, 256, 2), (20000, 512, 512, 2), (1100, 1024, 640, 1)])
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


# Few slices and one wave of few-row tiles; many outputs, for each 256 of which the operand is split anew; the smallest of more slices, and many rows.
@pytest.mark.parametrize("rows,n,k", [(2048, 512, 256), (4096, 256, 256), (1024, 1024, 256), (5000, 512, 256), (8000, 4096, 512), (1500, 4096, 512),
                                      (2048, 512, 512), (3000, 512, 384), (20000, 256, 256)])
def test_the_faster_form_is_taken(rows, n, k):
    """Either form in a graph, so that the host's part doesn't count: the one that is taken is within a tenth of the other (1.15 to 1.17 of it for
    few slices where rows x outputs alone decided)."""
    import fast_mimi_b200 as fm
    ops, lib = fm.ops, fm._native.load()
    x = torch.randn(rows, k, device="cuda")
    w = ops.split_half(torch.randn(n, k, device="cuda") * k ** -0.5)
    y = torch.empty(rows, n, device="cuda")
    stream = torch.cuda.Stream()

    def direct():
        assert lib.fm_linear_rows_f32(x.data_ptr(), w[0].data_ptr(), w[1].data_ptr(), y.data_ptr(), rows, 1, n, k, None, stream.cuda_stream) == 0

    def time(call):
        with torch.cuda.stream(stream):
            call()
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                for _ in range(8):
                    call()
            events = [torch.cuda.Event(enable_timing=True) for _ in range(9)]
            for ev in events:
                ev.record()
                graph.replay()
            stream.synchronize()
        return min(a.elapsed_time(b) for a, b in zip(events, events[1:]))

    times = time(lambda: ops._linear_parts(ops.split_half(x), w, (rows,), None)), time(direct)
    assert times[lib.fm_split_direct(rows, n, k)] < 1.1 * min(times), times
