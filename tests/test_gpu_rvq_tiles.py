"""The quantiser search of many vectors in one kernel against the chain of products and decision kernels, whose codes it has to give:
``return_candidates`` asks for the chain."""
from __future__ import annotations

import ctypes

import pytest
import torch


def _stack(residual, half, vectors, sq, e_max, codes, layers):
    from fast_mimi_b200 import _native
    return _native.RvqStack(residual, half, vectors, sq, (ctypes.c_float * len(e_max))(*e_max), codes, layers)


# (Of addresses that nothing reads: a call that went on would meet its error elsewhere.)
@pytest.mark.parametrize("books,e_max,layers,want", [(0x10010, 1.0, 2, -3), (0x10004, 1.0, 2, -3), (0x10000, 16385.0, 2, -1), (0x10000, float("nan"), 2, -1),
                                                     (0x10000, 1.0, 33, -1), (0x10000, 1.0, 0, -1), (0, 1.0, 2, -1)])
def test_what_the_kernel_cannot_take_is_refused(books, e_max, layers, want):
    """Its eight-wide loads and the FP16 parts of -|e|^2 / 2 set limits, whoever calls it."""
    from fast_mimi_b200 import _native
    stacks = (_native.RvqStack * 2)(_stack(0x20000, 0x30000, 0x40000, 0x50000, [1.0], 0x60000, 1),
                                    _stack(0x20000, 0x30000, books, 0x50000, [1.0, e_max] + [1.0] * 31, 0x60000, layers))
    assert _native.load().fm_rvq_encode_tiles_f32(stacks, 2, 18000, 2048, 4.5e-3, None, None) == want
    assert _native.load().fm_rvq_encode_tiles_f32(stacks, 1, 18000, 2048 + 128, 4.5e-3, None, None) == -1


def _books(layers, entries, gen, same=0):
    e = torch.randn(layers, entries, 256, device="cuda", generator=gen) * (0.6 ** torch.arange(layers, device="cuda").clamp(max=7))[:, None, None]
    if same:                                     # entries that nothing tells apart: the lowest index wins
        e[:, 100:100 + same] = e[:, 100:101]
    return e


def _tiles(x, *books, error=0):
    """Codes of one or two stacks over ``x`` from the kernel itself, whether or not it is the faster form."""
    import fast_mimi_b200 as fm
    from fast_mimi_b200 import _native
    codes = [torch.empty(b.layers, len(x), dtype=torch.int64, device="cuda") for b in books]
    stacks = (_native.RvqStack * len(books))(*[_stack(x.data_ptr(), b.half.data_ptr(), b.vectors.data_ptr(), b.sq.data_ptr(), b.e_max, c.data_ptr(), b.layers)
                                               for b, c in zip(books, codes)])
    st = fm.ops.new_status("cuda")
    rc = _native.load().fm_rvq_encode_tiles_f32(stacks, len(books), len(x), books[0].entries, fm.ops.RVQ_TAU_REL[torch.float32], st.data_ptr(),
                                                torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and fm.ops.read_status(st) == error
    return codes


# A tile is 256 vectors, 74 pairs of blocks take one each at a time: one pair and a tile hardly begun, a wave of tiles, one more, tiles that
# end inside a block's rows, two and three a pair, which then begin anew with other vectors behind the last layer.
@pytest.mark.gpu
@pytest.mark.parametrize("rows,layers,entries,scale", [(1, 2, 256, 1.0), (257, 3, 512, 1.0), (9217, 8, 2048, 1.0), (18944, 3, 2048, 1.0), (18945, 2, 2048, 1.0),
                                                       (18700, 5, 1024, 300.0), (33000, 2, 256, 1e-3), (38000, 2, 1536, 1.0), (50001, 1, 768, 1.0),
                                                       (3000, 32, 256, 1.0)])
def test_codes_equal_the_chains(rows, layers, entries, scale):
    import fast_mimi_b200 as fm
    gen = torch.Generator(device="cuda").manual_seed(rows)
    books = fm.ops.RVQCodebooks(_books(layers, entries, gen) * scale)
    x = torch.randn(rows, 256, device="cuda", generator=gen) * (1.5 * scale)
    x[5 % rows] = 0.0                            # all margin, no direction
    want, cand = fm.ops.rvq_encode(x, books, return_candidates=True)
    got, = _tiles(x, books)
    assert torch.equal(got, want) and torch.equal(fm.ops.rvq_encode(x, books), want)
    assert rows < 9000 or int(cand.max()) > 1    # exact distances did decide somewhere


# Both stacks dealt to pairs: a tile of either, the longer one first or second; several of both, so that a pair goes on from the first to the
# second and a few pairs have more of one and less of the other.
@pytest.mark.gpu
@pytest.mark.parametrize("rows,layers,entries", [(100, (1, 7), 2048), (9400, (7, 1), 2048), (9500, (3, 3), 512), (20000, (1, 3), 256), (64001, (1, 7), 2048)])
def test_codes_of_two_stacks_equal_the_chains(rows, layers, entries):
    import fast_mimi_b200 as fm
    gen = torch.Generator(device="cuda").manual_seed(rows)
    books = [fm.ops.RVQCodebooks(_books(n, entries, gen)) for n in layers]
    x = torch.randn(rows, 256, device="cuda", generator=gen) * 1.5
    for got, b in zip(_tiles(x, *books), books):
        assert torch.equal(got, fm.ops.rvq_encode(x, b, return_candidates=True)[0])


def _repeated(same, every, rows, layers=2, entries=2048):
    """``same`` equal entries in every codebook, and vectors of which one in ``every`` wants them, again for what is left."""
    import fast_mimi_b200 as fm
    gen = torch.Generator(device="cuda").manual_seed(same)
    e = _books(layers, entries, gen, same)
    x = torch.randn(rows, 256, device="cuda", generator=gen)
    x[::every] = e[0, 100] * 0.9
    return x, fm.ops.RVQCodebooks(e)


# more than a thread remembers; than a vector's four threads do; of every thread's share; every vector, a batch of one
@pytest.mark.gpu
@pytest.mark.parametrize("same,every,entries", [(9, 50, 2048), (40, 50, 2048), (40, 3, 512), (700, 50, 2048), (1900, 1, 2048), (9, 255, 256)])
def test_entries_that_are_the_same(same, every, entries):
    import fast_mimi_b200 as fm
    x, books = _repeated(same, every, 900, entries=entries)
    want = fm.ops.rvq_encode(x, books, return_candidates=True)[0]
    got, = _tiles(x, books)
    assert torch.equal(got, want) and bool((got[0, ::every] == 100).all())


# Repeated entries that every vector wants, one in fifty, one in ten; the chain looks at the marked entries alone.  The kernel takes 0.16 to
# 0.8 of its time; where full lists made all entries candidates it was 9 to 34 times the chain's, and with marks that a better score did not
# wipe out 1.3 times.
@pytest.mark.gpu
@pytest.mark.parametrize("same,every", [(9, 1), (40, 50), (40, 10), (600, 50)])
def test_entries_that_are_the_same_cost_no_more_than_in_the_chain(same, every):
    import fast_mimi_b200 as fm
    x, books = _repeated(same, every, 18000, layers=8)

    def time(**kw):
        fm.ops.rvq_encode(x, books, **kw)
        events = [torch.cuda.Event(enable_timing=True) for _ in range(6)]
        for ev in events:
            ev.record()
            fm.ops.rvq_encode(x, books, **kw)
        torch.cuda.synchronize()
        return min(a.elapsed_time(b) for a, b in zip(events, events[1:]))

    assert time() < 1.25 * time(return_candidates=True)


@pytest.mark.gpu
def test_scores_that_the_tensor_core_cuts_apart():
    """Two entries as far from a short vector as FP32 can tell (in steps of 1/2), whose scores x.e - |e|^2 / 2 end on different steps of 1/4:
    the lower index wins, as among equal ones.  Everything is an integer but x.e, 123 / 512 and 165 / 512 (cut to 16ths beside |e|^2 / 2), and what
    the margin takes of the vector's length and of FP16's subnormals is less than 1/4."""
    import fast_mimi_b200 as fm
    gen = torch.Generator().manual_seed(1)
    e = torch.randint(-250, 251, (1, 2048, 256), generator=gen).float()
    e[0, :, 255] = 1000.0
    e[0, 3, 255] = 0.0                           # shorter than the others by far more than any margin
    e[0, 3, :2] = torch.tensor([123.0, 165.0])
    e[0, 9] = e[0, 3]
    e[0, 9, :2] = torch.tensor([165.0, 123.0])
    square = float((e[0, 3].double() ** 2).sum())
    assert 2 ** 22 < square < 2 ** 23 and (e.double() ** 2).sum(-1).max() < 2 ** 24
    books = fm.ops.RVQCodebooks(e.cuda())
    x = torch.zeros(300, 256, device="cuda")
    x[::3, 0] = 2.0 ** -9
    assert 2e-3 * 4.5e-3 * books.e_max[0] + 3.1e-5 * books.e_max[0] < 2 * 0.25
    got, = _tiles(x, books)
    assert torch.equal(got, fm.ops.rvq_encode(x, books, return_candidates=True)[0]) and bool((got == 3).all())


@pytest.mark.gpu
@pytest.mark.parametrize("frames", [4100, 23, 70])        # many vectors in tiles; one wave of clusters, two
def test_both_stacks_of_a_split_quantiser(frames):
    """1 + 7 layers in one launch against either branch by itself."""
    import fast_mimi_b200 as fm
    gen = torch.Generator(device="cuda").manual_seed(3)
    branch = lambda n: fm.MimiRVQB200(_books(n, 2048, gen), torch.randn(256, 512, 1, device="cuda", generator=gen) * 512 ** -0.5, None)
    q = fm.MimiSplitRVQB200(branch(1), branch(7))
    e = torch.randn(3, 512, frames, device="cuda", generator=gen)
    got = q.encode(e)
    rows = e.permute(0, 2, 1).reshape(-1, 512)
    for branch, part in ((q.semantic, got[:1]), (q.acoustic, got[1:])):
        x = fm.ops.linear_split(rows, fm.ops.split_half(branch.input_proj))
        want = fm.ops.rvq_encode(x, branch.books, return_candidates=True)[0]
        assert torch.equal(part.reshape(len(part), -1), want)


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("nan"), float("inf"), 1e30])
def test_a_vector_that_is_not_finite(value):
    import fast_mimi_b200 as fm
    gen = torch.Generator(device="cuda").manual_seed(4)
    books = fm.ops.RVQCodebooks(_books(2, 2048, gen))
    x = torch.randn(12000, 256, device="cuda", generator=gen)
    x[4321, 7] = value
    got, = _tiles(x, books, error=105)
    st = fm.ops.new_status("cuda")
    want = fm.ops.rvq_encode(x, books, return_candidates=True, status=st)[0]
    assert fm.ops.read_status(st) == 105
    keep = torch.arange(len(x), device="cuda") != 4321
    assert torch.equal(got[0, keep], want[0, keep])        # (the chain's later kernels stop at the first error)
