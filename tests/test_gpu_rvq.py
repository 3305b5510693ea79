"""Residual vector quantisation on the GPU (tensor-core pre-selection + exact FP32 decision, ordered decode)
vs the reference's codes (golden fixture) and the CPU oracle."""
from __future__ import annotations

import pytest
import torch
import torch.nn.functional as F

from conftest import load_golden, rvq_recipe
from oracle import mimi_attention_oracle as O

pytestmark = pytest.mark.gpu


def _books(embed_sum, usage):
    return embed_sum / usage.clamp(min=1e-5)[:, :, None]


def test_rvq_codes_match_the_reference_fixture():
    import fast_mimi_b200 as fm
    g = load_golden("rvq_codes.npz")
    gen, embed_sum, usage, proj = rvq_recipe(31, 7)
    emb = torch.randn(2, 512, 40, generator=gen) * 3
    books = _books(embed_sum, usage)
    x = F.conv1d(emb, proj[:, :, None]).permute(0, 2, 1).reshape(-1, 256)
    gb = fm.ops.RVQCodebooks(books.cuda())
    codes, cand = fm.ops.rvq_encode(x.cuda(), gb, return_candidates=True)
    assert torch.equal(codes.cpu().view(7, 2, 40), g["codes"])
    assert int(cand.min()) >= 1 and float(cand.float().mean()) < 16       # a handful of exact evaluations per frame
    for dt in (torch.float16, torch.float32):                               # the forms with the scores in memory
        assert torch.equal(fm.ops.rvq_encode(x.cuda(), gb, scores_dtype=dt).cpu().view(7, 2, 40), g["codes"])
    dec = fm.ops.rvq_decode(codes, gb).cpu().view(2, 40, 256).permute(0, 2, 1)
    assert torch.equal(dec[:, :, ::13], g["quantized_probe"])             # ordered FP32 adds: bit-exact


@pytest.mark.parametrize("scores_dtype", [None, torch.float16, torch.float32])      # None: candidate records, no scores in memory
@pytest.mark.parametrize("rows,layers", [(1, 8), (257, 3), (6000, 8)])
def test_rvq_codes_match_the_oracle(rows, layers, scores_dtype):
    """Frame-level identity (all layers' codes equal) against the CPU oracle; inputs scaled so that the later
    layers see residuals two orders of magnitude smaller than the first."""
    import fast_mimi_b200 as fm
    gen, embed_sum, usage, _ = rvq_recipe(rows, layers)
    books = _books(embed_sum, usage)
    books = books * (0.5 ** torch.arange(layers, dtype=torch.float32))[:, None, None]    # finer codebooks deeper down
    x = torch.randn(rows, 256, generator=gen) * 1.5
    want = O.rvq_encode(x, books)
    gb = fm.ops.RVQCodebooks(books.cuda())
    got = fm.ops.rvq_encode(x.cuda(), gb, scores_dtype=scores_dtype).cpu()
    frames_same = int((got == want).all(dim=0).sum())
    # Where a frame differs, the two nearest entries are closer together than FP32 rounding resolves: the oracle
    # (like the reference) takes argmin over torch.cdist, which for more than 25 rows evaluates |x|^2 + |e|^2 - 2 x.e
    # through a matrix product, the kernel decides by sum_k (x_k - e_k)^2.  An FP64 evaluation of the exact
    # distances says which of the two is nearer to the truth at the first layer where they part.
    first_diff = (got != want).int().argmax(dim=0)
    differing = ((got != want).any(dim=0)).nonzero().flatten().tolist()
    ours_better = 0
    for r in differing:
        l = int(first_diff[r])
        resid = x[r].double()
        for j in range(l):
            resid = resid - books[j, got[j, r]].double()
        d = ((resid[None] - books[l].double()) ** 2).sum(-1)
        ours_better += int(d[got[l, r]] <= d[want[l, r]])
    print(f"rvq rows={rows} layers={layers} scores={scores_dtype}: {frames_same} of {rows} frames have all codes equal to "
          f"the oracle's; of the {len(differing)} others the kernel's choice is the nearer one in FP64 for {ours_better}")
    assert frames_same >= 0.995 * rows, frames_same
    assert torch.equal(fm.ops.rvq_decode(got.cuda(), gb).cpu(), O.rvq_decode(got, books))


@pytest.mark.parametrize("rows,n,k", [(1000, 256, 512), (64, 512, 256), (4099, 256, 512)])
def test_split_precision_linear_has_fp32_accuracy(rows, n, k):
    """The quantiser's input / output projections on the FP16 tensor core (hi + lo parts, FP32 accumulation) against
    an FP64 product and against the FP32 verification kernel."""
    import fast_mimi_b200 as fm
    g = torch.Generator().manual_seed(rows)
    x = (torch.randn(rows, k, generator=g) * 3).cuda()
    w = (torch.randn(n, k, generator=g) / k ** 0.5).cuda()
    got = fm.ops.linear_split(x, fm.ops.split_half(w))
    ref64 = (x.double() @ w.double().T)
    err = float((got.double() - ref64).abs().max() / ref64.abs().max())
    err32 = float((fm.ops.linear_fp32(x, w).double() - ref64).abs().max() / ref64.abs().max())
    print(f"split-precision linear {rows}x{k}->{n}: max error / max |y| = {err:.2e} (FP32 CUDA-core kernel: {err32:.2e})")
    assert err < 2e-6 and err < 2 * err32 + 1e-7       # as good as an FP32 product of the same operands


def test_non_finite_residual_is_reported_not_quantised():
    import fast_mimi_b200 as fm
    gb = fm.ops.RVQCodebooks(torch.randn(1, 256, 256).cuda())
    x = torch.randn(4, 256).cuda()
    x[2, 7] = float("nan")
    st = fm.ops.new_status("cuda")
    fm.ops.rvq_encode(x, gb, status=st)
    assert fm.ops.read_status(st) == 105
    with pytest.raises(RuntimeError, match="105"):
        fm.check_status(status=st)


def test_rvq_decode_rejects_out_of_range_codes():
    import fast_mimi_b200 as fm
    gb = fm.ops.RVQCodebooks(torch.randn(2, 256, 256).cuda())
    codes = torch.tensor([[0, 5], [256, 1]], dtype=torch.int64).cuda()
    with pytest.raises(RuntimeError):
        fm.ops.rvq_decode(codes, gb)


def test_split_quantizer_wrapper_matches_oracle_encode_and_decode():
    """MimiSplitRVQB200 built from modules that carry the reference's attribute names (layers[i].codebook.embed,
    1 x 1 input_proj / output_proj): encode codes and decode output against the oracle with the same projections."""
    import types
    import torch.nn as nn
    import fast_mimi_b200 as fm

    def branch(seed, layers):
        gen, embed_sum, usage, proj = rvq_recipe(seed, layers)
        books = _books(embed_sum, usage)
        mod = types.SimpleNamespace()
        mod.layers = [types.SimpleNamespace(codebook=types.SimpleNamespace(embed=books[i].cuda())) for i in range(layers)]
        mod.input_proj = nn.Conv1d(512, 256, 1, bias=False)
        mod.output_proj = nn.Conv1d(256, 512, 1, bias=False)
        with torch.no_grad():
            mod.input_proj.weight.copy_(proj[:, :, None])
            mod.output_proj.weight.copy_(torch.randn(512, 256, 1, generator=gen) / 16)
        mod.input_proj.cuda(); mod.output_proj.cuda()
        return mod, books

    sem, sem_books = branch(41, 1)
    aco, aco_books = branch(42, 7)
    split = types.SimpleNamespace(semantic_residual_vector_quantizer=sem, acoustic_residual_vector_quantizer=aco)
    native = fm.MimiSplitRVQB200.from_reference(split)
    emb = torch.randn(3, 512, 50, generator=torch.Generator().manual_seed(43)) * 3

    def oracle_encode(mod, books, n):
        x = F.conv1d(emb, mod.input_proj.weight.cpu()).permute(0, 2, 1).reshape(-1, 256)
        return O.rvq_encode(x, books, n).view(n, 3, 50)

    want = torch.cat((oracle_encode(sem, sem_books, 1), oracle_encode(aco, aco_books, 7)))
    got = native.encode(emb.cuda(), 8).cpu()
    assert got.shape == (8, 3, 50)
    same = int((got == want).all(dim=0).sum())
    print(f"split quantiser wrapper: {same} of 150 frames have all 8 codes equal to the oracle's")
    assert same >= 0.995 * 150
    assert torch.equal(native.encode(emb.cuda(), 3).cpu(), got[:3])

    codes = got.permute(1, 0, 2).contiguous()                       # [B, K, T] as the reference's decode takes them
    dec = native.decode(codes.cuda()).cpu()

    def oracle_decode(mod, books, c):                               # c [K, B*T]
        q = O.rvq_decode(c, books).view(3, 50, 256).permute(0, 2, 1)
        return F.conv1d(q, mod.output_proj.weight.cpu())

    flat = got.reshape(8, -1)
    ref = oracle_decode(sem, sem_books, flat[:1]) + oracle_decode(aco, aco_books, flat[1:])
    assert dec.shape == (3, 512, 50)
    assert O.rel_l2(dec, ref) < 1e-5
    with pytest.raises(ValueError):
        native.encode(emb.cuda(), 0)


@pytest.mark.parametrize("B,T,stacks", [(1, 1, 2), (3, 43, 2), (2, 300, 1), (64, 125, 2), (7, 1000, 1)])
def test_decode_with_projection_matches_fp64(B, T, stacks):
    """Ordered sums, hi + lo split, joint projection and the channel-major store, with few rows (split K) and many (pairs)."""
    import fast_mimi_b200 as fm
    g = torch.Generator().manual_seed(B * 100 + T)
    books = [torch.randn(n, 512, 256, generator=g) for n in ((1, 9)[:stacks] if stacks == 2 else (9,))]
    w = [torch.randn(512, 256, 1, generator=g) / 16 for _ in books]
    branch = [fm.MimiRVQB200(b.cuda(), None, p.cuda()) for b, p in zip(books, w)]
    q = fm.MimiSplitRVQB200(*branch) if stacks == 2 else branch[0]
    codes = torch.randint(0, 512, (B, 10 if stacks == 2 else 9, T), generator=g)
    want, l = 0, 0
    for b, p in zip(books, w):
        sums = sum(b[i][codes[:, l + i]].double() for i in range(len(b)))       # [B, T, 256]
        want, l = want + torch.einsum("btk,ck->bct", sums, p[:, :, 0].double()), l + len(b)
    got = q.decode(codes.cuda())
    assert got.shape == want.shape and got.is_contiguous()
    assert float((got.cpu().double() - want).abs().max() / want.abs().max()) < 2e-6
    codes[B - 1, 0, T - 1] = 512
    with pytest.raises(RuntimeError, match="outside the codebook"):
        q.decode(codes.cuda())


@pytest.mark.parametrize("rows", [1, 63, 500])
def test_search_repeats_exactly(rows):
    """The chain of dependent launches over 31 layers, whose kernels share SMs and rewrite the same few buffers layer by layer:
    every call gives the codes of the form that goes through memory one launch at a time."""
    import fast_mimi_b200 as fm
    gen, embed_sum, usage, _ = rvq_recipe(rows, 31)
    scale = 0.7 ** torch.arange(31.0)
    books = fm.ops.RVQCodebooks((_books(embed_sum, usage) * scale[:, None, None]).cuda())
    x = torch.randn(rows, 256, generator=gen).cuda()
    want = fm.ops.rvq_encode(x, books, scores_dtype=torch.float32)
    for _ in range(50):
        assert torch.equal(fm.ops.rvq_encode(x, books), want)
    fm.check_status()


@pytest.mark.parametrize("rows", [1, 70, 5000])
def test_search_one_layer_at_a_time(rows):
    """The calls a host that drives the layers itself makes (margins, candidate records, decision) give the codes of the whole
    search, and leave the residual and the margins of the layer behind the last one."""
    import fast_mimi_b200 as fm
    from fast_mimi_b200 import _native
    layers, entries = 4, 512
    books = fm.ops.RVQCodebooks(torch.randn(layers, entries, 256, generator=torch.Generator().manual_seed(2)).cuda())
    x = torch.randn(rows, 256, generator=torch.Generator().manual_seed(rows)).cuda() * 2
    want, n_want = fm.ops.rvq_encode(x, books, return_candidates=True)
    lib, st, stream = _native.load(), fm.ops.new_status("cuda"), torch.cuda.current_stream().cuda_stream
    resid, resid16, tau = x.clone(), torch.empty(rows, 256, dtype=torch.float16, device="cuda"), torch.empty(rows, device="cuda")
    records = torch.empty(rows, entries // 64, 4, dtype=torch.int32, device="cuda")
    codes, n_cand = torch.empty_like(want), torch.empty_like(n_want)
    tau_rel = fm.ops.RVQ_TAU_REL[torch.float32]
    run = lambda name, *args: _native.check(getattr(lib, name)(*(a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args), stream), name)
    run("fm_rvq_prepare_f32", resid, resid16, tau, rows, books.e_max[0], tau_rel)
    for l in range(layers):
        run("fm_rvq_candidates_f16", resid16, books.half[l], books.sq[l], tau, records, rows, entries, st)
        run("fm_rvq_select_rec_f32", records, books.vectors[l], resid, resid16, codes[l], n_cand[l], tau, rows, entries,
            books.e_max[min(l + 1, layers - 1)], tau_rel, st)
    assert torch.equal(codes, want) and torch.equal(n_cand, n_want)
    left = x
    for l in range(layers):
        left = left - books.vectors[l][want[l]]
    assert torch.equal(resid, left) and torch.equal(resid16, left.half())
    assert fm.ops.read_status(st) == 0


# one block per tile of K slices, two, both parts in one block (few rows), pairs of blocks; 12000: 128-wide units for a branch
@pytest.mark.parametrize("rows", [13, 200, 750, 1300, 4000, 6000, 12000, 20000])
def test_joint_decode_is_as_precise_as_the_branches(rows):
    """Both output projections in one product: its distance from 64 bits is that of two products, each in one accumulator (as
    calls of many rows have it), and their FP32 sum.  Bar: 5 % for the FP32 sums of K slices."""
    import fast_mimi_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(rows)
    n = lambda *s, std=1.0: torch.empty(s, device="cuda").normal_(0, std, generator=g)
    branch = lambda: fm.MimiRVQB200(n(1, 2048, 256), None, n(512, 256, 1, std=256 ** -0.5))
    q = fm.MimiSplitRVQB200(branch(), branch())
    codes = torch.randint(0, 2048, (1, 2, rows), device="cuda", generator=g)
    exact = sum(b.books.vectors[0].double()[codes[0, i]] @ b.output_proj.double().T for i, b in enumerate((q.semantic, q.acoustic))).T
    many = codes.repeat(1, 1, -(-6000 // rows))
    apart = q.semantic.decode(many[:, :1]) + q.acoustic.decode(many[:, 1:])
    assert O.rel_l2(q.decode(codes)[0], exact) < 1.05 * O.rel_l2(apart[0, :, :rows], exact)


@pytest.mark.parametrize("rows", [1, 63, 5000, 20001])
def test_split_precision_products_of_two_weights(rows):
    """Two weights behind one another give two matrices, with few rows and many, equal to the products one by one up to the
    order of FP32 sums."""
    import fast_mimi_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, 512, device="cuda", generator=g)
    w = torch.randn(512, 512, device="cuda", generator=g) / 512 ** 0.5
    got = fm.ops._linear_parts(fm.ops.split_half(x), fm.ops.split_half(w), (rows,), None, mats=2)
    want = (x.double() @ w.double().T).view(rows, 2, 256).transpose(0, 1)
    assert got.shape == want.shape and float((got - want).abs().max() / want.abs().max()) < 2e-6


@pytest.mark.parametrize("rows", [1, 31, 32, 33, 63, 224, 225])
@pytest.mark.parametrize("layers", [1, 2, 3, 32])
def test_search_of_few_vectors_in_one_kernel(rows, layers):
    """Without candidate counts few vectors take one kernel for the whole stack, with them the chain of products and decisions:
    the same codes, also where every entry has a twin (the lower index wins) and for a vector of zeros."""
    from fast_mimi_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows * 40 + layers)
    books = torch.randn(layers, 2048, 256, device="cuda", generator=g) * 0.6 ** torch.arange(layers, device="cuda").clamp(max=7)[:, None, None]
    books[-1, 1024:] = books[-1, :1024].flip(0)
    books = ops.RVQCodebooks(books)
    x = torch.randn(rows, 256, device="cuda", generator=g)
    x[rows // 2] = 0.0
    codes = ops.rvq_encode(x, books)
    chain, _ = ops.rvq_encode(x, books, return_candidates=True)
    assert torch.equal(codes, chain)
    assert int(codes[-1].max()) < 1024
    ops.check_status()


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_one_kernel_search_reports_a_vector_that_is_not_finite(value):
    from fast_mimi_b200 import ops
    books = ops.RVQCodebooks(torch.randn(3, 2048, 256, device="cuda"))
    x = torch.randn(40, 256, device="cuda")
    good = ops.rvq_encode(x, books)
    x[35, 7] = value
    status = ops.new_status("cuda")
    codes = ops.rvq_encode(x, books, status=status)
    assert ops.read_status(status) == 105
    keep = [i for i in range(40) if i != 35]
    assert torch.equal(codes[:, keep], good[:, keep])


@pytest.mark.parametrize("layers,n0", [(1, 1), (2, 1), (3, 3), (4, 1), (5, 2), (8, 1), (9, 3), (12, 12), (17, 16), (32, 1)])      # eight codes at once, then 1, 2, 4 or 8
def test_decoded_parts_of_both_stacks(layers, n0):
    """Sums in the layers' order, bit for bit, as FP16 hi + lo; codes outside a codebook are reported, wherever they stand."""
    import fast_mimi_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(layers)
    B, T, width = 3, 41, 256 if n0 == layers else 512
    books = [torch.randn(n, e, 256, device="cuda", generator=g) for n, e in ((n0, 256), (max(layers - n0, 1), 512))]
    codes = torch.randint(0, 256, (B, layers, T), device="cuda", generator=g)
    want = torch.zeros(B, T, width, device="cuda")
    for l in range(layers):
        stack = int(l >= n0)
        want[..., 256 * stack:256 * stack + 256] += books[stack][l - n0 if stack else l][codes[:, l]]

    def run():
        hi, lo = (torch.empty(B * T, width, dtype=torch.float16, device="cuda") for _ in range(2))
        bad = torch.zeros(1, dtype=torch.int32, device="cuda")
        rc = fm._native.load().fm_rvq_decode_split(codes.data_ptr(), books[0].data_ptr(), books[1].data_ptr() if n0 < layers else None, hi.data_ptr(),
                                                   lo.data_ptr(), B, T, layers, n0, 256, 512 if n0 < layers else 0, bad.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        return hi.view(B, T, width), lo.view(B, T, width), int(bad)

    hi, lo, bad = run()
    assert bad == 0 and torch.equal(hi, want.half()) and torch.equal(lo, (want - want.half().float()).half())
    for l, code in ((0, -1), (layers - 1, 512), (layers // 2, 1 << 40)):
        before = codes[1, l, 7].clone()
        codes[1, l, 7] = code
        assert run()[2] == 1
        codes[1, l, 7] = before


def test_decoding_one_code_takes_less_than_eight():
    """A frame's time is that of its codes: 64000 frames of one take a third of eight's (three quarters where the one was asked for
    eight times)."""
    import fast_mimi_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(5)
    books = torch.randn(8, 2048, 256, device="cuda", generator=g)
    hi, lo = (torch.empty(64000, 256, dtype=torch.float16, device="cuda") for _ in range(2))
    bad = torch.zeros(1, dtype=torch.int32, device="cuda")

    def time(layers):
        codes = torch.randint(0, 2048, (512, layers, 125), device="cuda", generator=g)
        events = [torch.cuda.Event(enable_timing=True) for _ in range(9)]
        for ev in events:
            ev.record()
            for _ in range(4):
                rc = fm._native.load().fm_rvq_decode_split(codes.data_ptr(), books.data_ptr(), None, hi.data_ptr(), lo.data_ptr(), 512, 125, layers, layers,
                                                           2048, 0, bad.data_ptr(), torch.cuda.current_stream().cuda_stream)
                assert rc == 0
        torch.cuda.synchronize()
        return min(a.elapsed_time(b) for a, b in zip(events, events[1:]))

    assert time(1) < 0.55 * time(8)


# rows: one, either side of what a cluster of 16 or 32 vectors takes, of where 16 give way to 32, of the last that one kernel takes; many
@pytest.mark.parametrize("B,T", [(1, 1), (1, 16), (1, 17), (3, 21), (1, 65), (1, 113), (2, 112), (1, 225), (2, 1100)])
@pytest.mark.parametrize("quantizers", [2, 8])
def test_calls_of_the_binding_are_the_checked_ones(B, T, quantizers):
    """Convolution, search, decode and upsampling through the binding give the bits of the checked calls behind them (which a type or
    device out of the ordinary still takes), for embeddings and codes of any layout; what must raise does, and leaves the next
    call alone."""
    import types
    import fast_mimi_b200 as fm
    from fast_mimi_b200 import _native, ops
    g = torch.Generator(device="cuda").manual_seed(T)
    normal = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    branch = lambda n: fm.MimiRVQB200(normal(n, 2048, 256) * 0.7, normal(256, 512, 1) / 512 ** 0.5, normal(512, 256, 1) / 16)
    split = fm.MimiSplitRVQB200(branch(1), branch(7))
    conv = torch.nn.Conv1d(512, 512, 4, 2, bias=False, device="cuda")
    down = fm.MimiDownsampleB200(types.SimpleNamespace(conv=conv, causal=True, pad_mode="replicate"))
    up = fm.MimiUpsampleB200(types.SimpleNamespace(conv=torch.nn.ConvTranspose1d(512, 512, 4, 2, groups=512, bias=False, device="cuda"), padding_left=0, padding_right=2))
    frames = normal(B, T, 512)
    want = down.frames(frames).transpose(1, 2)
    for x in (frames.transpose(1, 2), frames.transpose(1, 2).contiguous()):
        assert torch.equal(down(x), want)
        assert torch.equal(split.encode(x, quantizers), split.encode(x.contiguous(), quantizers))
    half = frames.half().transpose(1, 2)
    codes = split.encode(half, quantizers)                                     # not float32: the checked calls
    assert _native.bind().rvq_encode(half, *split._joint_in_parts(), (), 1.0, ops.default_status(half.device)) is None
    assert torch.equal(split.encode(half.float(), quantizers), codes)
    codes = codes.permute(1, 0, 2)                                             # [B, K, T], not contiguous
    y = split.decode(codes)
    assert torch.equal(y, split.decode(codes.contiguous()))
    sums = [ops.rvq_decode(codes[:, k].transpose(0, 1).reshape(-1, B * T).contiguous(), b.books).view(B, T, 256) for k, b in
            ((slice(0, 1), split.semantic), (slice(1, None), split.acoustic))]
    exact = sum(s.double() @ b.output_proj.double().T for s, b in zip(sums, (split.semantic, split.acoustic))).transpose(1, 2)
    assert O.rel_l2(y.double(), exact) < 1e-6
    assert torch.equal(up(y), ops.upsample2_channels(y, up._taps()).transpose(1, 2))
    assert torch.equal(up(y.double()), up.frames(y.double().transpose(1, 2)).transpose(1, 2).double())
    for wrong in (-1, 2048):
        bad = codes.clone()
        bad[-1, -1, -1] = wrong
        with pytest.raises(RuntimeError, match="outside the codebook"):
            split.decode(bad)
    bad = frames.clone()
    bad[0, 0, 0] = float("nan")
    with pytest.raises(RuntimeError, match="105"):
        split.encode(bad.transpose(1, 2), quantizers)
    ops.default_status(frames.device).zero_()
    assert torch.equal(split.decode(codes), y)


# rows: one, either side of what a cluster takes, the most that all clusters take with 16 vectors each (112 on a B200) and with 32 (224), one more
@pytest.mark.parametrize("rows", [1, 16, 17, 63, 112, 113, 160, 224, 225])
@pytest.mark.parametrize("quantizers", [2, 8, 16, 32])
def test_search_with_the_projections_inside_against_64_bits(rows, quantizers):
    """Both branches from FP32 embeddings, through the binding (up to 224 vectors one kernel that projects, too) and through the calls behind it.  Every code's entry is the
    nearest to what the codes in front of it leave of the exact projection, up to FP32: the projection is off by 1e-6 of its size at most and a
    distance moves by 2 sqrt(d) of that, for either of two entries; sums of 256 squares are off by 2^-24 times sqrt(256), likewise."""
    import fast_mimi_b200 as fm
    from fast_mimi_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows + quantizers)
    normal = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    books = lambda n: normal(n, 2048, 256) * (0.6 ** torch.arange(n, device="cuda").clamp(max=7))[:, None, None]
    branch = lambda n: fm.MimiRVQB200(books(n), normal(256, 512, 1) / 512 ** 0.5, normal(512, 256, 1) / 16)
    split = fm.MimiSplitRVQB200(branch(1), branch(31))
    e = normal(1, 512, rows)
    got = split.encode(e, quantizers)
    frames = e[0].T.contiguous()
    x = ops._linear_rows(frames, lambda: ops.split_half(frames), split._joint_in_parts(), (rows,), None, mats=2)
    checked = torch.empty(quantizers, rows, dtype=torch.int64, device="cuda")
    ops._rvq_search_stacks(x, (split.semantic.books, split.acoustic.books), (checked[:1], checked[1:]), ops._status_ptr(None, x))
    fm.check_status()
    for codes in (got.view(quantizers, rows), checked):
        for b, own in ((split.semantic, codes[:1]), (split.acoustic, codes[1:])):
            r = frames.double() @ b.input_proj.double().view(256, 512).T
            size = r.norm(dim=1)
            for l, c in enumerate(own):
                vectors = b.books.vectors[l].double()
                d = torch.cdist(r, vectors, compute_mode="donot_use_mm_for_euclid_dist") ** 2
                least, chosen = d.min(dim=1).values, d.gather(1, c[:, None])[:, 0]
                assert (chosen - least <= 4e-6 * size * least.sqrt() + 2e-6 * least).all(), (l, float((chosen - least).max()))
                r = r - vectors[c]


def test_calls_that_cannot_be_recorded_refuse_it():
    """torch.jit.trace of the search and of a transposed convolution whose weight learns is an error, not a graph without their kernels."""
    import types
    import fast_mimi_b200 as fm
    branch = lambda n: fm.MimiRVQB200(torch.randn(n, 2048, 256, device="cuda"), torch.randn(256, 512, 1, device="cuda"), torch.randn(512, 256, 1, device="cuda"))
    split = fm.MimiSplitRVQB200(branch(1), branch(7))
    up = fm.MimiUpsampleB200(types.SimpleNamespace(conv=torch.nn.ConvTranspose1d(512, 512, 4, 2, groups=512, bias=False, device="cuda"), padding_left=0, padding_right=2))
    x = torch.randn(2, 512, 30, device="cuda")
    for call in (split.encode, up):
        want = call(x)
        with pytest.raises(Exception):
            torch.jit.trace(lambda t: call(t), (x,))
        assert torch.equal(call(x), want)
    fm.check_status()
