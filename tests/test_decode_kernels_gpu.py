"""Kernels of decode steps and of the all-32-bit path at the sizes where they can go wrong: float32 attention that shares
its keys among a segment's rows, the biased split-key attention of single rows, the scan of single rows."""

import ctypes
import math
from dataclasses import replace
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from ninfer_amd_mi50_b200 import kernels
    kernels.load()
    return kernels


def ints(values):
    return torch.tensor(list(values), dtype=torch.int32, device="cuda")


def make_step(dtype, lens, pos0s, Hkv, D, page, seed):
    from ninfer_amd_mi50_b200.parts.base import StepContext
    g = torch.Generator().manual_seed(seed)
    need = [(p + n + page - 1) // page for p, n in zip(pos0s, lens)]
    order, at = torch.randperm(sum(need), generator=g).tolist(), 0
    bt = torch.full((len(lens), max(need) + 1), -1, dtype=torch.int32)
    for s, n in enumerate(need):
        bt[s, :n] = torch.tensor(order[at:at + n])
        at += n
    pages = torch.randn((sum(need), 2, Hkv, page, D), generator=g).to(dtype).cuda()
    positions = [p + i for p, n in zip(pos0s, lens) for i in range(n)]
    row_seg = [s for s, n in enumerate(lens) for _ in range(n)]
    row0 = [0]
    for n in lens:
        row0.append(row0[-1] + n)
    ctx = StepContext(dtype=dtype, device=torch.device("cuda"), T=len(positions), S=len(lens), token_ids=ints([0] * len(positions)),
                      positions=ints(positions), row_seg=ints(row_seg), seg_row0=ints(row0), seg_pos0=ints(pos0s),
                      seg_slot=ints(range(len(lens))), logit_rows=ints([]), seg_len_host=list(lens), seg_pos0_host=list(pos0s),
                      max_rows_per_seg=max(lens), max_context=max(p + n for p, n in zip(pos0s, lens)))
    return pages, bt.cuda(), ctx, positions, row_seg, g


def exact_attention(q, pages, bt, positions, row_seg, Hq, page, window, keep, scale, slopes=None, gate=None, sig=None, cap=0.0):
    """Row by row in 64 bits; q [T, Hq, D]."""
    out = torch.zeros_like(q, dtype=torch.float64)
    Hkv = pages.shape[2]
    for t, (p, s) in enumerate(zip(positions, row_seg)):
        j = torch.arange(p + 1, device="cuda")
        kv = pages[bt[s, j // page].long(), :, :, j % page].double()          # [keys, 2, Hkv, D]
        k, v = (kv[:, i].repeat_interleave(Hq // Hkv, 1) for i in (0, 1))
        x = torch.einsum("hd,jhd->hj", q[t].double(), k) * scale
        if cap:
            x = cap * torch.tanh(x / cap)
        if slopes is not None:
            x = x - slopes.double()[:, None] * (p - j)
        seen = (j > p - window) | (j < keep) if window else torch.ones_like(j, dtype=torch.bool)
        if sig is not None:
            w = torch.sigmoid(x + sig.double()[:, None]) * seen
        else:
            w = torch.softmax(x.masked_fill(~seen, -math.inf), -1)
        out[t] = torch.einsum("hj,jhd->hd", w, v)
        if gate is not None:
            out[t] *= torch.sigmoid(gate[t].double())[:, None]
    return out


STEPS = [([37, 1, 16, 2, 1, 17], [0, 130, 61, 5, 0, 250]), ([1, 1, 1], [0, 127, 400]), ([130], [129])]


@pytest.mark.parametrize("Hq,Hkv,D,page", [(6, 2, 48, 16), (4, 1, 128, 64), (3, 3, 256, 32), (4, 2, 64, 16), (5, 1, 20, 24),
                                          (40, 2, 32, 16)])
@pytest.mark.parametrize("lens,pos0s", STEPS)
@pytest.mark.parametrize("form", ["plain", "window", "kept", "cap", "sigmoid"])
def test_float32_attention_that_shares_keys(K, Hq, Hkv, D, page, lens, pos0s, form):
    """Against 64 bits, against the kernel of one warp a row (the same bits where no window shifts its blocks), and with
    a step's rows sent one by one (the same bits always)."""
    pages, bt, ctx, positions, row_seg, g = make_step(torch.float32, lens, pos0s, Hkv, D, page, 5)
    T = ctx.T
    q = torch.randn((T, Hq * D), generator=g).cuda()
    scale = D ** -0.5
    window = 70 if form in ("window", "kept") else 0
    keep = 5 if form == "kept" else 0
    slopes = torch.tensor([0.3 / (i + 1) for i in range(Hq)]).cuda() if form == "kept" else None
    gate = torch.randn((T, Hq), generator=g).cuda() if form == "kept" else None
    sig = torch.linspace(-1, 1, Hq).cuda() if form == "sigmoid" else None
    cap = 2.0 if form == "cap" else 0.0

    def run(ctx, rows=slice(None)):
        if form in ("plain", "cap", "window"):
            qkv = torch.cat([q[rows], torch.zeros((len(q[rows]), 2 * Hkv * D), device="cuda")], 1)
            return K.paged_attention(qkv, Hq, Hkv, D, pages, bt, page, ctx, window, scale, softcap=cap)
        return K.biased_window_attention(q[rows].contiguous(), Hq, Hkv, D, pages, bt, page, ctx, window, keep, scale, slopes,
                                         None if gate is None else gate[rows].contiguous(), 0, sig)

    out = run(ctx)
    want = exact_attention(q.view(T, Hq, D), pages, bt, positions, row_seg, Hq, page, window, keep, scale, slopes, gate, sig, cap)
    # sums of up to 401 products of 256 and of 401 weights, float32: some 2^-24 * sqrt(657) of the terms' size, times four
    bound = 6e-6 * max(1.0, want.abs().max().item())
    assert (out.view(T, Hq, D) - want).abs().max() <= bound
    # without the segments' rows: one warp a row and head
    warp = run(SimpleNamespace(positions=ctx.positions, row_seg=ctx.row_seg))
    if window == 0:
        assert torch.equal(out, warp)
    else:
        assert (out - warp).abs().max() <= bound
    at = 0
    for s, n in enumerate(lens):
        for i in (0, n - 1):
            one = replace(ctx, T=1, S=1, positions=ints([pos0s[s] + i]), row_seg=ints([s]), seg_row0=ints([0, 1]), seg_len_host=[1],
                          max_rows_per_seg=1, _tiles={})
            assert torch.equal(run(one, slice(at + i, at + i + 1))[0], out[at + i])
        at += n


@pytest.mark.parametrize("Hq,Hkv,D", [(16, 16, 128), (28, 4, 128), (6, 2, 64), (16, 1, 32), (8, 8, 256), (4, 2, 64)])
@pytest.mark.parametrize("lens", [[1] * 9, [1] * 33, [1] * 70, [1, 2, 3, 9] * 8 + [4], [8, 1, 9] * 23 + [1], [17, 16]])
@pytest.mark.parametrize("window,keep", [(0, 0), (40, 3)])
def test_float32_attention_of_many_segments(K, Hq, Hkv, D, lens, window, keep):
    """More segments than a warp looks over at once, of a run of rows, one less and one more; steps whose CTAs fit the device
    with four, two and one block of keys at a time, and tiles whose keys are one block beside others.  Against 64 bits and,
    where no window passes a key, the bits of one warp a row."""
    pos0s = [(0, 3, 31, 32, 33, 95, 96, 150)[(5 * s) % 8] for s in range(len(lens))]
    pages, bt, ctx, positions, row_seg, g = make_step(torch.float32, lens, pos0s, Hkv, D, 16, 21)
    q = torch.randn((ctx.T, Hq * D), generator=g).cuda()
    slopes = torch.tensor([0.3 / (i + 1) for i in range(Hq)]).cuda()

    def run(ctx):
        return K.biased_window_attention(q, Hq, Hkv, D, pages, bt, 16, ctx, window, keep, D ** -0.5, slopes, None, 0, None)
    out = run(ctx)
    want = exact_attention(q.view(ctx.T, Hq, D), pages, bt, positions, row_seg, Hq, 16, window, keep, D ** -0.5, slopes)
    assert (out.view(ctx.T, Hq, D) - want).abs().max() <= 6e-6 * max(1.0, want.abs().max().item())     # (the bound above)
    if window == 0:
        assert torch.equal(out, run(SimpleNamespace(positions=ctx.positions, row_seg=ctx.row_seg)))


@pytest.mark.parametrize("rows,Hq,Hkv,D,keys", [(64, 16, 16, 128, 32), (32, 16, 16, 128, 8), (64, 16, 16, 64, 8), (16, 28, 4, 128, 8),
                                                (64, 28, 4, 128, 8), (8, 32, 2, 128, 8), (64, 8, 8, 256, 16), (64, 16, 16, 128, 257)])
def test_float32_attention_of_short_rows_is_no_slower_than_one_warp_a_row(K, rows, Hq, Hkv, D, keys):
    """Single rows of requests with few keys, where CTAs that come in rounds took up to five times as long; 1.3 times is
    more than any of these differs by from run to run."""
    pages, bt, ctx, _, _, g = make_step(torch.float32, [1] * rows, [keys - 1] * rows, Hkv, D, 16, 22)
    qkv = torch.randn((rows, (Hq + 2 * Hkv) * D), generator=g).cuda()

    def timed(ctx):
        run = lambda: K.paged_attention(qkv, Hq, Hkv, D, pages, bt, 16, ctx, 0, D ** -0.5)
        run()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(20):
                run()
        times = []
        for _ in range(7):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    assert timed(ctx) <= 1.3 * timed(SimpleNamespace(positions=ctx.positions, row_seg=ctx.row_seg))


def test_float32_attention_keeps_a_number_that_is_not_finite_behind_its_row(K):
    """Later rows of a segment hold NaN: rows before them see nothing of it."""
    pages, bt, ctx, positions, row_seg, g = make_step(torch.float32, [40], [3], 2, 64, 16, 6)
    q = torch.randn((40, 4 * 64 + 2 * 2 * 64), generator=g).cuda()
    good = K.paged_attention(q, 4, 2, 64, pages, bt, 16, ctx, 0, 0.125)
    page, slot = int(bt[0, 23 // 16]), 23 % 16
    pages[page, :, :, slot] = math.nan                        # position 23, row 20
    bad = K.paged_attention(q, 4, 2, 64, pages, bt, 16, ctx, 0, 0.125)
    assert torch.equal(bad[:20], good[:20]) and bad[20:].isnan().any(1).all()


@pytest.mark.parametrize("Hq,Hkv,D,page", [(4, 4, 128, 64), (6, 2, 64, 16), (20, 2, 32, 32), (2, 1, 16, 32)])
@pytest.mark.parametrize("window,keep", [(0, 0), (300, 4), (128, 130), (1024, 4), (1, 1), (129, 0)])
@pytest.mark.parametrize("mixed", [False, True])
def test_biased_attention_of_single_rows(K, Hq, Hkv, D, page, window, keep, mixed):
    pos0s = [0, 127, 128, 299, 300, 428, 431, 1500, 1023, 1024, 1151, 1152]
    lens = [1] * len(pos0s)
    if mixed:
        lens[2] = 9
    pages, bt, ctx, positions, row_seg, g = make_step(torch.bfloat16, lens, pos0s, Hkv, D, page, 7)
    T = ctx.T
    q = torch.randn((T, Hq * D), generator=g).bfloat16().cuda()
    slopes = torch.tensor([0.05 / (i + 1) for i in range(Hq)]).cuda()
    gate = torch.randn((T, Hq + 3), generator=g).cuda()
    out = K.biased_window_attention(q, Hq, Hkv, D, pages, bt, page, ctx, window, keep, D ** -0.5, slopes, gate, 3)
    want = exact_attention(q.view(T, Hq, D), pages, bt, positions, row_seg, Hq, page, window, keep if window else 0, D ** -0.5,
                           slopes, gate[:, 3:])
    # weights and outputs rounded to bfloat16 once each: 2^-8 of the values' size (up to 4.5 of unit variance)
    assert (out.view(T, Hq, D) - want).abs().max() <= 2 ** -8 * 4.5
    K.check_status()


@pytest.mark.parametrize("blocks,Hq,Hkv", [(1024, 4, 2), (1025, 4, 2), (16, 136, 1)])
def test_biased_attention_of_single_rows_where_a_merge_ends(K, blocks, Hq, Hkv):
    """A step whose context bound is as many key blocks as a merge takes, one more, and a key head of more
    query heads than the split kernel is given: answered all the same."""
    D, page = 64, 16
    pages, bt, ctx, positions, row_seg, g = make_step(torch.bfloat16, [1, 1, 1], [0, 300, 1151], Hkv, D, page, 11)
    ctx = replace(ctx, max_context=blocks * 128, _tiles={})
    q = torch.randn((ctx.T, Hq * D), generator=g).bfloat16().cuda()
    slopes = torch.tensor([0.05 / (i + 1) for i in range(Hq)]).cuda()
    gate = torch.randn((ctx.T, Hq), generator=g).cuda()
    out = K.biased_window_attention(q, Hq, Hkv, D, pages, bt, page, ctx, 0, 0, D ** -0.5, slopes, gate, 0)
    want = exact_attention(q.view(ctx.T, Hq, D), pages, bt, positions, row_seg, Hq, page, 0, 0, D ** -0.5, slopes, gate)
    assert (out.view(ctx.T, Hq, D) - want).abs().max() <= 2 ** -8 * 4.5      # (the bound of the test above)
    K.check_status()


def test_biased_attention_of_heads_beyond_the_split_kernels_biased_form(K):
    """Heads of 256 in bfloat16 are answered by one warp a row and head, and no split kernel is built for them."""
    Hq, Hkv, D, page = 4, 2, 256, 16
    pages, bt, ctx, positions, row_seg, g = make_step(torch.bfloat16, [1, 1, 1], [0, 130, 300], Hkv, D, page, 13)
    q = torch.randn((3, Hq * D), generator=g).bfloat16().cuda()
    slopes = torch.tensor([0.05 / (i + 1) for i in range(Hq)]).cuda()
    out = K.biased_window_attention(q, Hq, Hkv, D, pages, bt, page, ctx, 100, 4, D ** -0.5, slopes)
    want = exact_attention(q.view(3, Hq, D), pages, bt, positions, row_seg, Hq, page, 100, 4, D ** -0.5, slopes)
    assert (out.view(3, Hq, D) - want).abs().max() <= 2 ** -8 * 4.5      # (the bound of the tests above)
    n, none = ctypes.c_int, None
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    ws = torch.empty((3 * Hq * 3 * (D + 2),), device="cuda")
    rc = K.load().nf_decode_attention_biased(p(q), n(Hq * D), p(pages), p(bt), n(bt.shape[1]), p(ctx.positions), p(ctx.row_seg), p(out),
                                             p(ws), p(ws[3 * Hq * 3 * D:]), none, n(3), n(Hq), n(Hkv), n(D), n(page), n(pages.shape[0]),
                                             n(100), ctypes.c_float(D ** -0.5), n(3), p(slopes), n(4), none, n(0), none)
    assert rc != 0 and b"256" in K.load().nf_last_error()


@pytest.mark.parametrize("heads,P,N,groups", [(8, 64, 128, 2), (6, 20, 64, 3), (3, 7, 16, 1), (4, 33, 200, 4), (2, 64, 256, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_scan_of_single_rows_has_the_walking_kernels_bits(K, heads, P, N, groups, dtype):
    _, _, ctx, _, _, g = make_step(dtype, [1, 1, 1], [0, 5, 9], 1, 16, 16, 8)
    ctx.seg_slot = ints([2, 0, 3])
    C = heads * P + 2 * groups * N
    xbc = torch.randn((3, C), generator=g).to(dtype).cuda()
    dt = torch.randn((3, heads + 5), generator=g).to(dtype).cuda()
    bias, rate, D = (torch.randn((heads,), generator=g).cuda() for _ in range(3))
    state = torch.randn((4, 10 + heads * P * N), generator=g).cuda()
    results = []
    for bound in (1, 2):                                      # 2: a bound of two rows a segment, so that rows are walked
        st = state.clone()
        y = K.ssd_scan(xbc, 0, heads * P, heads * P + groups * N, dt, 5, bias, rate, D, st, 10,
                       replace(ctx, max_rows_per_seg=bound, _tiles={}), heads, P, N, groups)
        results.append((y, st))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("heads,P,N,groups,rows", [(8, 64, 128, 2, 1), (64, 64, 128, 8, 8), (3, 7, 16, 1, 3)])
@pytest.mark.parametrize("behind_convolution", [False, True])
def test_scan_of_single_rows_again_and_again_on_one_state(K, heads, P, N, groups, rows, behind_convolution):
    """Sixty steps from and into one state with no copy between: by themselves, and behind the convolution of a layer with
    what its call says.  The bits are those of the kernel that walks rows, which reads the state after its wait."""
    dtype = torch.bfloat16
    _, _, ctx, _, _, g = make_step(dtype, [1] * rows, [5] * rows, 1, 16, 16, 9)
    C, taps = heads * P + 2 * groups * N, 4
    src = [torch.randn((rows, C), generator=g).to(dtype).cuda() for _ in range(3)]
    dt = torch.randn((rows, heads), generator=g).to(dtype).cuda()
    w, b = torch.randn((taps, C), generator=g).cuda(), torch.randn((C,), generator=g).cuda()
    bias, rate, D = (torch.randn((heads,), generator=g).cuda() for _ in range(3))
    first = torch.randn((rows, (taps - 1) * C + heads * P * N), generator=g).cuda()
    results = []
    for bound in (1, 2):                                      # 2: rows are walked
        c = replace(ctx, max_rows_per_seg=bound, _tiles={})
        state, ys = first.clone(), []
        for i in range(60):
            xbc = K.causal_conv_silu(src[i % 3], 0, C, w, b, state, ctx) if behind_convolution else src[i % 3]
            ys.append(K.ssd_scan(xbc, 0, heads * P, heads * P + groups * N, dt, 0, bias, rate, D, state, (taps - 1) * C, c, heads,
                                 P, N, groups, **({"state_settled": True} if behind_convolution else {})))
        results.append((torch.stack(ys), state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
