"""Row-wise kernels of prompt steps that move runs of four numbers: against the forms that move one at a time (which columns
off a 16-byte boundary still take), bit for bit, at the edges of a run of rows."""

import pytest
import torch

from test_decode_kernels_gpu import ints, make_step

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from ninfer_amd_mi50_b200 import kernels
    kernels.load()
    return kernels


@pytest.mark.parametrize("M", [1, 63, 64, 67, 130])
@pytest.mark.parametrize("inner", [4, 1028, 1031])
@pytest.mark.parametrize("act", [None, (2, 7.0, 1.702)])
def test_gated_activation_of_sums(K, M, inner, act):
    g = torch.Generator().manual_seed(1)
    gu, bias = torch.randn((M, 2 * inner), generator=g).cuda() * 4, torch.randn((2 * inner,), generator=g).cuda()
    for b in (None, bias):
        for src, dtype in ((gu, torch.bfloat16), (gu, torch.float32), (gu.bfloat16(), torch.bfloat16)):
            out = K.gated_bias_act(src, b, act, dtype)
            x = src.double() + (0.0 if b is None else b.double())
            gate, up = x[:, :inner], x[:, inner:]
            if act is None:
                want = gate * torch.sigmoid(gate) * up
            else:
                gate, up = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
                want = gate * torch.sigmoid(1.702 * gate) * (up + 1.0)
            # float32 arithmetic of a few roundings, then one to the result's type
            torch.testing.assert_close(out.double(), want, rtol=2 ** -8 if dtype == torch.bfloat16 else 1e-5, atol=1e-5)


@pytest.mark.parametrize("D,rot", [(128, 0), (64, 64), (64, 16), (32, 8), (20, 0)])
@pytest.mark.parametrize("silu", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_queries_and_keys_prepared_in_runs_of_four(K, D, rot, silu, dtype):
    H, V = 5, 16
    _, _, ctx, _, _, g = make_step(dtype, [19, 2], [3, 0], 1, 16, 16, 11)
    src = torch.randn((ctx.T, H * (2 * D + V) + 4), generator=g).to(dtype).cuda()
    shifted = torch.empty((ctx.T, src.shape[1] + 4), dtype=dtype, device="cuda")
    shifted[:, 1:-3] = src                                    # the same columns, off a boundary
    freq = torch.rand((max(1, rot // 2),), generator=g).cuda()
    decay = torch.linspace(0.8, 0.99, H).cuda()
    outs = []
    for x, c in ((src, 0), (shifted, 1)):
        state = torch.zeros((2, H * V * D), device="cuda")
        outs.append((K.decay_linear_attention(x, c, c + H * D, c + 2 * H * D, decay, freq if rot else None, rot, 0.5, silu, state,
                                              ctx, H, D, V), state))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("lens", [[64], [65, 1, 3], [15, 16, 17, 18], [1, 2, 200]])
@pytest.mark.parametrize("C,taps", [(8, 4), (264, 2), (1032, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_convolution_with_rows_in_flight(K, lens, C, taps, dtype):
    """Several requests in a tile of sixteen rows, tiles that end early; the row-by-row form takes the columns off a boundary."""
    _, _, ctx, _, _, g = make_step(dtype, lens, [7] * len(lens), 1, 16, 16, 12)
    src = torch.randn((ctx.T, C + 8), generator=g).to(dtype).cuda()
    shifted = torch.empty((ctx.T, C + 17), dtype=dtype, device="cuda")
    shifted[:, 1:-8] = src
    w, b = torch.randn((taps, C), generator=g).cuda(), torch.randn((C,), generator=g).cuda()
    state = torch.randn((len(lens), (taps - 1) * C), generator=g).cuda()
    outs = []
    for x, c in ((src, 8), (shifted, 9)):
        st = state.clone()
        outs.append((K.causal_conv_silu(x, c, C, w, b, st, ctx), st))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("rows", [4, 5, 8, 9, 16, 24, 25, 32, 33])
@pytest.mark.parametrize("n,k", [(32, 64), (100, 2048), (2048, 256), (6144, 128)])
def test_float32_products_of_few_rows(K, rows, n, k):
    """A row's bits are the same in every tile."""
    g = torch.Generator().manual_seed(2)
    x, w = torch.randn((rows, k), generator=g).cuda(), torch.randn((n, k), generator=g).cuda()
    out = K.linear(x, w)
    assert torch.equal(out, torch.cat([K.linear(x[r:r + 1].contiguous(), w) for r in range(rows)]))
    # a chain of k float32 products and sums
    assert (out - x.double() @ w.double().T).abs().max() <= 2 ** -24 * k ** 0.5 * 5 * k ** 0.5


@pytest.mark.parametrize("hidden", [64, 1024, 2048, 2052, 4096, 6144, 8192])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norms_whose_ctas_walk_rows(K, hidden, dtype):
    """More rows than CTAs: every row's bits are those it has alone (one row a CTA), and the values are right."""
    rows = 148 * 12 * 2 + 5 if hidden <= 2052 else 148 * 4 + 3
    g = torch.Generator().manual_seed(3)
    h = torch.randn((rows, hidden), generator=g).cuda()
    a, b = (torch.randn((rows, hidden), generator=g).to(dtype).cuda() for _ in range(2))
    w, w2 = torch.rand((hidden,), generator=g).cuda() + 0.5, torch.rand((hidden,), generator=g).cuda() + 0.5
    some = [0, 1, rows // 2, rows - 2, rows - 1]
    tol = dict(rtol=2 ** -8, atol=2 ** -8) if dtype == torch.bfloat16 else dict(rtol=2e-5, atol=2e-5)

    def layernorm(h, a, b):
        h, out = h.clone(), torch.empty_like(a)
        K.add_layernorm(h, a, None, w, 1e-6, out)
        return h, out

    def scaled(h, a, b):
        h = h.clone()
        return h, K.scaled_norm_add(h, a, None, w, w2, 1e-6, dtype)

    def residual(h, a, b):
        h, out = h.clone(), torch.empty_like(a)
        K.residual_norm(h, w2, 1e-6, out, a=a, scale_a=0.5, b=b, scale_b=2.0, inner_weight=w, inner_eps=1e-6)
        return h, out

    def gated(h, a, b):
        return (K.group_rmsnorm_gate(h, a, 0, w, 1e-6, 1, 1, dtype),)

    rms = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6)
    x = h.double() + a.double()
    mean = x - x.mean(-1, keepdim=True)
    s = h.double() + rms(a.double()) * w.double() * w2.double()
    r = h.double() + rms(0.5 * a.double() + 2.0 * b.double()) * w.double()
    wants = {layernorm: (x, mean / torch.sqrt((mean * mean).mean(-1, keepdim=True) + 1e-6) * w.double()), scaled: (s, s),
             residual: (r, rms(r) * w2.double()), gated: (rms(h.double()) * w.double() * torch.sigmoid(a.double()),)}
    for fn, want in wants.items():
        got = fn(h, a, b)
        alone = [torch.cat(t) for t in zip(*(fn(h[i:i + 1].contiguous(), a[i:i + 1].contiguous(), b[i:i + 1].contiguous()) for i in some))]
        for t, one, v in zip(got, alone, want):
            assert torch.equal(t[some], one), fn.__name__
            torch.testing.assert_close(t.double(), v, **(tol if t.dtype == torch.bfloat16 else dict(rtol=2e-5, atol=2e-5)))


def median_time(fn):
    """Of twenty calls in a graph, the fastest of seven replays."""
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(20):
            fn()
    times = []
    for _ in range(7):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        graph.replay()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times)


@pytest.mark.parametrize("inner", [704, 1408, 5632])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_activation_of_one_row_more_takes_no_jump(K, inner, dtype):
    """64 rows took up to twice as long as 63 when a thread took four of them."""
    times = []
    for rows in (63, 64):
        gu = torch.randn((rows, 2 * inner), device="cuda").to(dtype)
        times.append(median_time(lambda: K.gated_bias_act(gu, None, None, torch.bfloat16)))
    assert times[1] <= 1.3 * times[0]


def test_norms_of_wide_rows_take_their_numbers_time(K):
    """1,024 rows of 8,192 against 4,096 of 2,048, as many numbers: 1.4 times as long while wide rows were walked."""
    times = {}
    for rows, hidden in ((4096, 2048), (1024, 8192)):
        h, a, w = torch.randn((rows, hidden), device="cuda"), torch.randn((rows, hidden), device="cuda").bfloat16(), torch.rand((hidden,), device="cuda")
        out = torch.empty_like(a)
        times[hidden] = (median_time(lambda: K.group_rmsnorm_gate(h, a, 0, w, 1e-6, 1, 1, torch.bfloat16)),
                         median_time(lambda: K.add_layernorm(h, a, None, w, 1e-6, out)))
    assert times[8192][0] <= 1.15 * times[2048][0] and times[8192][1] <= 1.15 * times[2048][1]
