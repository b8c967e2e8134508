"""What a decode step does with few rows (csrc/ssm.cu's convolution of single rows, csrc/qk_norm_append.cu's norm over whole
rows) against float64, at sizes that the forms in runs of four take and at sizes that they leave to the others."""

import pytest
import torch

from test_chunk_recurrence_gpu import context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [2, 3, 4, 5])
@pytest.mark.parametrize("C,col0,more", [(8, 0, 0), (264, 8, 16), (2056, 8, 0), (36, 4, 3), (33, 1, 0)])
def test_convolution_of_single_rows(K, C, col0, more, dtype):
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(K * C)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T = 3
    ctx = context([1] * T)
    src, taps, bias, state = rand(T, C + col0 + 8).to(dtype), rand(K, C), rand(C), rand(T + 2, (K - 1) * C + more)
    before = state.clone()
    out = kernels.causal_conv_silu(src, col0, C, taps, bias, state, ctx)
    for t in range(T):
        slot = T - t
        held = before[slot, :(K - 1) * C].double().view(K - 1, C)
        u = torch.cat([held, src[t:t + 1, col0:col0 + C].double()])
        x = (u * taps.double()).sum(0) + bias.double()
        want = x * torch.sigmoid(x)
        bound = 4e-6 if dtype == torch.float32 else 2.0 ** -8        # (five products and sums; bfloat16: the result's rounding)
        assert ((out[t].double() - want).abs() / (want.abs() + 0.1)).max().item() <= bound
        assert torch.equal(state[slot, :(K - 1) * C].view(K - 1, C), u[1:].float())
    for slot in (0, T + 1):
        assert torch.equal(state[slot], before[slot])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("Hq,Hkv,D", [(2, 1, 16), (16, 16, 128), (33, 3, 64), (64, 8, 128), (80, 8, 128), (3, 1, 18)])
@pytest.mark.parametrize("with_bias", [False, True])
def test_norm_over_whole_rows(Hq, Hkv, D, with_bias, dtype):
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(Hq * D)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T, page, nq, nk, eps = 3, 16, Hq * D, Hkv * D, 1e-5
    ctx = context([1] * T)                            # at positions 0, 7 and 14
    proj, wq, wk = rand(T, nq + nk + 4), rand(nq), rand(nk)
    bq, bk = (rand(nq), rand(nk)) if with_bias else (None, None)
    pages, table = torch.zeros(T + 1, 2, Hkv, page, D, dtype=dtype, device="cuda"), torch.tensor([[2], [0], [3]], dtype=torch.int32, device="cuda")
    q = kernels.qk_whole_norm_append(proj, 0, nq, bq, bk, wq, wk, eps, Hq, Hkv, D, ctx, pages, table, page, True)
    rms = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    plus = lambda x, b: x.double() + (b.double() if b is not None else 0.0)
    bound = 4e-6 if dtype == torch.float32 else 2.0 ** -8
    near = lambda got, want: ((got.double() - want).abs() / (want.abs() + 1e-2)).max().item() <= bound
    assert near(q, rms(plus(proj[:, :nq], bq)) * wq.double())
    k = plus(proj[:, nq:nq + nk], bk)
    for t in range(T):
        held = pages[table[t, 0], :, :, 7 * t]
        assert near(held[0].reshape(-1), (rms(k) * wk.double())[t]) and near(held[1].reshape(-1), k[t])
    assert int((pages != 0).any(-1).sum()) == 2 * Hkv * T


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_row_normed_in_steps_of_any_size(dtype):
    """The norm over whole rows before a rotation: a row's bits do not hang on how many rows the step has."""
    from ninfer_amd_mi50_b200 import kernels
    Hq, Hkv, D, page, n = 17, 3, 64, 16, 149
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    proj, wq, wk, freq = rand(n, (Hq + 2 * Hkv) * D), rand(Hq * D), rand(Hkv * D), rand(16)
    seen = []
    for T in (1, 148, 149):
        ctx = context([1] * T)
        ctx.positions = torch.arange(T, dtype=torch.int32, device="cuda") % page
        pages = torch.zeros(n, 2, Hkv, page, D, dtype=dtype, device="cuda")
        table = torch.arange(T, dtype=torch.int32, device="cuda").view(T, 1)
        q = kernels.whole_norm_rope_append(proj[:T], 0, Hq * D, (Hq + Hkv) * D, None, None, None, wq, wk, 1e-5, freq, 32, 1.0,
                                           Hq, Hkv, D, D, ctx, pages, table, page, dtype)
        seen.append((q, pages))
    for q, pages in seen[:2]:
        T = q.shape[0]
        assert torch.equal(q, seen[2][0][:T]) and torch.equal(pages[:T], seen[2][1][:T])
