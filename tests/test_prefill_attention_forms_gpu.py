"""The forms of the tcgen05 prefill attention (csrc/attention_prefill_tc.cu) at the edges of a tile and of a window."""

import math

import pytest
import torch

from test_kernels_gpu import _step_context, make_cache_case, tol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,page", [(64, 32), (128, 64)])
@pytest.mark.parametrize("window", [0, 1, 129, 200])
@pytest.mark.parametrize("form", ["softmax", "capped", "sigmoid", "biased"])
def test_forms_at_the_edges(D, page, window, form, monkeypatch):
    from ninfer_amd_mi50_b200 import kernels
    dtype, Hq, Hkv, scale = torch.bfloat16, 4, 2, 1 / math.sqrt(D)
    seg_lens, pos0s = [2, 127, 128, 129, 255, 256, 257, 385], [700, 0, 5, 127, 0, 128, 63, 300]
    n_pages = sum((p + n + page - 1) // page for p, n in zip(pos0s, seg_lens)) + 2
    pages, bt, c, qkv = make_cache_case(dtype, Hq, Hkv, D, page, seg_lens, pos0s, n_pages, 7 + window)
    bias = torch.linspace(-1.0, 1.0, Hq, device="cuda")
    gate = torch.linspace(-3.0, 3.0, qkv.shape[0] * (Hq + 1), device="cuda").view(-1, Hq + 1)
    keep = 5 if window != 129 else 150                # (150: kept keys that reach into a second block)

    def attend(rows, lens, at, table, how):
        for k, v in how.items():
            monkeypatch.setitem(kernels.TUNING, k, v)
        part = type(c)(positions=c.positions[rows], row_seg=torch.repeat_interleave(
            torch.arange(len(lens), device="cuda"), torch.tensor(lens, device="cuda")).int())
        ctx = _step_context(part, lens, at, dtype, 1024)
        q = qkv[rows].contiguous()
        if form == "sigmoid":
            return kernels.biased_window_attention(q[:, :Hq * D].contiguous(), Hq, Hkv, D, pages, table, page, ctx, window, 0,
                                                   scale, None, sigmoid_bias=bias)
        if form == "biased":
            return kernels.biased_window_attention(q[:, :Hq * D].contiguous(), Hq, Hkv, D, pages, table, page, ctx, window, keep,
                                                   scale, 0.01 * (bias + 1.0), gate[rows].contiguous(), 1)
        return kernels.paged_attention(q, Hq, Hkv, D, pages, table, page, ctx, window, scale,
                                       softcap=20.0 if form == "capped" else 0.0)

    fast = {"prefill_attention_tc_min_rows": 1, "bf16_attention": "auto"}
    every = list(range(sum(seg_lens)))
    out = attend(every, seg_lens, pos0s, bt, fast)
    assert kernels.tensor_core_status() == 0
    ref = attend(every, seg_lens, pos0s, bt, {"bf16_attention": "generic"})
    # sigmoid weights are not normalised: up to 685 of them below 1, each rounded to 2^-9, on values of unit size miss by
    # 2^-9 / sqrt(3) sqrt(685 / 3) = 0.017 on average, six times that at most
    torch.testing.assert_close(out.float(), ref.float(), **tol(dtype, 6.4 if form == "sigmoid" else 1.0))
    # the longest segment again, in portions that begin elsewhere in a tile: a row's sums depend on its position alone
    first, n, p0 = sum(seg_lens[:-1]), seg_lens[-1], pos0s[-1]
    for a, b in ((0, 130), (130, n)):
        rows = list(range(first + a, first + b))
        again = attend(rows, [b - a], [p0 + a], bt[-1:].contiguous(), fast)
        assert torch.equal(again, out[rows])


@pytest.mark.parametrize("D,page", [(64, 32), (128, 64)])
@pytest.mark.parametrize("window", [0, 300])
def test_biased_form_leaves_out_what_a_page_held_before(D, page, window, monkeypatch):
    """Rows of a request's last page behind its end, which hold another's infinities and NaN: the same bits."""
    from ninfer_amd_mi50_b200 import kernels
    dtype, Hq, Hkv = torch.bfloat16, 4, 2
    seg_lens, pos0s = [2, 127, 129, 250], [700, 0, 5, 130]
    ends = [p + n for p, n in zip(pos0s, seg_lens)]
    n_pages = sum((e + page - 1) // page for e in ends) + 2
    pages, bt, c, qkv = make_cache_case(dtype, Hq, Hkv, D, page, seg_lens, pos0s, n_pages, 3)
    monkeypatch.setitem(kernels.TUNING, "prefill_attention_tc_min_rows", 1)
    ctx, q = _step_context(c, seg_lens, pos0s, dtype, 1024), qkv[:, :Hq * D].contiguous()
    slopes = torch.linspace(0.0, 0.02, Hq, device="cuda")

    def attend():
        out = kernels.biased_window_attention(q, Hq, Hkv, D, pages, bt, page, ctx, window, 5, 0.1, slopes)
        assert kernels.tensor_core_status() == 0
        return out

    want = attend()
    for s, e in enumerate(ends):
        if e % page:
            pages[bt[s, e // page], :, :, e % page:] = float("nan")
            pages[bt[s, e // page], :, :, e % page:, ::2] = float("inf")
    assert torch.equal(attend(), want) and want.isfinite().all()


@pytest.mark.parametrize("D,page", [(64, 32), (128, 64)])
@pytest.mark.parametrize("form", ["softmax", "biased"])
@pytest.mark.parametrize("heights", ["rising", "uneven"])
def test_reference_maximum_that_rises_block_after_block(D, page, form, heights, monkeypatch):
    """Scores that outgrow the reference maximum by more than 2^8 in every block of 128 keys, or in two out of three: O is
    scaled, by a millionth or less, while the product of the block before may still be adding to it."""
    from ninfer_amd_mi50_b200 import kernels
    dtype, Hq, Hkv, scale = torch.bfloat16, 4, 2, 1 / math.sqrt(D)
    seg_lens, pos0s = [129, 300, 128, 257], [0, 723, 896, 40]
    n_pages = sum((p + n + page - 1) // page for p, n in zip(pos0s, seg_lens)) + 2
    pages, bt, c, qkv = make_cache_case(dtype, Hq, Hkv, D, page, seg_lens, pos0s, n_pages, 17)
    slopes = None
    if form == "biased":
        slopes = torch.tensor([0.05, 0.12, 0.2, 0.3], device="cuda")      # 9 to 55 powers of two a block
        if heights == "uneven":
            slopes = torch.tensor([0.04, 0.044, 0.05, 0.06], device="cuda")      # around the 8 that a maximum is left at
    else:
        # the first number of every query undoes the scale: that of a key is what its score has more, 7 (10 powers of two) a block
        qkv.view(len(qkv), -1, D)[:, :Hq, 0] = math.sqrt(D)
        step = [0, 7, 14, 8, 22, 30, 29, 45, 60, 61, 70] if heights == "uneven" else [7 * b for b in range(11)]
        for s, (n, p0) in enumerate(zip(seg_lens, pos0s)):
            j = torch.arange(p0 + n, device="cuda")
            pages[bt[s, j // page].long(), 0, :, j % page, 0] = torch.tensor(step, device="cuda").to(dtype)[j // 128][:, None]
    q = qkv[:, :Hq * D].contiguous()

    def attend(**how):
        for k, v in how.items():
            monkeypatch.setitem(kernels.TUNING, k, v)
        ctx = _step_context(c, seg_lens, pos0s, dtype, 1024)
        if form == "biased":
            return kernels.biased_window_attention(q, Hq, Hkv, D, pages, bt, page, ctx, 0, 0, scale, slopes)
        return kernels.paged_attention(qkv, Hq, Hkv, D, pages, bt, page, ctx, 0, scale)

    out = attend(prefill_attention_tc_min_rows=1, bf16_attention="auto")
    again = [attend() for _ in range(20)]
    assert kernels.tensor_core_status() == 0
    torch.testing.assert_close(out.float(), attend(bf16_attention="generic").float(), **tol(dtype))
    assert all(torch.equal(o, out) for o in again)
