"""Decode attention whose key blocks meet in a thread-block cluster (csrc/attention_decode.cu): the same bits as the blocks
merged by a second kernel, at the edges of a block and of a cluster."""

import math
from types import SimpleNamespace

import pytest
import torch

from test_kernels_gpu import make_cache_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,Hq,Hkv", [(16, 3, 1), (64, 4, 2), (128, 16, 16), (128, 28, 4), (256, 4, 2)])
@pytest.mark.parametrize("window", [0, 200])
@pytest.mark.parametrize("form", ["softmax", "capped"])
def test_same_bits_in_a_cluster(D, Hq, Hkv, window, form):
    from ninfer_amd_mi50_b200 import kernels
    from ninfer_amd_mi50_b200.kernels import ops
    lib, page = ops._lib.load(), 16
    for lengths, bound in (([1, 128], 128), ([129], 256), ([1000, 3], 1024), ([1024], 1024), ([256], 1024), ([1025], 1100)):
        pages, bt, c, qkv = make_cache_case(torch.bfloat16, Hq, Hkv, D, page, [1] * len(lengths), [n - 1 for n in lengths],
                                            sum((n + page - 1) // page for n in lengths) + 1, sum(lengths))
        ctx = SimpleNamespace(positions=c.positions, row_seg=c.row_seg, all_single=True, max_context=bound)
        outs = []
        try:
            for on in (0, 1):
                lib.nf_set_decode_cluster(on)
                outs.append(kernels.paged_attention(qkv, Hq, Hkv, D, pages, bt, page, ctx, window, 1 / math.sqrt(D),
                                                    softcap=20.0 if form == "capped" else 0.0))
        finally:
            lib.nf_set_decode_cluster(1)
        assert torch.equal(outs[0], outs[1]), (lengths, bound)
        assert outs[0].float().abs().sum() > 0


@pytest.mark.parametrize("D,Hq,Hkv,lengths,bound,clusters", [
    (16, 3, 1, [1000, 3], 1024, True), (64, 4, 2, [129], 256, True), (128, 16, 16, [1, 128], 128, True),
    (128, 16, 16, [1000], 1024, True), (128, 28, 4, [200], 256, True), (64, 8, 8, [700, 2, 513], 768, True),
    (128, 16, 16, [1000, 3], 1024, False),      # 256 CTAs
    (128, 28, 4, [1, 128], 128, False),         # a CTA would add up seven numbers a thread
    (128, 4, 2, [1025], 1100, False),           # nine blocks
    (256, 4, 2, [129], 256, False)])            # too much shared memory
@pytest.mark.parametrize("form", ["softmax", "capped", "sigmoid"])
@pytest.mark.parametrize("listed", [False, True])
def test_which_launches_are_clusters(D, Hq, Hkv, lengths, bound, clusters, form, listed):
    """Every form, for all rows of a step and for rows listed out of a longer one (whose places in the launch are not
    theirs in the step)."""
    from ninfer_amd_mi50_b200.kernels import ops
    lib, page = ops._lib.load(), 16
    before = [2] * 3 if listed else []          # rows of the step that are not listed
    lens = before + lengths
    pages, bt, c, qkv = make_cache_case(torch.bfloat16, Hq, Hkv, D, page, [1] * len(lens), [n - 1 for n in lens],
                                        sum((n + page - 1) // page for n in lens) + 1, sum(lens))
    ctx = SimpleNamespace(positions=c.positions, row_seg=c.row_seg, all_single=True, max_context=bound)
    rows = torch.arange(len(before), len(lens), dtype=torch.int32, device="cuda").flip(0).contiguous() if listed else None
    bias = torch.linspace(-1.0, 0.5, Hq, device="cuda") if form == "sigmoid" else None
    outs, ran = [], []
    try:
        for on in (0, 1):
            lib.nf_set_decode_cluster(on)
            lib.nf_decode_cluster_launches()
            out = torch.zeros(len(lens), Hq * D, dtype=torch.bfloat16, device="cuda")
            ops._decode_attention(qkv, Hq, Hkv, D, pages, bt, page, ctx, 0, 1 / math.sqrt(D), out, rows, len(lengths),
                                  sigmoid_bias=bias, softcap=20.0 if form == "capped" else 0.0)
            ran.append(int(lib.nf_decode_cluster_launches()))
            outs.append(out)
    finally:
        lib.nf_set_decode_cluster(1)
    assert ran == [0, int(clusters)]
    assert torch.equal(outs[0], outs[1])
    assert (outs[0][len(before):].float().abs().sum(1) > 0).all() and not outs[0][:len(before)].any()
