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
