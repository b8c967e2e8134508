"""Latent attention with rotated dimensions and a sink over expanded keys and values, beside the folded form, both
against float64."""

import pytest
import torch

from test_chunk_recurrence_gpu import context

pytestmark = pytest.mark.gpu

H, D, DR, R, PAGE = 3, 128, 64, 64, 64


@pytest.mark.parametrize("lens", [[128], [129, 1, 127], [300, 2], [257, 640]])
@pytest.mark.parametrize("sharp", [False, True])
def test_expanded_against_folded(lens, sharp, monkeypatch):
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ctx = context(lens)
    T, held = sum(lens), [p + n for p, n in zip(ctx.seg_pos0_host, lens)]
    pages_of, pages = [], rand(64, PAGE, R + DR).bfloat16()
    for n in held:                                           # every request's pages, not in order
        first = sum(len(p) for p in pages_of)
        pages_of.append([63 - first - i for i in range((n + PAGE - 1) // PAGE)])
    width = max(len(p) for p in pages_of)
    table = torch.tensor([p + [-1] * (width - len(p)) for p in pages_of], dtype=torch.int32, device="cuda")
    q = (rand(T, H * (D + DR)) * (3.0 if sharp else 1.0)).bfloat16()        # sharp: rows that rest on one key
    w_kv = (rand(2 * H * D, R) * R ** -0.5).bfloat16()
    sink, scale = rand(H) * 2, (D + DR) ** -0.5
    sink[0] = 60.0 if sharp else -60.0                       # a sink that takes everything, one that takes nothing
    monkeypatch.setitem(kernels.TUNING, "latent_expand_rotated_min_ops", 0)      # (short ones too)
    assert kernels.can_expand_latent(q, H, D, D, R, ctx, DR)
    got = torch.zeros((T, H * D), dtype=q.dtype, device="cuda")
    kernels.expanded_latent_attention(q, w_kv, H, D, pages, table, PAGE, ctx, scale, got, Dr=DR, sink=sink)
    kernels.check_status("expanded latent attention")
    w_uk, w_uv = w_kv[:H * D].view(H, D, R), w_kv[H * D:].view(H, D, R)
    q_heads = q.view(T, H, D + DR)
    o_lat = kernels.latent_attention(kernels.heads_linear(q_heads[:, :, :D].transpose(0, 1), w_uk), q, D + DR, D, DR, pages, table,
                                     PAGE, ctx, sink, scale)
    folded = kernels.heads_linear(o_lat, w_uv.transpose(1, 2)).transpose(0, 1).reshape(T, H * D)
    row, off = 0, ([], [])
    for s, n in enumerate(lens):
        if n > 1:
            c = torch.cat([pages[p] for p in pages_of[s]])[:held[s]].double()
            k, v = (torch.einsum("jr,hdr->hjd", c[:, :R], w.double()) for w in (w_uk, w_uv))
            qd = q_heads[row:row + n].double().transpose(0, 1)
            score = (qd[..., :D] @ k.transpose(1, 2) + qd[..., D:] @ c[:, R:].T) * scale
            seen = torch.arange(held[s], device="cuda")[None] <= ctx.positions[row:row + n, None]
            score = torch.cat([score.masked_fill(~seen, -torch.inf), sink.double()[:, None, None].expand(H, n, 1)], -1)
            want = (torch.softmax(score, -1)[..., :-1] @ v).transpose(0, 1)
            o = [x[row:row + n].view(n, H, D).double() for x in (got, folded)]
            if sharp:
                assert o[0][:, 0].abs().max() < 1e-15
            for e, x in zip(off, o):
                e += [(x[:, h] - want[:, h]).norm() / want[:, h].norm() for h in range(1, H)]
        else:
            assert torch.equal(got[row], torch.zeros_like(got[row]))         # left as it was
        row += n
    # both round what stands before and after the softmax to bfloat16 (2^-9 of a value each), at different places: the form
    # that takes over may not be further off (a tenth is what the few rows of a segment of two scatter by)
    new, old = (torch.stack(e).square().mean().sqrt().item() for e in off)
    assert new <= 1.1 * old, (new, old)
