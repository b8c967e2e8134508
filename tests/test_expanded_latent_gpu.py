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


def test_a_segment_decides_for_itself():
    """A short portion with rotated dimensions keeps the folded form beside a long one that is expanded: beside decoded
    rows or behind the long one (its rows are then picked out), it gives what it gives alone."""
    from ninfer_amd_mi50_b200 import kernels
    from ninfer_amd_mi50_b200.config.model_config import PartSpec
    from ninfer_amd_mi50_b200.parts.base import CacheView
    from ninfer_amd_mi50_b200.parts.latent_attention import LatentAttention
    heads, R, width, short, long = 16, 512, 256, 40, 1024
    part = LatentAttention(width, heads, D, DR, D, R, None, (D + DR) ** -0.5, 1e-5, PartSpec.make("rotary_half_split", head_dim=DR, theta=1e4),
                           "x.")
    g = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    shapes = {t.name: (t.shape, t.role) for t in part.tensor_specs()}
    part.load(lambda name: rand(*shapes[name][0]) if shapes[name][1] == "vector" else
              (rand(*shapes[name][0]) * shapes[name][0][1] ** -0.5).bfloat16())
    rows = {n: rand(n, width).bfloat16() for n in (short, long, 1)}

    def run(lens):
        ctx = context(lens)
        ctx.seg_pos0_host, ctx.seg_pos0 = [0] * len(lens), torch.zeros_like(ctx.seg_pos0)
        ctx.positions, ctx.max_context = torch.cat([torch.arange(n, dtype=torch.int32, device="cuda") for n in lens]), max(lens)
        per = (max(lens) + PAGE - 1) // PAGE
        table = torch.arange(len(lens) * per, dtype=torch.int32, device="cuda").view(len(lens), per)
        pages = torch.zeros(len(lens) * per, PAGE, R + DR, dtype=torch.bfloat16, device="cuda")
        out = part.forward(torch.cat([rows[n] for n in lens]), ctx, CacheView(part.cache_spec(), pages, table, PAGE), None)
        kernels.check_status("latent attention")
        q = torch.empty(ctx.T, heads * (D + DR), dtype=torch.bfloat16, device="cuda")
        at = sum(lens[:lens.index(short)])
        return out[at:at + short].double(), kernels.can_expand_latent(q, heads, D, D, R, ctx, DR)

    alone, expanded = run([short])
    assert not expanded
    for lens in ([short, long], [1, short, long], [long, short], [1, long, short, 1]):
        # products of other row counts may round a few numbers the other way (2^-9 of each); the expanded form rounds all of
        # them at other places, 4e-3
        got, expanded = run(lens)
        assert ((got - alone).norm() / alone.norm()).item() <= 1e-3, lens
        assert expanded == [(lens.index(long),)]


@pytest.mark.parametrize("lens", [[2], [63, 1, 64], [257], [500, 300]])
@pytest.mark.parametrize("rank", [64, 72, 512])
def test_expanded_by_the_packed_product(lens, rank):
    """The latents read where they lie in the cached rows, by the experts' product, against the plain one."""
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + rank)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ctx = context(lens)
    T, per = sum(lens), (ctx.max_context + PAGE - 1) // PAGE
    table = torch.arange(len(lens) * per, dtype=torch.int32, device="cuda").flip(0).contiguous().view(len(lens), per)
    pages = rand(len(lens) * per, PAGE, rank + DR).bfloat16()
    q, w_kv = rand(T, H * (D + DR)).bfloat16(), (rand(2 * H * D, rank) * rank ** -0.5).bfloat16()
    outs = []
    for packed in (None, kernels.pack_weights(w_kv[None], swiglu=False)):
        out = torch.zeros((T, H * D), dtype=q.dtype, device="cuda")
        kernels.expanded_latent_attention(q, w_kv, H, D, pages, table, PAGE, ctx, (D + DR) ** -0.5, out, Dr=DR, packed=packed)
        kernels.check_status("expanded latent attention")
        assert kernels.tensor_core_status() == 0
        outs.append(out.double())
    # the same bfloat16 keys and values but where two orders of a float32 sum fall on either side of a rounding: such a
    # number is off by 2^-8 of itself, one in some hundreds
    assert ((outs[0] - outs[1]).norm() / outs[0].norm()).item() <= 1e-3
    assert outs[0].abs().sum() > 0


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_folded_rows_before_a_split_that_is_not_finite(bad):
    """A cached row that is not finite leaves alone the rows of the portion that see no key of its key block (64 keys), a
    split of its own here: the merge leaves out what such a split adds up."""
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(9)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    heads, p, n = 2, 56, 16                                  # positions 56 to 71
    ctx = context([n])
    ctx.seg_pos0_host, ctx.seg_pos0, ctx.max_context = [p], ctx.seg_pos0 + p, p + n
    ctx.positions = ctx.positions + p
    pages, table = rand(2, PAGE, R + DR).bfloat16(), torch.tensor([[1, 0]], dtype=torch.int32, device="cuda")
    q, q_abs = rand(n, heads * (D + DR)).bfloat16(), rand(heads, n, R).bfloat16()
    run = lambda: kernels.latent_attention(q_abs, q, D + DR, D, DR, pages, table, PAGE, ctx, None, 0.1)
    want = run()
    pages[0, 5, 3] = bad                                     # position 69
    got = run()
    assert torch.equal(got[:, :64 - p], want[:, :64 - p]) and not got[:, 69 - p:].isfinite().all()


@pytest.mark.parametrize("rotated", [0, DR])
@pytest.mark.parametrize("lens", [[257, 40], [2, 129, 130], [100, 1, 28]])
def test_requests_do_not_meet_in_a_block(lens, rotated):
    """Requests lie one after the other in the expanded matrix, and a block of 128 keys reaches from one into the next: what
    is not finite there stays behind."""
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ctx = context(lens)
    per = (ctx.max_context + PAGE - 1) // PAGE
    table = torch.arange(len(lens) * per, dtype=torch.int32, device="cuda").view(len(lens), per)
    pages = rand(len(lens) * per, PAGE, R + rotated).bfloat16()
    q, w_kv = rand(sum(lens), H * (D + rotated)).bfloat16(), (rand(2 * H * D, R) * R ** -0.5).bfloat16()

    def attend():
        out = torch.zeros((sum(lens), H * D), dtype=q.dtype, device="cuda")
        kernels.expanded_latent_attention(q, w_kv, H, D, pages, table, PAGE, ctx, 0.1, out, Dr=rotated)
        assert kernels.tensor_core_status() == 0
        return out

    want, before = attend(), sum(lens[:-1])
    pages[(len(lens) - 1) * per:, :, ::2] = float("inf")     # the last request's rows
    pages[(len(lens) - 1) * per:, :, 1] = float("nan")
    got = attend()
    assert torch.equal(got[:before], want[:before]) and not got[before:].isfinite().any()
