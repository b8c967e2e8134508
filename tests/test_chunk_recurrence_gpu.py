"""The chunked recurrences (csrc/chunk_recurrence.cu) against the recurrence walked row by row in float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu

# segments at the edges of a chunk (64 and 128 rows) and of its sixteens, beside short ones that the row-by-row kernel
# keeps, and more than a warp's lanes of them; the last two are several groups of chunks when the scratch is small
LENGTHS = [[64], [65, 1, 63], [127, 128, 129], [80, 3, 257], [1] * 33 + [70, 2, 200], [700], [300, 2, 130, 200, 70]]


def context(lens):
    from ninfer_amd_mi50_b200.parts.base import StepContext
    dev = torch.device("cuda")
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    S, T = len(lens), sum(lens)
    row0 = [sum(lens[:i]) for i in range(S + 1)]
    pos0 = [7 * s for s in range(S)]
    return StepContext(dtype=torch.bfloat16, device=dev, T=T, S=S, token_ids=ints([0] * T),
                       positions=ints([p + i for p, n in zip(pos0, lens) for i in range(n)]),
                       row_seg=ints([s for s, n in enumerate(lens) for _ in range(n)]), seg_row0=ints(row0), seg_pos0=ints(pos0),
                       seg_slot=ints([S - s for s in range(S)]), logit_rows=ints([0]), seg_len_host=list(lens),
                       seg_pos0_host=pos0, max_rows_per_seg=max(lens), max_context=max(p + n for p, n in zip(pos0, lens)))


def walk(q, k, v, a, w, S):
    """q, k [T, H, D], v [T, H, V], a, w [T, H], S [H, V, D], all float64."""
    out = []
    for t in range(len(q)):
        S = a[t][:, None, None] * S + (w[t][:, None] * v[t])[:, :, None] * k[t][:, None, :]
        out.append(torch.einsum("hvd,hd->hv", S, q[t]))
    return torch.stack(out), S


def close(got, want, what, bound=2e-6):
    # float32 throughout: every number carries 24 bits and sums run over at most a few hundred terms (their error grows
    # with the root of that); a dropped part of an operand (8 of its 24 bits) would show as 1e-5
    err = ((got.double() - want).norm() / want.norm()).item()
    assert err <= bound, f"{what}: {err:.2e}"


@pytest.mark.parametrize("lens", LENGTHS)
@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("slow", [False, True])
def test_scan_in_chunks(lens, N, slow, monkeypatch):
    from ninfer_amd_mi50_b200 import kernels
    monkeypatch.setitem(kernels.TUNING, "chunk_scan_min_rows", 63)
    H, P, G = 6, 64, 2
    if sum(lens) >= 700:
        monkeypatch.setitem(kernels.TUNING, "chunk_recurrence_max_mb", 1)
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + N)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ctx, T, C = context(lens), sum(lens), H * P + 2 * G * N
    xbc, proj = rand(T, C).bfloat16(), rand(T, 8 + H + 2).bfloat16()
    dt_bias, A_log, D = rand(H), rand(H) - (4.0 if slow else 0.0), rand(H)
    A_log[0] = 6.0                                    # decays that underflow
    off = 16
    state = rand(len(lens) + 2, off + H * P * N)
    before = state.double().clone()
    y = kernels.ssd_scan(xbc, 0, H * P, H * P + G * N, proj, 8, dt_bias, A_log, D, state, off, ctx, H, P, N, G)
    x = xbc.double()
    dt = torch.nn.functional.softplus(proj[:, 8:8 + H].double() + dt_bias.double(), threshold=1e9)
    heads = lambda c: x[:, c:c + G * N].view(T, G, N).repeat_interleave(H // G, 1)
    v, row = x[:, :H * P].view(T, H, P), 0
    for s, n in enumerate(lens):
        r, slot = slice(row, row + n), len(lens) - s
        want, S = walk(heads(H * P + G * N)[r], heads(H * P)[r], v[r], torch.exp(-torch.exp(A_log.double()) * dt[r]), dt[r],
                       before[slot, off:].view(H, P, N))
        close(y[r].view(n, H, P), want + D.double()[:, None] * v[r], f"outputs of segment {s}")
        close(state[slot, off:].view(H, P, N), S, f"state of segment {s}")
        row += n
    for slot in (0, len(lens) + 1):
        assert torch.equal(state[slot].double(), before[slot])
    assert torch.equal(state[:, :off].double(), before[:, :off])


@pytest.mark.parametrize("lens", LENGTHS)
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("silu", [False, True])
def test_linear_attention_in_chunks(lens, D, silu, monkeypatch):
    from ninfer_amd_mi50_b200 import kernels
    monkeypatch.setitem(kernels.TUNING, "chunk_linear_min_rows", 63)
    H, V = 5, 128
    if sum(lens) >= 700:
        monkeypatch.setitem(kernels.TUNING, "chunk_recurrence_max_mb", 1)
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + D)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ctx, T, width = context(lens), sum(lens), 2 * H * D + H * V
    src = rand(T, width + 8).bfloat16()
    decay = torch.tensor([1.0 - 2.0 ** -8, 0.9, 0.5, 1.0, 1e-30], device="cuda")
    freq = torch.tensor([1000.0 ** (-2.0 * i / D) for i in range(D // 2)], device="cuda")
    state = rand(len(lens) + 2, H * V * D)
    before = state.double().clone()
    out = kernels.decay_linear_attention(src, 0, H * D, 2 * H * D, decay, freq, D, 0.25, silu, state, ctx, H, D, V)
    act = torch.nn.functional.silu if silu else (lambda x: x)
    q, k, v = (act(src[:, c:c + H * d].double()).view(T, H, d) for c, d in ((0, D), (H * D, D), (2 * H * D, V)))
    angle = ctx.positions.float()[:, None] * freq            # the kernel's angle, a float32 product
    c, s = torch.cos(angle.double())[:, None], torch.sin(angle.double())[:, None]
    turn = lambda x: torch.cat([x[..., :D // 2] * c - x[..., D // 2:] * s, x[..., D // 2:] * c + x[..., :D // 2] * s], -1)
    q, k, row = turn(q), turn(k) * 0.25, 0
    ones = torch.ones(T, H, dtype=torch.float64, device="cuda")
    for i, n in enumerate(lens):
        r, slot = slice(row, row + n), len(lens) - i
        want, S = walk(q[r], k[r], v[r], ones[r] * decay.double(), ones[r], before[slot].view(H, V, D))
        close(out[r].view(n, H, V), want, f"outputs of segment {i}")
        close(state[slot].view(H, V, D), S, f"state of segment {i}")
        row += n
    for slot in (0, len(lens) + 1):
        assert torch.equal(state[slot].double(), before[slot])


@pytest.mark.parametrize("lens", LENGTHS)
@pytest.mark.parametrize("D,V", [(64, 64), (128, 128)])
@pytest.mark.parametrize("alike", [False, True])
def test_delta_rule_in_chunks(lens, D, V, alike, monkeypatch):
    from ninfer_amd_mi50_b200 import kernels
    monkeypatch.setitem(kernels.TUNING, "chunk_delta_min_rows", 63)
    H, G, off = 4, 2, 8
    if sum(lens) >= 700:
        monkeypatch.setitem(kernels.TUNING, "chunk_recurrence_max_mb", 1)
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + D)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ctx, T = context(lens), sum(lens)
    qkv, ab = rand(T, 2 * G * D + H * V + 8), rand(T, 2 * H + 3)
    if alike:                                         # keys that share a direction, written in full and hardly forgotten
        qkv[:, G * D:2 * G * D] = rand(1, G * D) + 0.5 * qkv[:, G * D:2 * G * D]
        ab[:, 1:1 + H] -= 6.0
        ab[:, 1 + H:1 + 2 * H] += 6.0
    qkv, ab = qkv.bfloat16(), ab.bfloat16()
    dt_bias, A_log = rand(H), rand(H)
    A_log[0] = 6.0 if not alike else A_log[0]         # decays that underflow
    state = rand(len(lens) + 2, off + H * V * D)
    before = state.double().clone()
    out = kernels.delta_rule(qkv, 0, G * D, 2 * G * D, ab, 1, 1 + H, dt_bias, A_log, D ** -0.5, state, off, ctx, H, G, D, V)
    unit = lambda x: (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
    q, k = (unit(qkv[:, c:c + G * D].double().view(T, G, D)) for c in (0, G * D))
    q, v = q * D ** -0.5, qkv[:, 2 * G * D:2 * G * D + H * V].double().view(T, H, V)
    gate = torch.exp(-torch.exp(A_log.double()) * torch.nn.functional.softplus(ab[:, 1:1 + H].double() + dt_bias.double(), threshold=1e9))
    beta = torch.sigmoid(ab[:, 1 + H:1 + 2 * H].double())
    # what is written for a key that resembles the ones before it is a difference of nearly equal numbers, row after row:
    # walked one by one in float32 such segments miss by up to 4.4e-6 (700 rows, D = 128)
    row, bound = 0, 8e-6 if alike else 2e-6
    for s, n in enumerate(lens):
        slot, want = len(lens) - s, []
        S = before[slot, off:].view(H, V, D)
        for t in range(row, row + n):
            S = gate[t][:, None, None] * S
            new = beta[t][:, None] * (v[t] - torch.einsum("hvd,hd->hv", S, k[t]))
            S = S + new[:, :, None] * k[t][:, None, :]
            want.append(torch.einsum("hvd,hd->hv", S, q[t]))
        close(out[row:row + n].view(n, H, V), torch.stack(want), f"outputs of segment {s}", bound)
        close(state[slot, off:].view(H, V, D), S, f"state of segment {s}", bound)
        row += n
    for slot in (0, len(lens) + 1):
        assert torch.equal(state[slot].double(), before[slot])
    assert torch.equal(state[:, :off].double(), before[:, :off])


@pytest.mark.parametrize("kind", ["scan", "linear", "delta"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [5, 70, 139])
def test_what_is_not_finite_stays_behind_its_row(kind, bad, at, monkeypatch):
    """A query, key, value or gate that is not a number, or infinite, leaves the rows before it as they were, bit for bit;
    a value also every other column of its head."""
    from ninfer_amd_mi50_b200 import kernels
    monkeypatch.setitem(kernels.TUNING, f"chunk_{kind}_min_rows", 63)
    lens, g = [141, 64], torch.Generator(device="cuda").manual_seed(at)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ctx, T = context(lens), sum(lens)
    H, G, D, V = 4, 2, 128, 64 if kind == "scan" else 128
    keys = H if kind == "linear" else G                       # heads that q and k have
    src, gates = rand(T, 2 * keys * D + H * V).bfloat16(), rand(T, 2 * H).bfloat16()
    q0, k0, v0 = 0, keys * D, 2 * keys * D
    bias, rate, first = rand(H), rand(H), rand(len(lens) + 2, H * V * D)

    def run(src, gates):
        state = first.clone()
        if kind == "scan":
            out = kernels.ssd_scan(src, v0, k0, q0, gates, 0, bias, rate, bias, state, 0, ctx, H, V, D, G)
        elif kind == "linear":
            out = kernels.decay_linear_attention(src, q0, k0, v0, torch.sigmoid(bias), None, 0, 1.0, False, state, ctx, H, D, V)
        else:
            out = kernels.delta_rule(src, q0, k0, v0, gates, 0, H, bias, rate, 0.1, state, 0, ctx, H, G, D, V)
        return out.view(T, H, V), state.view(-1, H, V, D)

    want, end = run(src, gates)
    assert want.isfinite().all() and end.isfinite().all()
    for col, of_row in ((q0 + 3, True), (k0 + 3, False), (v0 + 7, False)) + (((None, False),) if kind != "linear" else ()):
        s, ga = src.clone(), gates.clone()
        (ga if col is None else s)[at, 0 if col is None else col] = bad
        if col is None and bad > 0 and kind == "scan":
            continue                                          # (an infinite step size: a decay of nothing, fine to walk over)
        out, state = run(s, ga)
        assert torch.equal(out[:at], want[:at]), (col, "rows before")
        assert torch.equal(out[lens[0]:], want[lens[0]:]) and torch.equal(state[1], end[1]), (col, "the other request")
        if col == v0 + 7:
            assert not out[at:lens[0], 0, 7].isfinite().any() and not state[2, 0, 7].isfinite().all()
            others = torch.arange(V, device="cuda") != 7
            assert torch.equal(out[:, 0, others], want[:, 0, others]) and torch.equal(out[:, 1:], want[:, 1:])
        elif of_row:
            assert not out[at, 0].isfinite().any() and torch.equal(out[at + 1:], want[at + 1:]) and torch.equal(state, end)
        elif not (col is None and bad > 0):                   # (an infinite gate of the delta rule forgets everything)
            assert not out[at, 0].isfinite().any()


@pytest.mark.parametrize("lens,heads,chunks,walk", [
    ([128], 64, False, True),                          # too little for three launches more
    ([279, 162, 202, 244, 254, 40], 8, False, True),   # neither long nor much: one form, not both
    ([279, 162, 202, 244, 254, 64], 64, True, False),  # much work together
    ([1024], 4, True, False),                          # a long chain
    ([1, 1024, 63, 64], 4, True, True),                # what is too short for a chunk is walked beside it
    ([1] * 64, 64, False, True)])
def test_which_form_a_step_takes(lens, heads, chunks, walk, monkeypatch):
    from ninfer_amd_mi50_b200 import kernels
    from ninfer_amd_mi50_b200.kernels import ops
    P, N, G, called, call = 64, 128, 1, [], ops._lib.call
    monkeypatch.setattr(ops._lib, "call", lambda name, *a: (called.append(name), call(name, *a))[1])
    ctx, T = context(lens), sum(lens)
    xbc, dt = (torch.zeros(T, c, dtype=torch.bfloat16, device="cuda") for c in (heads * P + 2 * G * N, heads))
    one = torch.ones(heads, device="cuda")
    state = torch.zeros(len(lens) + 2, heads * P * N, device="cuda")
    kernels.ssd_scan(xbc, 0, heads * P, heads * P + G * N, dt, 0, one, one, one, state, 0, ctx, heads, P, N, G)
    assert called == ["nf_chunk_scan"] * chunks + ["nf_ssd_scan"] * walk


@pytest.mark.parametrize("kind", ["scan", "linear", "delta"])
def test_a_cut_shows_in_roundings_only(kind):
    """A prompt in one portion, and cut into portions of which some run in chunks (with TUNING as it stands) and some are
    walked: the same results and state but for float32 roundings."""
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T, H, G, D, V = 2300, 4, 2, 128, 64 if kind == "scan" else 128
    keys = H if kind == "linear" else G
    src, gates = rand(T, 2 * keys * D + H * V).bfloat16(), rand(T, 2 * H).bfloat16()
    bias, rate, first = rand(H), rand(H) - 3.0, rand(3, H * V * D)

    def run(cuts):
        state, outs, at = first.clone(), [], 0
        for n in cuts:
            ctx, s, ga = context([n]), src[at:at + n].contiguous(), gates[at:at + n].contiguous()
            if kind == "scan":
                o = kernels.ssd_scan(s, 2 * keys * D, keys * D, 0, ga, 0, bias, rate, bias, state, 0, ctx, H, V, D, G)
            elif kind == "linear":
                o = kernels.decay_linear_attention(s, 0, keys * D, 2 * keys * D, torch.sigmoid(bias), None, 0, 1.0, False, state,
                                                   ctx, H, D, V)
            else:
                o = kernels.delta_rule(s, 0, keys * D, 2 * keys * D, ga, 0, H, bias, rate, 0.1, state, 0, ctx, H, G, D, V)
            outs.append(o)
            at += n
        assert at == T
        return torch.cat(outs), state

    want = run([T])
    for cuts in ([1100, 1200], [1024, 1, 1023, 252], [300, 2000], [400, 700, 1000, 200]):
        got = run(cuts)
        for a, b in zip(got, want):
            close(a, b.double(), cuts, 4e-6)          # twice what one form may miss the exact result by
        assert not torch.equal(got[0], want[0]) or kind != "scan"       # (the forms do differ: this compares two)
