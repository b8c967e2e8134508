"""The row norms and gates of csrc/norms.cu against float64, at widths that their wide form takes (runs of four, one to four
a thread) and at widths and offsets that it leaves to the others."""

import pytest
import torch

pytestmark = pytest.mark.gpu

WIDTHS = [4, 6, 124, 2044, 2048, 2052, 4100, 8192, 8196]


def close(got, want, dtype, what):
    # float32: every factor is rounded once or twice and the sums of squares in trees, a few 2^-24 of a result; bfloat16
    # results carry one rounding more (2^-9)
    bound = 2e-6 if got.dtype == torch.float32 else 2.0 ** -8
    err = ((got.double() - want).abs() / (want.abs() + 1e-3)).max().item()
    assert err <= bound, f"{what}: {err:.2e}"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", WIDTHS)
@pytest.mark.parametrize("col0", [0, 3, 8])
def test_norms_and_gates(n, col0, dtype):
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(n + col0)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T, eps, parts = 5, 1e-5, 2 if n % 2 == 0 and n < 4000 else 1
    rms = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    src, w, y = rand(T, n + col0 + 8).to(dtype), rand(n), rand(T, n)
    z = src[:, col0:col0 + n].double()
    close(kernels.rms_norm_slice(src, col0, n, w, eps), rms(z) * w.double(), dtype, "rms_norm_slice")
    grouped = lambda x: rms(x.view(T, parts, n // parts)).view(T, n)
    silu = lambda x: x * torch.sigmoid(x)
    close(kernels.gated_group_rmsnorm(y, src, col0, w, eps, parts, dtype), grouped(y.double() * silu(z)) * w.double(), dtype, "gated_group_rmsnorm")
    for gate, act in ((0, silu), (1, torch.sigmoid)):
        close(kernels.group_rmsnorm_gate(y, src, col0, w if gate else None, eps, parts, gate, dtype),
              grouped(y.double()) * (w.double() if gate else 1.0) * act(z), dtype, "group_rmsnorm_gate")
    delta, bias, scale, h = rand(T, n).to(dtype), rand(n), rand(n), rand(T, n)
    want = h.double() + scale.double() * rms(delta.double() + bias.double()) * w.double()
    out = kernels.scaled_norm_add(h, delta, bias, w, scale, eps, dtype)
    # (a sum of two terms: the bound is on their magnitudes, which a difference of nearly equal ones does not keep)
    assert (h.double() - want).abs().max().item() <= 4e-6 * want.abs().max().item()
    assert torch.equal(out, h.to(dtype))
    a, b = rand(T, n).to(dtype), rand(T, n).to(dtype)
    want = (rms(a.double()) * w.double() + rms(b.double()) * bias.double()) * 0.5
    got = kernels.mean_of_rmsnorms([a, b], [w, bias], eps)
    assert (got.double() - want).abs().max().item() <= 2e-6 * want.abs().max().item()
    heads, m = 3, n // 2
    v, gs = rand(heads, T, m).to(dtype), rand(T, heads * m + col0 + 8).to(dtype)
    for per_head in (False, True):
        gate = gs[:, col0:col0 + (heads if per_head else heads * m)].double().view(T, heads, -1)
        close(kernels.heads_sigmoid_gate(v, gs, col0, per_head), (v.double().transpose(0, 1) * torch.sigmoid(gate)).reshape(T, heads * m),
              dtype, "heads_sigmoid_gate")
