"""The float32 products (csrc/gemm_f32.cu) at the edges of their tiles, against float64 and against the kernel that
serves rows which cannot be read 16 bytes at a time (the same sums in the same order: the same bits)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def close(got, want, K):
    # K products summed one after the other in float32: the error grows as sqrt(K) 2^-24 of the sum's norm; four times that
    assert (got.double() - want).norm() <= 4 * K ** 0.5 * 2 ** -24 * want.norm()


@pytest.mark.parametrize("M", [1, 4, 5, 16, 17, 33, 64, 65, 129, 300])
@pytest.mark.parametrize("N,K", [(1, 4), (33, 36), (64, 256), (130, 100)])
def test_dense(M, N, K):
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N)
    x, w = (torch.randn(r, K, generator=g, device="cuda") for r in (M, N))
    close(kernels.linear(x, w), x.double() @ w.double().T, K)
    if N % 2 == 0:
        gate, up = (x.double() @ w.double().T).split(N // 2, 1)
        close(kernels.linear_swiglu(x, w), torch.nn.functional.silu(gate) * up, 4 * K)
    close(kernels.linear_relu2(x, w), torch.relu(x.double() @ w.double().T) ** 2, 4 * K)
    # one element further on, the rows are no longer aligned
    wide = torch.randn(N * K + 1, generator=g, device="cuda")
    moved = wide[1:].view(N, K)
    assert moved.data_ptr() % 16 != 0
    assert torch.equal(kernels.linear(x, moved), kernels.linear(x, moved.clone()))


@pytest.mark.parametrize("T,E,k", [(1, 8, 2), (3, 60, 4), (40, 8, 2), (90, 4, 2), (200, 3, 3)])
def test_experts(T, E, k):
    from ninfer_amd_mi50_b200 import kernels
    H, inner = 68, 36
    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda") * 0.3
    x, w13, w2 = rand(T, H), rand(E, 2 * inner, H), rand(E, H, inner)
    idx = torch.stack([torch.randperm(E, generator=g, device="cuda")[:k] for _ in range(T)]).int()
    idx[: T // 2, 0], idx[: T // 2, 1] = 0, 1               # experts with many rows beside those with few or none
    plan = kernels.moe_plan(idx, E)
    y = kernels.moe_experts(x, w13, w2, plan, k)
    got = y[plan.inv.long().view(T, k).flatten()].view(T, k, H)
    e = idx.long()
    gate, up = torch.einsum("tkih,th->tki", w13.double()[e], x.double()).split(inner, 2)
    close(got, torch.einsum("tkhi,tki->tkh", w2.double()[e], torch.nn.functional.silu(gate) * up), 4 * (H + inner))


@pytest.mark.parametrize("N,K", [(32800, 2048), (20000, 2048)])
def test_matrices_beyond_l2(N, K):
    """More than twice L2 and more than once: other tiles for few rows, the same bits."""
    from ninfer_amd_mi50_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(N)
    wide = torch.randn(N * K + 1, generator=g, device="cuda")
    moved = wide[1:].view(N, K)                                # one element on: the kernel for rows that are not aligned
    w = moved.clone()
    for M in (4, 5, 10, 11, 24, 25):
        x = torch.randn(M, K, generator=g, device="cuda")
        got = kernels.linear(x, w)
        assert torch.equal(got, kernels.linear(x, moved)), M
        if M == 11:
            close(got, x.double() @ w.double().T, K)
            assert torch.equal(kernels.linear_swiglu(x, w), kernels.linear_swiglu(x, moved))
