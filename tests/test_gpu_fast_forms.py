"""Kernels that have a fast form for aligned or common sizes: the fast form against the general one, or against 64-bit
sums, at the sizes where a tile ends, a remainder begins or the rule changes over."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def K():
    from servelab_b200.ops import kernels
    return kernels


def gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


# ------------------------------------------------- float32 product in 16-byte pieces
@pytest.mark.parametrize("M", [1, 15, 16, 17, 33, 64, 65, 257])
@pytest.mark.parametrize("N,Kd", [(1, 4), (63, 36), (64, 64), (130, 100), (1152, 896), (9728, 32)])
def test_float32_product_is_that_of_the_plain_kernel(M, N, Kd):
    """Rows of a width that is no multiple of 4 go to the plain kernel: the same bits, since both add in k order."""
    g = gen(M * 7 + N)
    a, w = torch.randn(M, Kd + 4, device=DEV, generator=g), torch.randn(N, Kd + 4, device=DEV, generator=g)
    bias = torch.randn(N, device=DEV, generator=g)
    wide_a, wide_w = torch.empty(M, Kd + 5, device=DEV), torch.empty(N, Kd + 5, device=DEV)
    wide_a[:, 1:], wide_w[:, 1:] = a, w
    for b in (None, bias):
        fast, plain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
        K().gemm_simt(a[:, :Kd], w[:, :Kd], fast, b)
        K().gemm_simt(wide_a[:, 1:Kd + 1], wide_w[:, 1:Kd + 1], plain, b)
        assert torch.equal(fast, plain)
    # three products at once, a row's batches side by side (as the heads of a layer lie)
    heads_a, heads_w = torch.randn(M, 3, Kd, device=DEV, generator=g), torch.randn(3, N, Kd, device=DEV, generator=g)
    out = torch.empty(M, 3, N, device=DEV)
    K().gemm_simt_batched(heads_a, heads_w, out)
    one = torch.empty(M, N, device=DEV)
    for h in range(3):
        K().gemm_simt(heads_a[:, h].contiguous(), heads_w[h], one)
        assert torch.equal(out[:, h], one)
