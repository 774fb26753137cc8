"""Kernels at the sizes where a new tile, copy width or split can go wrong, against plain float64 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from vllm_lite_b200.csrc import ops as o
    return o


# every tile of the float32 product (8 x 32, 32 x 32, 64 x 64, 128 x 128), its edges, K with and without 16-byte copies
@pytest.mark.parametrize("N,K", [(1, 1), (31, 4), (33, 63), (320, 96), (333, 97), (700, 260), (8193, 68)])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 33, 64, 65, 130])
def test_gemm_f32_tiles(M, N, K):
    gen = torch.Generator(device=DEV).manual_seed(M * 131 + N + K)
    a, w = torch.randn(M, K, device=DEV, generator=gen), torch.randn(N, K, device=DEV, generator=gen)
    out = torch.full((M, N), float("nan"), device=DEV)
    ops().gemm_f32(a, w, out)
    ref = a.double() @ w.double().T
    # K roundings of a running sum of products of the same sizes: at most K 2^-24 sum |a| |w|
    bound = (K + 1) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((out.double() - ref).abs() <= bound).all())
    one = torch.empty(1, N, device=DEV)
    ops().gemm_f32(a[M - 1:].contiguous(), w, one)
    assert torch.equal(one[0], out[M - 1])               # whichever tile made the row


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,I,group", [(1, 8, 0), (3, 4096, 0), (5, 12, 0), (2, 7, 0), (3, 64, 8), (3, 64, 16), (5, 36, 4), (7, 48, 24)])
def test_silu_mul_layouts(T, I, group, dtype):
    gu = (torch.randn(T, 2 * I, device=DEV) * 4).to(dtype)
    out = torch.empty(T, I, device=DEV, dtype=dtype)
    ops().silu_mul(gu, out, group=group)
    parts = gu.double().view(T, -1, 2, group or I)
    g, u = parts[:, :, 0].reshape(T, I), parts[:, :, 1].reshape(T, I)
    ref = g / (1 + torch.exp(-g)) * u
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6      # one rounding / a handful of them
    assert bool(((out.double() - ref).abs() <= rel * ref.abs() + 1e-30).all())
