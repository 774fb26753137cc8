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
