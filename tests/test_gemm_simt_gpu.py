"""The FMA GEMM's tiles and K slices against float64: 128 x 128, 64 x 64 and 64 x 16 tiles, one to eight slices (clusters along
K), operands that cannot be read as vectors, both orders of B, batches.  Bound: fp32 products and sums in blocks, each at
most K * 2^-24 of the sum of magnitudes, checked as 2^-24 * (K + 8) * |A| |B| per element (bf16: plus one rounding, 2^-8)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import gpu_ops as G  # noqa: E402


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("b0,b1,m,n,k", [(1, 1, 64, 512, 784), (1, 1, 64, 10, 512), (1, 1, 1, 1000, 777), (1, 1, 1021, 512, 784), (1, 1, 200, 130, 33), (1, 1, 129, 65, 256),
                                         (2, 3, 70, 40, 300), (1, 1, 5, 3, 1), (1, 1, 64, 16, 4099), (1, 1, 4096, 300, 64), (7, 1, 130, 257, 100)])
@pytest.mark.parametrize("kmajor", [True, False])
def test_fma_gemm(dtype, b0, b1, m, n, k, kmajor):
    g = torch.Generator().manual_seed(m + n + k)
    a = torch.randn(b0, b1, m, k, generator=g).cuda().to(dtype)
    b = torch.randn(b0, b1, *((n, k) if kmajor else (k, n)), generator=g).cuda().to(dtype)
    bk = b.transpose(-1, -2) if kmajor else b                  # [.., K, N]
    shift, res = torch.randn(n, generator=g).cuda(), torch.randn(b0, b1, m, n, generator=g).cuda().to(dtype)
    want = (a.double() @ bk.double()) * 0.5 + shift.double() + res.double()
    bound = (k + 8) * 2.0 ** -24 * (a.double().abs() @ bk.double().abs() + shift.double().abs() + res.double().abs())
    out = torch.full((b0, b1, m, n), float("nan"), device="cuda", dtype=dtype)
    if dtype is torch.bfloat16:                                # keep bf16 operands on the FMA path: its products stay below 2^18 or B rows are unaligned
        bound = bound + 2.0 ** -7 * want.abs()
    G.gemm(a, bk, out, shift=shift, res=res, alpha=0.5, prec="fp32" if dtype is torch.float32 else "bf16")
    assert ((out.double() - want).abs() <= bound).all()


def test_k_slices_are_reproducible_and_streams_share_nothing():
    a, b = torch.randn(1, 1, 64, 784, device="cuda"), torch.randn(1, 1, 512, 784, device="cuda").transpose(-1, -2)
    outs, streams = [torch.empty(1, 1, 64, 512, device="cuda") for _ in range(8)], [torch.cuda.Stream() for _ in range(8)]
    torch.cuda.synchronize()
    for o, s in zip(outs, streams):
        with torch.cuda.stream(s):
            G.gemm(a, b, o)
    torch.cuda.synchronize()
    assert all(torch.equal(outs[0], o) for o in outs)
