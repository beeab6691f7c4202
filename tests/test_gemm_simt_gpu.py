"""The two FMA GEMM kernels against float64: 128 x 128, 64 x 64 and 64 x 16 tiles of one to eight slices (clusters along K), the
other kernel's tiles and its slices through the workspace, operands that cannot be read as vectors, both orders of B, batches.
Bound: fp32 products and sums in blocks, each at
most K * 2^-24 of the sum of magnitudes, checked as 2^-24 * (K + 8) * |A| |B| per element (bf16: plus one rounding, 2^-8)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import gpu_ops as G  # noqa: E402


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("b0,b1,m,n,k", [(1, 1, 64, 512, 784), (1, 1, 64, 10, 512), (1, 1, 1, 1000, 777), (1, 1, 1021, 512, 784), (1, 1, 200, 130, 33), (1, 1, 129, 65, 256),
                                         (2, 3, 70, 40, 300), (1, 1, 5, 3, 1), (1, 1, 64, 16, 4099), (1, 1, 4096, 300, 64), (7, 1, 130, 257, 100),
                                         (1, 1, 2048, 2048, 256), (1, 1, 16, 300, 4096), (1, 1, 200, 1000, 1024), (1, 1, 600, 4096, 256)])
@pytest.mark.parametrize("kmajor", [True, False])
@pytest.mark.parametrize("scratch", [False, True])
def test_fma_gemm(dtype, b0, b1, m, n, k, kmajor, scratch):
    g = torch.Generator().manual_seed(m + n + k)

    def rows(r, c):                                            # a row stride of 4 more than a multiple of 8 elements: bf16 rows that TMA
        return torch.randn(b0, b1, r, c + (4 - c) % 8, generator=g).cuda().to(dtype)[..., :c]      # cannot start on stay on the FMA path

    a, b = rows(m, k), rows(n, k) if kmajor else rows(k, n)
    bk = b.transpose(-1, -2) if kmajor else b                  # [.., K, N]
    shift, res = torch.randn(n, generator=g).cuda(), torch.randn(b0, b1, m, n, generator=g).cuda().to(dtype)
    want = (a.double() @ bk.double()) * 0.5 + shift.double() + res.double()
    bound = (k + 8) * 2.0 ** -24 * (a.double().abs() @ bk.double().abs() + shift.double().abs() + res.double().abs())
    out = torch.full((b0, b1, m, n), float("nan"), device="cuda", dtype=dtype)
    if dtype is torch.bfloat16:
        bound = bound + 2.0 ** -8 * want.abs()                 # the result's rounding
    ws = torch.zeros(16 << 20, dtype=torch.uint8, device="cuda") if scratch else None
    G.gemm(a, bk, out, shift=shift, res=res, alpha=0.5, prec="fp32" if dtype is torch.float32 else "bf16", workspace=ws)
    assert ((out.double() - want).abs() <= bound).all()
    assert ws is None or int(ws[:4096].max()) == 0             # arrival counters are zero between launches


# The first product is 1 and each other one 2^-25, which a sum that holds 1 loses: what is missing from the result is the length
# of the sum the 1 went to.  Calls of few tiles have always summed a K slice of the idle SMs at a time, of at least 128.
@pytest.mark.parametrize("m,n,k", [(64, 10, 25088), (64, 10, 2048), (1, 1000, 2048), (16, 300, 4096), (64, 512, 784), (200, 300, 1024), (256, 256, 2048)])
def test_sums_of_calls_with_few_tiles_are_short(m, n, k):
    a, b = torch.ones(1, 1, m, k, device="cuda"), torch.full((1, 1, n, k), 2.0 ** -25, device="cuda")
    b[..., 0] = 1.0
    out = torch.empty(1, 1, m, n, device="cuda")
    G.gemm(a, b.transpose(2, 3), out, workspace=torch.zeros(16 << 20, dtype=torch.uint8, device="cuda"))
    slices = min(148 // (-(-m // 64) * -(-n // 64)), 32, k // 128)
    length = -(-(-(-k // slices)) // 16) * 16
    missing = 1.0 + (k - 1) * 2.0 ** -25 - out.double()
    assert missing.abs().max().item() <= length * 2.0 ** -25 + slices * 2.0 ** -24      # (and the roundings of the slices' sum)


def test_more_columns_than_a_grid_has_rows_of_64():
    n = 64 * 65535 + 100
    a, b = torch.randn(1, 1, 1, 8, device="cuda"), torch.randn(1, 1, n, 8, device="cuda")
    out = torch.full((1, 1, 1, n), float("nan"), device="cuda")
    G.gemm(a, b.transpose(2, 3), out)
    want = a.double() @ b.double().transpose(2, 3)
    assert ((out.double() - want).abs() <= 16 * 2.0 ** -24 * (a.double().abs() @ b.double().abs().transpose(2, 3))).all()


def test_k_slices_are_reproducible_and_streams_share_nothing():
    a, b = torch.randn(1, 1, 64, 784, device="cuda"), torch.randn(1, 1, 512, 784, device="cuda").transpose(-1, -2)
    outs, streams = [torch.empty(1, 1, 64, 512, device="cuda") for _ in range(8)], [torch.cuda.Stream() for _ in range(8)]
    torch.cuda.synchronize()
    for o, s in zip(outs, streams):
        with torch.cuda.stream(s):
            G.gemm(a, b, o)
    torch.cuda.synchronize()
    assert all(torch.equal(outs[0], o) for o in outs)


def test_the_entry_point_with_its_own_array_at_a_long_k():
    """64 x 10 x 8192 goes to the kernel whose K slices meet in that array; the second call finds what the first left there."""
    from ctypes import byref, c_void_p

    from llcompiler_b200 import _capi as C
    m, n, k = 64, 10, 8192
    a, b = torch.randn(1, 1, m, k, device="cuda"), torch.randn(1, 1, n, k, device="cuda")
    want, mag = a.double() @ b.double().transpose(2, 3), a.double().abs() @ b.double().abs().transpose(2, 3)
    for _ in range(2):
        out = torch.full((1, 1, m, n), float("nan"), device="cuda")
        p = C.LlcGemmParams()
        p.a, p.b, p.out = (c_void_p(t.data_ptr()) for t in (a, b, out))
        p.in_dtype = p.out_dtype = p.res_dtype = 4
        p.precision, p.alpha, p.act = C.PREC["fp32"], 1.0, C.ACT["none"]
        p.b0, p.b1, p.m, p.n, p.k, p.a_sm, p.b_sk, p.b_sn, p.o_sm = 1, 1, m, n, k, k, 1, k, n
        C.check(C.lib().llc_cuda_gemm_static_scratch(byref(p), c_void_p(torch.cuda.current_stream().cuda_stream)))
        torch.cuda.synchronize()
        assert ((out.double() - want).abs() <= (k // 32 + 40) * 2.0 ** -24 * mag).all()      # 32 slices, summed in order
