"""The elementwise chain kernels (row form and transposing tiles) against PyTorch on the same fp32 operations.  Sums,
products, maxima and ReLU are single correctly rounded fp32 operations and the storage conversion is round-to-nearest on
both sides, so the results are equal bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import gpu_ops as G  # noqa: E402


def _rand(shape, dtype, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).cuda().to(dtype)


def _nhwc(n, c, h, w, dtype, seed):
    return _rand((n, h, w, c), dtype, seed).permute(0, 3, 1, 2)


# tile edges: 64 x 64 tiles; extents that are multiples of 8, of 4, odd; below and above one tile
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("n,c,h,w", [(2, 64, 8, 8), (1, 32, 1, 8), (3, 72, 7, 7), (2, 128, 14, 14), (1, 33, 9, 13), (2, 100, 5, 12), (1, 512, 28, 28), (2, 65, 29, 29)])
def test_transposing_add_relu(dtype, n, c, h, w):
    a, b = _nhwc(n, c, h, w, dtype, 1), _rand((n, c, h, w), dtype, 2)
    want = torch.relu(a.float() + b.float()).to(dtype)
    out = torch.full_like(b, float("nan"))
    G.eltwise(out, [a, b], "ld0;ld1;add,0,1;relu,2")                  # NHWC + NCHW -> NCHW
    assert torch.equal(out, want.contiguous())
    out2 = torch.empty(n, h, w, c, device="cuda", dtype=dtype).permute(0, 3, 1, 2)
    G.eltwise(out2, [b, a], "ld0;ld1;sub,1,0;#0.5;mul,2,3;neg,4")      # -> NHWC, operands swapped in the subtraction
    assert torch.equal(out2, (-((a.float() - b.float()) * 0.5)).to(dtype))
    scale = _rand((c,), torch.float32, 3).view(1, c, 1, 1).expand(n, c, h, w)
    out3 = torch.empty_like(b)
    G.eltwise(out3, [a, scale, a], "ld0;ld1;mul,0,1;ld2;add,2,3")      # two transposed operands and a per-channel one
    assert torch.equal(out3, (a.float() * scale + a.float()).to(dtype).contiguous())


def test_transposing_copy_of_misaligned_views():
    base = _rand((2, 14, 14, 130), torch.bfloat16, 4)
    src = base[..., 1:129].permute(0, 3, 1, 2)                         # channels start 2 bytes past a 16-byte boundary
    out = torch.empty(2, 128, 14, 14, device="cuda", dtype=torch.bfloat16)
    G.eltwise(out, [src], "ld0")
    assert torch.equal(out, src.contiguous())
    wide = torch.zeros(2, 128, 14, 15, device="cuda", dtype=torch.bfloat16)
    G.eltwise(wide[..., 1:], [src], "ld0")                             # output rows of 14 inside 15, odd start
    assert torch.equal(wide[..., 1:], src) and not wide[..., 0].any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,d", [(1, 8), (5, 16), (3, 768), (130, 400), (7, 8192), (1000, 24)])
def test_rows(dtype, rows, d):
    a, b = _rand((rows, d), dtype, 5), _rand((1, d), dtype, 6).expand(rows, d)
    out = torch.empty_like(a)
    G.eltwise(out, [a, b], "ld0;ld1;add,0,1")
    assert torch.equal(out, (a.float() + b.float()).to(dtype))
    col = _rand((rows, 1), torch.float32, 7).expand(rows, d)
    G.eltwise(out, [a, col], "ld0;mul,0,0;ld1;max,2,1;#-1.5;min,4,3")  # the running value times itself, a per-row operand, swapped order
    assert torch.equal(out, torch.minimum(torch.maximum(a.float() * a.float(), col), torch.tensor(-1.5, device="cuda")).to(dtype))
    # three dims that do not merge, mixed storage types
    x = _rand((rows, 4, 2 * d), torch.float32, 8)[:, :, :d]
    y = torch.empty(rows, 4, d, device="cuda", dtype=dtype)
    G.eltwise(y, [x, a.view(rows, 1, d).expand(rows, 4, d)], "ld0;ld1;add,0,1;abs,2")
    assert torch.equal(y, (x + a.view(rows, 1, d).float()).abs().to(dtype))


# One step of every kind, with a second operand, a constant and itself, in both orders; one and two pieces per thread (below and
# above 1.2 M elements, 3.6 M in fp32).  The general kernel (odd columns) does the same fp32 operations; 2^-22 covers contractions.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(3, 768), (5, 7, 1032), (3200, 768), (900, 5, 1032)])
def test_one_step_programs(dtype, shape):
    x, y = _rand(shape, dtype, 10), _rand(shape, dtype, 11).abs() + 0.25
    unary = ["relu", "abs", "sqrt", "rsqrt", "exp", "gelu", "tanh", "erf", "sigmoid", "neg", "trunc", "tf32lo", "cast"]
    binary = ["add", "sub", "mul", "div", "max", "min", "pow", "eq", "ne", "ge", "gt", "le", "lt"]
    progs = ["ld1;%s,0" % o for o in unary] + ["ld0;ld1;%s,%s" % (o, r) for o in binary for r in ("0,1", "1,0") if (o, r) != ("pow", "0,1")]
    progs += ["ld1;#1.5;%s,%s" % (o, r) for o in ("sub", "div", "pow", "ge") for r in ("0,1", "1,0")] + ["ld1;mul,0,0", "ld1;div,0,0"]
    for prog in progs:
        out, want = torch.full_like(x, float("nan")), torch.full((*shape[:-1], shape[-1] + 1), float("nan"), device="cuda", dtype=dtype)[..., :-1]
        G.eltwise(out, [x, y], prog)
        G.eltwise(want[..., :-1], [x[..., :-1], y[..., :-1]], prog)
        torch.testing.assert_close(out[..., :-1].float(), want[..., :-1].float(), rtol=2.0 ** -22 if dtype is torch.float32 else 2.0 ** -8, atol=1e-38, msg=prog)
        assert not out.isnan().any(), prog


def test_rows_of_other_types():
    m = torch.randint(0, 2, (5, 384), generator=torch.Generator().manual_seed(9)).cuda()
    for t in (m, m.int(), m.bool(), m.half(), m.to(torch.int8)):
        out = torch.empty(5, 384, device="cuda")
        G.eltwise(out, [t], "#1;ld0;cast,1;sub,0,2;#-10000;mul,3,4")
        assert torch.equal(out, (1.0 - m.float()) * -10000.0)


def test_special_values_and_non_chain_programs_agree_with_the_general_path():
    v = torch.tensor([float("nan"), float("inf"), -float("inf"), -0.0, 3.0, -3.0, 1e-40, 65504.0] * 8, device="cuda")
    x, y = v.view(1, 64).repeat(40, 1), v.flip(0).view(64, 1).repeat(1, 40).t()
    for prog in ("ld0;ld1;max,0,1;relu,2", "ld0;ld1;div,1,0;sqrt,2", "ld0;ld1;min,0,1;exp,2", "ld0;ld1;gt,0,1;ld0;where,2,3,1"):
        big = torch.empty(40, 64, device="cuda")
        G.eltwise(big, [x, y], prog)
        small = torch.empty(40, 65, device="cuda")[:, :63]              # 63 columns: the general kernel
        G.eltwise(small, [x[:, :63], y[:, :63]], prog)
        assert torch.equal(torch.nan_to_num(big[:, :63], 7.0), torch.nan_to_num(small, 7.0)), prog
