"""K slices and accumulators of the tensor-core kernel: every slice count, the tile widths and kinds that can be cut, what they
leave in the workspace they meet in, and the length of the sums.

Per-element bound: the products of the operands below are exact in fp32, an accumulator truncates each addition (2^-23 of what
it holds), so a sum of k products is off by at most (k + 8) * 2^-23 of the sum of magnitudes, wherever it is cut; tf32x3
drops A_lo * B_lo and reads A_lo, B_lo to 11 bits, 3 * 2^-20 of the magnitudes; a bf16 result is rounded once, 2^-8."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

import gpu_ops as G  # noqa: E402
from llcompiler_b200 import _capi as C  # noqa: E402


@pytest.fixture(autouse=True)
def _every_size(monkeypatch):
    monkeypatch.setenv("LLC_TC_MIN_MACS_LOG2", "0")


def _rand(*shape, seed, prec):
    x = torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).cuda()
    if prec == "tf32":
        x = (x.view(torch.int32) & -8192).view(torch.float32)      # what the tensor core reads of an fp32 operand
    return x.bfloat16() if prec == "bf16" else x


def _bound(k, mag, prec):
    return ((k + 8) * 2.0 ** -23 + (3 * 2.0 ** -20 if prec == "tf32x3" else 0.0)) * mag


def _workspace():
    return torch.zeros(16 << 20, dtype=torch.uint8, device="cuda")


# Calls of few tiles: no accumulator may add up more than the slices over the idle SMs would (four, of at least four K
# blocks).  The first product is 1 and each other one 2^-29, which an accumulator that holds 1 loses: what is missing from the
# result is the length of the sum the 1 went to.
@pytest.mark.parametrize("prec,block", [("bf16", 64), ("tf32", 32)])
@pytest.mark.parametrize("m,n,k", [(64, 128, 1024), (32, 768, 768), (128, 3072, 768), (300, 768, 768), (300, 768, 3072), (6272, 64, 1024), (64, 64, 1000)])
def test_sums_of_calls_with_few_tiles_are_short(prec, block, m, n, k):
    dt = torch.bfloat16 if prec == "bf16" else torch.float32
    a, b = torch.ones(1, 1, m, k, device="cuda", dtype=dt), torch.full((1, 1, n, k), 2.0 ** -29, device="cuda", dtype=dt)
    b[..., 0] = 1.0
    out = torch.empty(1, 1, m, n, device="cuda")
    G.gemm(a, b.transpose(2, 3), out, prec=prec, workspace=_workspace())
    blocks = -(-k // block)
    slices = min(3 if m == 6272 else 4, blocks // 4)                # 49 tiles leave room for three
    chain = -(-blocks // slices) * block
    missing = 1.0 + (k - 1) * 2.0 ** -29 - out.double()
    assert C.lib().llc_cuda_status() == 0
    assert missing.abs().max().item() <= chain * 2.0 ** -29 + 4 * 2.0 ** -23       # (and the roundings of the four partial sums' additions)


# Ragged rows and columns, K tails, batches, tiles of every width, units on nearly every SM (1024 x 768, 6272 x 64).
SHAPES = [(1, 1, 100, 72, 1000), (1, 1, 300, 256, 1536), (2, 3, 70, 200, 640), (1, 1, 1024, 768, 1096), (1, 1, 6272, 64, 1024)]


@pytest.mark.parametrize("slices", [2, 3, 4])
@pytest.mark.parametrize("prec", ["bf16", "tf32", "tf32x3"])
@pytest.mark.parametrize("b0,b1,m,n,k", SHAPES)
@pytest.mark.parametrize("res", [None, "bf16", "f32"])
def test_slices_meet(monkeypatch, slices, prec, b0, b1, m, n, k, res):
    monkeypatch.setenv("LLC_TC_SLICES", str(slices))
    a, b = _rand(b0, b1, m, k, seed=1, prec=prec), _rand(b0, b1, n, k, seed=2, prec=prec)
    shift = _rand(n, seed=3, prec="f32")
    r = None if res is None else _rand(b0, b1, m, n, seed=4, prec="f32").to(torch.bfloat16 if res == "bf16" else torch.float32)
    want = a.double() @ b.double().transpose(2, 3) + shift.double() + (r.double() if r is not None else 0.0)
    mag = a.double().abs() @ b.double().abs().transpose(2, 3) + shift.double().abs() + (r.double().abs() if r is not None else 0.0)
    want = torch.relu(want)
    ws = _workspace()
    for dt in (torch.float32, torch.bfloat16):
        bound = _bound(k, mag, prec) + (2.0 ** -8 * want.abs() if dt is torch.bfloat16 else 0.0)
        for _ in range(2):                                          # the second launch finds what the first left in the workspace
            out = torch.full((b0, b1, m, n), float("nan"), device="cuda", dtype=dt)
            G.gemm(a, b.transpose(2, 3), out, shift=shift, res=r, act="relu", prec=prec, workspace=ws)
            assert ((out.double() - want).abs() <= bound).all()
    assert C.lib().llc_cuda_status() == 0
    assert int(ws[:4096].max()) == 0                                # arrival counters are zero between launches
    if slices == 2:
        assert int(ws[4096:].max()) != 0                            # the slices did meet


@pytest.mark.parametrize("slices", [2, 3, 4])
@pytest.mark.parametrize("prec", ["bf16", "tf32", "tf32x3"])
def test_slices_of_a_convolution_meet(monkeypatch, slices, prec):
    monkeypatch.setenv("LLC_TC_SLICES", str(slices))
    x, w = _rand(3, 9, 7, 128, seed=1, prec=prec), _rand(200, 3, 3, 128, seed=2, prec=prec)
    out = torch.full((3, 5, 4, 200), float("nan"), device="cuda")
    G.conv2d(x, w, out, (2, 2), (1, 1), prec=prec, workspace=_workspace())
    conv = lambda p, q: F.conv2d(p.double().permute(0, 3, 1, 2), q.double().permute(0, 3, 1, 2), None, 2, 1).permute(0, 2, 3, 1)  # noqa: E731
    assert ((out.double() - conv(x, w)).abs() <= _bound(9 * 128, conv(x.abs(), w.abs()), prec)).all()
    assert C.lib().llc_cuda_status() == 0


# Launches on several streams at once, each with a workspace of its own.
@pytest.mark.parametrize("m,n,k", [(100, 72, 1000), (1024, 768, 1096)])
def test_overlapping_launches(monkeypatch, m, n, k):
    monkeypatch.setenv("LLC_TC_SLICES", "3")
    a, b = _rand(1, 1, m, k, seed=1, prec="bf16"), _rand(1, 1, n, k, seed=2, prec="bf16").transpose(2, 3)
    outs, streams, spaces = [torch.empty(1, 1, m, n, device="cuda") for _ in range(8)], [torch.cuda.Stream() for _ in range(8)], [_workspace() for _ in range(8)]
    torch.cuda.synchronize()
    for _ in range(3):
        for o, s, ws in zip(outs, streams, spaces):
            with torch.cuda.stream(s):
                G.gemm(a, b, o, prec="bf16", workspace=ws)
    torch.cuda.synchronize()
    assert all(torch.equal(outs[0], o) for o in outs)
    assert ((outs[0].double() - a.double() @ b.double()).abs() <= _bound(k, a.double().abs() @ b.double().abs(), "bf16")).all()
    assert C.lib().llc_cuda_status() == 0
