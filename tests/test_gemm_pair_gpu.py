"""CTA-pair tiles (256 x 256, cta_group::2) of the tensor-core GEMM and convolution against float64 on the same operands, and
the per-column factors of every tile kind.  LLC_TC_PAIR=2 sends every shape to the pair kernels.  Bounds (2-norm): bf16
results carry one rounding of 2^-9 of each value, at most 2^-9 = 2e-3 in norm; tf32 operands are cut to 10 mantissa bits,
at most 2^-10 each, so 2e-3 for a product and less for sums of independent ones."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

import gpu_ops as G  # noqa: E402
from llcompiler_b200 import _capi as C  # noqa: E402

DT = {"bf16": torch.bfloat16, "tf32": torch.float32}


def _rand(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).cuda()


def _close(got, want):
    assert C.lib().llc_cuda_status() == 0
    assert ((got.double() - want).norm() / want.norm()).item() < 2e-3


@pytest.fixture(autouse=True)
def _every_shape(monkeypatch):
    monkeypatch.setenv("LLC_TC_MIN_MACS_LOG2", "0")


# one tile; rows that end in the first or the second CTA of a pair; ragged columns; K tails; several rounds per CTA; batches
@pytest.mark.parametrize("prec", ["bf16", "tf32"])
@pytest.mark.parametrize("b0,b1,m,n,k", [(1, 1, 256, 256, 64), (1, 1, 100, 256, 128), (1, 1, 129, 264, 96), (1, 1, 385, 136, 200), (1, 1, 20000, 520, 72), (2, 3, 300, 256, 128)])
@pytest.mark.parametrize("res", [False, True])
def test_pair_gemm(monkeypatch, prec, b0, b1, m, n, k, res):
    monkeypatch.setenv("LLC_TC_PAIR", "2")
    dt = DT[prec]
    a, b = _rand(b0, b1, m, k, seed=1).to(dt), _rand(b0, b1, n, k, seed=2).to(dt)
    scale, shift = _rand(n, seed=3), _rand(n + 1, seed=4)[1:]          # factors that do not start on a 16-byte boundary
    r = _rand(b0, b1, m, n, seed=5).to(dt) if res else None
    out = torch.full((b0, b1, m, n), float("nan"), device="cuda", dtype=dt)
    G.gemm(a, b.transpose(-1, -2), out, scale=scale, shift=shift, res=r, alpha=0.5, act="relu", prec=prec)
    want = 0.5 * scale.double() * (a.double() @ b.double().transpose(-1, -2)) + shift.double()
    _close(out, torch.relu(want + r.double() if res else want))


@pytest.mark.parametrize("prec", ["bf16", "tf32"])
@pytest.mark.parametrize("n,c,h,f,k,s", [(1, 64, 8, 256, 3, 1), (3, 128, 9, 136, 3, 2), (40, 64, 28, 256, 1, 2), (2, 64, 30, 300, 3, 1)])
def test_pair_conv(monkeypatch, prec, n, c, h, f, k, s):
    monkeypatch.setenv("LLC_TC_PAIR", "2")
    dt, p = DT[prec], k // 2
    oh = (h + 2 * p - k) // s + 1
    f -= f % (8 if prec == "bf16" else 4)
    x, w = _rand(n, h, h, c, seed=1).to(dt), _rand(f, k, k, c, seed=2).to(dt)
    scale, shift, r = _rand(f, seed=3), _rand(f, seed=4), _rand(n, oh, oh, f, seed=5).to(dt)
    out = torch.full((n, oh, oh, f), float("nan"), device="cuda", dtype=dt)
    G.conv2d(x, w, out, (s, s), (p, p), scale=scale, shift=shift, res=r, prec=prec)
    want = F.conv2d(x.double().permute(0, 3, 1, 2), w.double().permute(0, 3, 1, 2), stride=s, padding=p).permute(0, 2, 3, 1)
    _close(out, want * scale.double() + shift.double() + r.double())


# single-CTA tiles of every width, several column tiles per CTA, with and without each factor
@pytest.mark.parametrize("n", [64, 128, 250, 768])
@pytest.mark.parametrize("factors", ["", "shift", "scale", "both"])
@pytest.mark.parametrize("pair", ["0", "1"])
def test_column_factors(monkeypatch, n, factors, pair):
    monkeypatch.setenv("LLC_TC_PAIR", pair)
    a, b = _rand(30000, 64, seed=1).bfloat16(), _rand(n, 64, seed=2).bfloat16()
    scale = _rand(n, seed=3) if factors in ("scale", "both") else None
    shift = _rand(n, seed=4) if factors in ("shift", "both") else None
    out = torch.empty(1, 1, 30000, n, device="cuda", dtype=torch.bfloat16)
    G.gemm(a[None, None], b.t()[None, None], out, scale=scale, shift=shift, prec="bf16")
    want = a.double() @ b.double().t()
    want = want * (scale.double() if scale is not None else 1.0) + (shift.double() if shift is not None else 0.0)
    _close(out[0, 0], want)
