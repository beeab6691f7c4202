"""The embed_norm kernel equals gather, add and LayerNorm run one after the other (the same fp32 operations on the same
rounded sums: bit for bit in its vector form), counts bad ids and treats their table row as zeros; the executor uses it
exactly where nothing else reads what is between the three steps."""
import copy
import ctypes

import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu

import gpu_ops as G  # noqa: E402
from helpers import compile_with  # noqa: E402
from llcompiler_b200 import _capi as C  # noqa: E402
from llcompiler_b200.compiler import LLCompiler  # noqa: E402
from oracle.models import max_rel_err  # noqa: E402


def _embed_norm(table, ids, add, gamma, beta, out, eps, period, s0, s1, bad=None):
    p = C.LlcEmbedNormParams()
    ptr = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())
    p.table, p.ids, p.add, p.gamma, p.beta, p.out, p.bad_ids = ptr(table), ptr(ids), ptr(add), ptr(gamma), ptr(beta), ptr(out), ptr(bad)
    p.dtype = 8 if table.dtype is torch.bfloat16 else 4
    p.rows, p.d, p.vocab, p.period, p.add_s0, p.add_s1, p.eps = out.shape[0], out.shape[1], table.shape[0], period, s0, s1, eps
    C.check(C.lib().llc_cuda_embed_norm(ctypes.byref(p), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))


# one and several vectors per lane, partly filled ones, several rows per warp; rows that take the block form (30, 5000)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("b,s,d", [(1, 1, 8), (3, 11, 264), (2, 384, 768), (300, 37, 768), (1, 5, 1024), (2, 3, 30), (1, 2, 5000)])
@pytest.mark.parametrize("form", ["none", "position", "full"])
def test_matches_the_three_steps(dtype, b, s, d, form):
    g = torch.Generator().manual_seed(b + s + d)
    table, gamma, beta = (torch.randn(n, generator=g).cuda().to(dtype) for n in ((100, d), (d,), (d,)))
    ids = torch.randint(0, 100, (b * s,), generator=g).cuda()
    ids[b * s // 2] = 100                                               # one id past the table
    add = None if form == "none" else torch.randn(s if form == "position" else b * s, d, generator=g).cuda().to(dtype)
    x = torch.empty(b * s, d, device="cuda", dtype=dtype)
    G.gather(table, ids, x)
    if add is not None:
        y = torch.empty_like(x)
        G.eltwise(y.view(b, s, d), [x.view(b, s, d), add.view(1, s, d).expand(b, s, d) if form == "position" else add.view(b, s, d)], "ld0;ld1;add,0,1")
        x = y
    want, bad = torch.empty_like(x), torch.zeros(1, dtype=torch.int32, device="cuda")
    G.layernorm(x, gamma, beta, want, 1e-6)
    for off in (0, 1):                                                  # a result that starts off a 16-byte boundary takes the block form
        out = torch.full((b * s * d + 1,), float("nan"), device="cuda", dtype=dtype)[off:off + b * s * d].view(b * s, d)
        bad.zero_()
        _embed_norm(table, ids, add, gamma, beta, out, 1e-6, s, 0 if form == "position" else s * d, d, bad)
        assert bad.item() == 1
        if off == 0 and d % 8 == 0 and d <= 1024:
            assert torch.equal(out, want)
        else:                                                           # another order of the row sums: a few ulp of fp32, one of the storage type
            assert torch.allclose(out.float(), want.float(), rtol=2e-2 if dtype is torch.bfloat16 else 1e-4, atol=1e-2 if dtype is torch.bfloat16 else 1e-4)


class _Front(nn.Module):
    def __init__(self, form, d=32):
        super().__init__()
        self.form = form
        self.tok, self.pos, self.ln = nn.Embedding(50, d), nn.Embedding(16, d), nn.LayerNorm(d)
        self.register_buffer("pos_ids", torch.arange(16))

    def forward(self, ids, extra):
        t, p = self.tok(ids), self.pos(self.pos_ids[:ids.shape[1]])
        if self.form == "token":                    # no add
            return self.ln(t)
        if self.form == "position":
            return self.ln(t + p)
        if self.form == "position_first":
            return self.ln(p + t)
        if self.form == "full":                     # an added row per token, in caller memory
            return self.ln(t + extra)
        if self.form == "sum_read_twice":           # the sum has another reader
            return self.ln(t + p) + (t + p)
        if self.form == "token_read_twice":
            return self.ln(t + p), t * 2.0
        if self.form == "three":                    # more than one add
            return self.ln(t + p + extra)
        if self.form == "scaled":
            return self.ln(t * 3.0 + p)
        raise ValueError(self.form)


def _run(m, dynamic, *args):
    comp = LLCompiler()
    with torch.no_grad():
        out = compile_with(comp, copy.deepcopy(m).cuda(), dynamic)(*(a.cuda() for a in args))
    torch.cuda.synchronize()
    return out, comp.compiled[0].engine


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("form,fused", [("token", True), ("position", True), ("position_first", True), ("full", True), ("sum_read_twice", False), ("token_read_twice", False),
                                        ("three", False), ("scaled", False)])
def test_fronts(form, fused, dtype):
    torch.manual_seed(0)
    m = _Front(form).to(dtype).eval()
    ids, extra = torch.randint(0, 50, (3, 11)), torch.randn(3, 11, 32).to(dtype)
    got, eng = _run(m, False, ids, extra)
    with torch.no_grad():
        want = m.float()(ids, extra.float())
    for g, w in zip(got, want) if isinstance(want, tuple) else [(got, want)]:
        assert max_rel_err(g, w) < (1e-5 if dtype is torch.float32 else 3e-2)
    assert (eng.executor.last_launch_count() == 1) == fused
    if form == "full":                              # the added tensor may start anywhere
        off = torch.cat([extra.flatten()[:1], extra.flatten()])[1:].view(3, 11, 32)
        shifted = torch.empty(3 * 11 * 32 + 1, dtype=dtype, device="cuda")[1:].view(3, 11, 32)
        shifted.copy_(off)
        with torch.no_grad():
            assert max_rel_err(eng.run(ids.cuda(), shifted)[0], want) < (1e-5 if dtype is torch.float32 else 3e-2)


def test_odd_widths_and_symbolic_lengths_stay_correct():
    torch.manual_seed(0)
    for d, dynamic in ((30, False), (32, True)):
        m = _Front("position", d).eval()
        ids, extra = torch.randint(0, 50, (3, 11)), torch.randn(3, 11, d)
        got, eng = _run(m, dynamic, ids, extra)
        with torch.no_grad():
            assert max_rel_err(got, m(ids, extra)) < 1e-5
