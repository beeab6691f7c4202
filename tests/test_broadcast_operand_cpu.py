"""Residuals and masks that are computed from broadcast operands: computed once per distinct element, read back through
stride 0, and the same function as the model in every broadcast form."""
import math

import pytest
import torch

from helpers import InterpreterCompiler, compile_with
from oracle.models import max_rel_err


class _Scores(torch.nn.Module):
    def forward(self, q, k, v, m):                       # heads beside the head size, as the projections leave them
        q, k, v = (t.permute(0, 2, 1, 3) for t in (q, k, v))
        s = torch.matmul(q, k.transpose(-1, -2)) / math.sqrt(64) + (1.0 - m.to(q.dtype)) * -100.0
        return torch.matmul(torch.softmax(s, dim=-1), v)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mask_shape,elements", [((2, 1, 1, 24), 48), ((2, 1, 16, 24), 768), ((1, 3, 1, 1), 3), ((1, 1, 16, 1), 16), ((2, 3, 16, 24), 2304), ((1, 1, 1, 1), 1)])
def test_masks_of_every_broadcast_form(dtype, mask_shape, elements):
    if dtype is torch.bfloat16 and mask_shape[3] == 1:
        elements *= 24                                   # fused attention reads masks along the keys: there they keep their extent
    g = torch.Generator().manual_seed(3)
    q, k, v = (torch.randn(2, n, 3, 64, generator=g).to(dtype) for n in (16, 24, 24))
    m = torch.randint(0, 2, mask_shape, generator=g)
    comp = InterpreterCompiler()
    fn = compile_with(comp, _Scores(), False)
    with torch.no_grad():
        got, want = fn(q, k, v, m), _Scores()(q.float(), k.float(), v.float(), m)
    assert max_rel_err(got, want) < (1e-5 if dtype is torch.float32 else 2e-2)
    steps = [s for s in comp.compiled[0].engine.text.splitlines() if s.startswith("step eltwise") and "#-100" in s]
    assert len(steps) == 1
    # bf16 attention is one step, with fp32 scores, for every form of mask (offsets on whole rows of bf16 scores lose them)
    assert ("step attention" in comp.compiled[0].engine.text) == (dtype is torch.bfloat16)
    out = steps[0].split("out=")[1].split("[")[1].split(";")[0]
    assert math.prod(int(e) for e in out.split(",")) == elements, steps[0]


@pytest.mark.parametrize("offset", [-1.0, -100.0, -10000.0])
@pytest.mark.parametrize("mask_shape", [(2, 1, 16, 1), (1, 3, 1, 1), (16, 1), (1, 1, 1, 1), (2, 1, 1, 24), (24,)])
def test_masks_do_not_cost_bf16_attention_its_fp32_scores(mask_shape, offset):
    """An offset that is the same for all keys of a row changes nothing: the error stays that of bf16 operands and results
    (2^-8 of the largest value), however large the offset is."""
    class Scores(torch.nn.Module):
        def forward(self, q, k, v, m):
            q, k, v = (t.permute(0, 2, 1, 3) for t in (q, k, v))
            s = torch.matmul(q, k.transpose(-1, -2)) / math.sqrt(64) + (1.0 - m.to(q.dtype)) * offset
            return torch.matmul(torch.softmax(s, dim=-1), v)

    g = torch.Generator().manual_seed(3)
    q, k, v = (torch.randn(2, n, 3, 64, generator=g).bfloat16() for n in (16, 24, 24))
    m = torch.randint(0, 2, mask_shape, generator=g)
    comp = InterpreterCompiler()
    fn = compile_with(comp, Scores(), False)
    with torch.no_grad():
        got, want = fn(q, k, v, m), Scores()(q.double(), k.double(), v.double(), m)
    assert max_rel_err(got, want) < 2 * 2.0 ** -8        # (probabilities and results are rounded to bf16)
    assert "step attention" in comp.compiled[0].engine.text


class _Residual(torch.nn.Module):
    def __init__(self):
        super().__init__()
        self.fc = torch.nn.Linear(32, 48)

    def forward(self, x, r):
        return torch.relu(self.fc(x) + torch.tanh(r) * 2.0)


@pytest.mark.parametrize("shape", [(10, 48), (1, 48), (10, 1), (1, 1)])
@pytest.mark.parametrize("dynamic", [False, True])
def test_broadcast_residuals_of_a_linear_layer(shape, dynamic):
    torch.manual_seed(0)
    m = _Residual()
    x, r = torch.randn(10, 32), torch.randn(shape)
    comp = InterpreterCompiler()
    fn = compile_with(comp, m, dynamic)
    with torch.no_grad():
        assert max_rel_err(fn(x, r), m(x, r)) < 1e-5
