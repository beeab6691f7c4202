"""Performance cases of the compiled-inference path.

Every case is a model or a single block in plain PyTorch that goes through the framework's public way in,
torch.compile(backend=LLCompiler()), once; what is measured is Torch_ExecutionEngine.run on tensors that live on
the GPU, one call after the other, as a serving loop makes them.  Sizes are those of the benchmark configurations
(MLP 784-512-10, ResNet-18/50 at 224x224, the d768/h12 encoder layer, BERT-base) and the ranges around them.

Kinds:
  mlp         Linear-ReLU-Linear, fp32 on the FMA path (precision "auto"): the latency-bound classifier head
  encoder     pre-LayerNorm encoder layer, fp32 storage with TF32 matmuls
  bert_layer  post-LayerNorm encoder layer with a padding mask, bf16
  embed       token + position embedding and LayerNorm, bf16
  bert        embeddings and n layers: a whole call, hidden states out
  basic       ResNet-18/34 block, fp32 at precision tf32x3 (fp32-grade results on tensor cores)
  bottleneck  ResNet-50 block, bf16
  stem        7x7/2 convolution, batch norm, ReLU, 3x3/2 max-pool, bf16
  resnet18    the whole network, fp32 at precision tf32x3, logits out
"""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F

from llcompiler_b200.compiler import LLCompiler

DEVICE = "cuda"
HEADS, HEAD = 12, 64
DTYPE = {"f32": torch.float32, "bf16": torch.bfloat16}


# ---- the models, in plain PyTorch ------------------------------------------------------------------
class Mlp(nn.Module):
    def __init__(self, d_in, hidden, d_out):
        super().__init__()
        self.fc1, self.fc2 = nn.Linear(d_in, hidden), nn.Linear(hidden, d_out)

    def forward(self, x):
        return self.fc2(torch.relu(self.fc1(x)))


class Attention(nn.Module):
    def __init__(self, heads):
        super().__init__()
        d = heads * HEAD
        self.h = heads
        self.q, self.k, self.v, self.o = nn.Linear(d, d), nn.Linear(d, d), nn.Linear(d, d), nn.Linear(d, d)

    def forward(self, x, add_mask=None):
        b, s, d = x.shape
        q = self.q(x).view(b, s, self.h, HEAD).permute(0, 2, 1, 3)
        k = self.k(x).view(b, s, self.h, HEAD).permute(0, 2, 1, 3)
        v = self.v(x).view(b, s, self.h, HEAD).permute(0, 2, 1, 3)
        scores = torch.matmul(q, k.transpose(-1, -2)) / math.sqrt(HEAD)
        if add_mask is not None:
            scores = scores + add_mask
        ctx = torch.matmul(torch.softmax(scores, dim=-1), v).permute(0, 2, 1, 3).reshape(b, s, d)
        return self.o(ctx)


class PreNormLayer(nn.Module):
    def __init__(self, heads, d_ff):
        super().__init__()
        d = heads * HEAD
        self.ln1, self.attn, self.ln2 = nn.LayerNorm(d), Attention(heads), nn.LayerNorm(d)
        self.ff1, self.ff2 = nn.Linear(d, d_ff), nn.Linear(d_ff, d)

    def forward(self, x):
        x = x + self.attn(self.ln1(x))
        return x + self.ff2(F.gelu(self.ff1(self.ln2(x))))


class PostNormLayer(nn.Module):
    def __init__(self, heads, d_ff):
        super().__init__()
        d = heads * HEAD
        self.attn, self.ln1 = Attention(heads), nn.LayerNorm(d, eps=1e-12)
        self.ff1, self.ff2, self.ln2 = nn.Linear(d, d_ff), nn.Linear(d_ff, d), nn.LayerNorm(d, eps=1e-12)

    def forward(self, x, add_mask):
        x = self.ln1(x + self.attn(x, add_mask))
        return self.ln2(x + self.ff2(F.gelu(self.ff1(x))))


def additive_mask(mask, dtype):
    return (1.0 - mask.to(dtype))[:, None, None, :] * -10000.0


class BertLayer(nn.Module):
    def __init__(self, heads, d_ff):
        super().__init__()
        self.layer = PostNormLayer(heads, d_ff)

    def forward(self, x, mask):
        return self.layer(x, additive_mask(mask, x.dtype))


class Embed(nn.Module):
    def __init__(self, vocab, max_pos, d):
        super().__init__()
        self.tok, self.pos, self.ln = nn.Embedding(vocab, d), nn.Embedding(max_pos, d), nn.LayerNorm(d, eps=1e-12)
        self.register_buffer("pos_ids", torch.arange(max_pos), persistent=False)

    def forward(self, ids):
        return self.ln(self.tok(ids) + self.pos(self.pos_ids[:ids.shape[1]]))


class Bert(nn.Module):
    def __init__(self, layers, vocab, max_pos, heads, d_ff):
        super().__init__()
        self.embed = Embed(vocab, max_pos, heads * HEAD)
        self.layers = nn.ModuleList([PostNormLayer(heads, d_ff) for _ in range(layers)])

    def forward(self, ids, mask):
        x = self.embed(ids)
        add_mask = additive_mask(mask, x.dtype)
        for layer in self.layers:
            x = layer(x, add_mask)
        return x


def conv(c_in, c_out, k, stride=1):
    return nn.Conv2d(c_in, c_out, k, stride, k // 2, bias=False)


class Basic(nn.Module):
    def __init__(self, c_in, c, stride):
        super().__init__()
        self.c1, self.b1 = conv(c_in, c, 3, stride), nn.BatchNorm2d(c)
        self.c2, self.b2 = conv(c, c, 3), nn.BatchNorm2d(c)
        self.down = nn.Sequential(conv(c_in, c, 1, stride), nn.BatchNorm2d(c)) if stride != 1 or c_in != c else None

    def forward(self, x):
        y = self.b2(self.c2(torch.relu(self.b1(self.c1(x)))))
        return torch.relu(y + (x if self.down is None else self.down(x)))


class Bottleneck(nn.Module):
    def __init__(self, c_in, c, stride):
        super().__init__()
        self.c1, self.b1 = conv(c_in, c, 1), nn.BatchNorm2d(c)
        self.c2, self.b2 = conv(c, c, 3, stride), nn.BatchNorm2d(c)
        self.c3, self.b3 = conv(c, 4 * c, 1), nn.BatchNorm2d(4 * c)
        self.down = nn.Sequential(conv(c_in, 4 * c, 1, stride), nn.BatchNorm2d(4 * c)) if stride != 1 or c_in != 4 * c else None

    def forward(self, x):
        y = torch.relu(self.b1(self.c1(x)))
        y = self.b3(self.c3(torch.relu(self.b2(self.c2(y)))))
        return torch.relu(y + (x if self.down is None else self.down(x)))


class Stem(nn.Module):
    def __init__(self):
        super().__init__()
        self.c, self.b, self.pool = conv(3, 64, 7, 2), nn.BatchNorm2d(64), nn.MaxPool2d(3, 2, 1)

    def forward(self, x):
        return self.pool(torch.relu(self.b(self.c(x))))


class ResNet18(nn.Module):
    def __init__(self, classes):
        super().__init__()
        self.stem = Stem()
        blocks, c_in = [], 64
        for c, stride in ((64, 1), (128, 2), (256, 2), (512, 2)):
            blocks += [Basic(c_in, c, stride), Basic(c, c, 1)]
            c_in = c
        self.blocks, self.pool, self.fc = nn.Sequential(*blocks), nn.AdaptiveAvgPool2d(1), nn.Linear(512, classes)

    def forward(self, x):
        return self.fc(torch.flatten(self.pool(self.blocks(self.stem(x))), 1))


# ---- cases -----------------------------------------------------------------------------------------
VOCAB, MAX_POS, D_FF = 30522, 512, 3072


def listed():
    return [
        # the smallest call: the MLP classifier at its configured batch, two launches, latency only
        {"name": "mlp_b64", "kind": "mlp", "batch": 64, "d_in": 784, "hidden": 512, "d_out": 10, "dynamic": False},
        # the same model with a symbolic batch, at an odd size
        {"name": "mlp_b1021_dynamic", "kind": "mlp", "batch": 1021, "d_in": 784, "hidden": 512, "d_out": 10, "dynamic": True},
        # fp32 encoder layer with TF32 matmuls at the two configured sequence lengths: a short request and a long one
        {"name": "encoder_tf32_s128", "kind": "encoder", "batch": 8, "seq": 128},
        {"name": "encoder_tf32_s512", "kind": "encoder", "batch": 8, "seq": 512},
        # one BERT-base layer: an online request batch with padding, a ragged one, and the full offline batch
        {"name": "bert_layer_b8_s128", "kind": "bert_layer", "batch": 8, "seq": 128, "padded": True},
        {"name": "bert_layer_b13_s217", "kind": "bert_layer", "batch": 13, "seq": 217, "padded": True},
        {"name": "bert_layer_b256_s384", "kind": "bert_layer", "batch": 256, "seq": 384, "padded": False},
        # the memory-bound front of the same model at the offline batch
        {"name": "bert_embed_b256_s384", "kind": "embed", "batch": 256, "seq": 384},
        # a whole BERT-base call at a serving batch
        {"name": "bert_base_b16_s384", "kind": "bert", "layers": 12, "batch": 16, "seq": 384, "padded": True},
        # ResNet-50: the stem at the offline batch, and the block of its second stage
        {"name": "stem_bf16_b256", "kind": "stem", "batch": 256, "size": 224},
        {"name": "bottleneck_bf16_b256", "kind": "bottleneck", "batch": 256, "c_in": 512, "c": 128, "stride": 1, "size": 28},
        # a whole ResNet-18 call in fp32-grade precision
        {"name": "resnet18_tf32x3_b32", "kind": "resnet18", "batch": 32, "size": 224},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["mlp", "encoder", "bert_layer", "bert_layer", "embed", "basic", "bottleneck", "bottleneck", "stem", "resnet18"])
    if kind == "mlp":
        return {"kind": kind, "batch": _log(rng, 1, 4096), "d_in": rng.choice([784, 768, 512, 1000]), "hidden": rng.choice([256, 512, 777, 1024]),
                "d_out": rng.choice([10, 100, 1000]), "dynamic": rng.random() < 0.5}
    if kind == "encoder":
        return {"kind": kind, "batch": _log(rng, 1, 16), "seq": _log(rng, 32, 512)}
    if kind == "bert_layer":
        return {"kind": kind, "batch": _log(rng, 1, 256), "seq": _log(rng, 24, 384), "padded": rng.random() < 0.7}
    if kind == "embed":
        return {"kind": kind, "batch": _log(rng, 1, 256), "seq": _log(rng, 24, 512)}
    if kind in ("basic", "bottleneck"):
        c, size = rng.choice([(64, 56), (128, 28), (256, 14), (512, 7)])
        down = rng.random() < 0.3
        wide = c if kind == "basic" else 4 * c
        c_in = wide // 2 if down and c > 64 else wide if not down else 64
        stride = 2 if down and c > 64 else 1
        return {"kind": kind, "batch": _log(rng, 1, 32 if kind == "basic" else 256), "c_in": c_in, "c": c, "stride": stride, "size": size * stride + rng.choice([0, 0, 1])}
    if kind == "stem":
        return {"kind": kind, "batch": _log(rng, 1, 256), "size": rng.choice([224, 224, 192, 161])}
    return {"kind": kind, "batch": _log(rng, 1, 32), "size": rng.choice([224, 192])}


def _dtype(case):
    return DTYPE["f32" if case["kind"] in ("mlp", "encoder", "basic", "resnet18") else "bf16"]


def _precision(case):
    return {"encoder": "tf32", "basic": "tf32x3", "resnet18": "tf32x3"}.get(case["kind"], "auto")


def _model(case, seed, dtype):
    """The module with weights drawn from the seed, at the scales trained networks have."""
    kind = case["kind"]
    with torch.device(DEVICE):
        if kind == "mlp":
            m = Mlp(case["d_in"], case["hidden"], case["d_out"])
        elif kind == "encoder":
            m = PreNormLayer(HEADS, D_FF)
        elif kind == "bert_layer":
            m = BertLayer(HEADS, D_FF)
        elif kind == "embed":
            m = Embed(VOCAB, MAX_POS, HEADS * HEAD)
        elif kind == "bert":
            m = Bert(case["layers"], VOCAB, MAX_POS, HEADS, D_FF)
        elif kind == "basic":
            m = Basic(case["c_in"], case["c"], case["stride"])
        elif kind == "bottleneck":
            m = Bottleneck(case["c_in"], case["c"], case["stride"])
        elif kind == "stem":
            m = Stem()
        else:
            m = ResNet18(1000)
    g = torch.Generator(DEVICE).manual_seed(seed)
    bert = kind in ("bert_layer", "embed", "bert")

    def normal(t, mean, std):
        t.copy_(torch.randn(t.shape, generator=g, device=t.device) * std + mean)

    with torch.no_grad():
        for mod in m.modules():
            if isinstance(mod, nn.Linear):
                normal(mod.weight, 0.0, 0.02 if bert else mod.in_features ** -0.5)
                normal(mod.bias, 0.0, 0.02)
            elif isinstance(mod, nn.Embedding):
                normal(mod.weight, 0.0, 0.02)
            elif isinstance(mod, nn.LayerNorm):
                normal(mod.weight, 1.0, 0.1)
                normal(mod.bias, 0.0, 0.1)
            elif isinstance(mod, nn.Conv2d):
                normal(mod.weight, 0.0, (2.0 / (mod.weight.shape[1] * mod.weight.shape[2] * mod.weight.shape[3])) ** 0.5)
            elif isinstance(mod, nn.BatchNorm2d):
                normal(mod.weight, 1.0, 0.1)
                normal(mod.bias, 0.0, 0.1)
                normal(mod.running_mean, 0.0, 0.1)
                mod.running_var.copy_(0.5 + torch.rand(mod.running_var.shape, generator=g, device=DEVICE))
    return m.to(dtype).eval()


def _inputs(case, seed, dtype):
    g = torch.Generator(DEVICE).manual_seed(seed + 7919)
    kind, b = case["kind"], case["batch"]

    def randn(*shape):
        return torch.randn(shape, generator=g, device=DEVICE).to(dtype)

    def mask(s):
        m = torch.ones(b, s, dtype=torch.int64, device=DEVICE)
        if case["padded"]:
            lengths = torch.randint((s + 1) // 2, s + 1, (b, 1), generator=g, device=DEVICE)
            m = (torch.arange(s, device=DEVICE)[None] < lengths).to(torch.int64)
        return m

    if kind == "mlp":
        return (randn(b, case["d_in"]),)
    if kind == "encoder":
        return (randn(b, case["seq"], HEADS * HEAD),)
    if kind == "bert_layer":
        return (randn(b, case["seq"], HEADS * HEAD), mask(case["seq"]))
    if kind in ("embed", "bert"):
        ids = torch.randint(0, VOCAB, (b, case["seq"]), generator=g, device=DEVICE, dtype=torch.int64)
        return (ids,) if kind == "embed" else (ids, mask(case["seq"]))
    if kind in ("basic", "bottleneck"):
        return (torch.relu(randn(b, case["c_in"], case["size"], case["size"])),)     # what the block before it hands over
    return (randn(b, 3, case["size"], case["size"]),)


def prepare(case, seed):
    dtype = _dtype(case)
    model, inputs = _model(case, seed, dtype), _inputs(case, seed, dtype)
    compiler = LLCompiler(precision=_precision(case))
    torch._dynamo.reset()
    fn = torch.compile(model, backend=compiler, dynamic=case.get("dynamic", False), fullgraph=True)
    with torch.no_grad():
        fn(*inputs)
    symbols = (case["batch"],) if case.get("dynamic", False) and case["batch"] > 1 else ()   # a batch of one is specialised
    return {"engine": compiler.compiled[0].engine, "args": symbols + inputs}


def run(state):
    return state["engine"].run(*state["args"])


def _numel(*shape):
    return math.prod(shape)


def work(case):
    """Every input, weight and output once at its storage width; the multiply-adds of the matmuls and convolutions."""
    kind, b = case["kind"], case["batch"]
    eb = 4 if _dtype(case) is torch.float32 else 2
    d = HEADS * HEAD

    def layer(tokens, s):
        weights = 4 * d * d + 2 * d * D_FF
        return 2.0 * tokens * weights + 4.0 * tokens * s * d, weights + 9 * d + D_FF

    if kind == "mlp":
        i, h, o = case["d_in"], case["hidden"], case["d_out"]
        return {"flops": 2.0 * b * (i * h + h * o), "bytes": eb * (b * (i + o) + i * h + h * o + h + o)}
    if kind in ("encoder", "bert_layer"):
        tokens = b * case["seq"]
        flops, weights = layer(tokens, case["seq"])
        return {"flops": flops, "bytes": eb * (2 * tokens * d + weights) + (8 * tokens if kind == "bert_layer" else 0)}
    if kind == "embed":
        tokens = b * case["seq"]
        return {"flops": 0.0, "bytes": 8 * tokens + eb * d * (min(tokens, VOCAB) + case["seq"] + tokens + 2)}
    if kind == "bert":
        tokens = b * case["seq"]
        flops, weights = layer(tokens, case["seq"])
        n = case["layers"]
        return {"flops": n * flops, "bytes": 16 * tokens + eb * (d * (min(tokens, VOCAB) + case["seq"] + tokens + 2) + n * weights)}

    def conv_out(size, stride):
        return (size - 1) // stride + 1

    def block(c_in, c, stride, size, wide):
        o = conv_out(size, stride)
        if wide == 1:
            w = [(c_in * c * 9, o), (c * c * 9, o)]
        else:
            w = [(c_in * c, size), (c * c * 9, o), (c * 4 * c, o)]
        if stride != 1 or c_in != wide * c:
            w.append((c_in * wide * c, o))
        return sum(2.0 * b * n * s * s for n, s in w), sum(n for n, _ in w), o

    if kind in ("basic", "bottleneck"):
        wide = 1 if kind == "basic" else 4
        flops, weights, o = block(case["c_in"], case["c"], case["stride"], case["size"], wide)
        return {"flops": flops, "bytes": eb * (weights + b * (case["c_in"] * case["size"] ** 2 + wide * case["c"] * o * o))}
    o = conv_out(case["size"], 2)
    stem_flops, p = 2.0 * b * 64 * 147 * o * o, conv_out(o, 2)
    if kind == "stem":
        return {"flops": stem_flops, "bytes": eb * (b * 3 * case["size"] ** 2 + 64 * 147 + b * 64 * p * p)}
    flops, weights, c_in, size = stem_flops, 64 * 147, 64, p
    for c, stride in ((64, 1), (128, 2), (256, 2), (512, 2)):
        for ci, st in ((c_in, stride), (c, 1)):
            f, w, size = block(ci, c, st, size, 1)
            flops, weights = flops + f, weights + w
        c_in = c
    return {"flops": flops + 2.0 * b * 512 * 1000, "bytes": eb * (b * 3 * case["size"] ** 2 + weights + 512 * 1000 + b * 1000)}


def tolerance(case):
    """About four times the error measured against exact(): fp32 sums 5e-7, tf32x3 3e-6 per block and 4.5e-5 through the
    whole ResNet-18, TF32 matmuls 1.1e-3, bf16 storage 1.7e-3 to 3.4e-3 per block and 1.1e-2 through twelve layers."""
    return {"rel": {
        "mlp": 4e-6,
        "encoder": 4e-3,
        "bert_layer": 1.4e-2,
        "embed": 1e-2,
        "bert": 4e-2,
        "basic": 1e-5,
        "bottleneck": 1e-2,
        "stem": 7e-3,
        "resnet18": 1.8e-4,
    }[case["kind"]]}


def exact(case, seed):
    """The same module in 64-bit PyTorch eager on the same weights and inputs, a slice of the batch at a time."""
    dtype = _dtype(case)
    model, inputs = _model(case, seed, dtype).double(), _inputs(case, seed, dtype)
    inputs = tuple(t.double() if t.is_floating_point() else t for t in inputs)
    with torch.no_grad():
        return [torch.cat([model(*(t[i:i + 32] for t in inputs)) for i in range(0, case["batch"], 32)])]
