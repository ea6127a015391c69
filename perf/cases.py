"""The work this framework is used for, as cases that can be timed one by one.

A case is a dict of plain values. `prepare` builds what a program has in hand before the call (inputs on the GPU, and the
model, optimizer or quantised layer it keeps), `run` is one pass through the public entry points, `work` the bytes and
operations the pass cannot do without, `tolerance` how far another correct implementation at the same precision may be.

The kinds follow the benchmark configurations of this repository (MLP, looped-transformer LM, fine-grained MoE, Mamba LM,
attention sweep) and its inference entry points (LM logits, quantised linear layers, `blas.sgemm`).
"""
from __future__ import annotations

import torch

from rust_neural_network_b200 import blas
from rust_neural_network_b200 import loss as losses
from rust_neural_network_b200 import nn
from rust_neural_network_b200.config import PRESETS, build_model
from rust_neural_network_b200.int8 import Int8Linear
from rust_neural_network_b200.models.moe import FineGrainedMoE
from rust_neural_network_b200.ops import functional as F
from rust_neural_network_b200.ops.linear_attention import linear_attention
from rust_neural_network_b200.ops.mx import MxLinear
from rust_neural_network_b200.optim import Adam
from rust_neural_network_b200.train import Trainer

DEV = "cuda"
VOCAB_MAMBA = 8192                # two Mamba layers with a vocabulary in proportion, so that the head does not hide the scan
LM = PRESETS["looped_lm"]


def listed():
    return [
        # the smallest training step: the 784-256-128-10 classifier, batch 32, fp32, one CUDA-graph replay per step
        dict(name="mlp_step", kind="mlp", dims="784-256-128-10", batch=32),
        # the BLAS entry point at the size the original project quotes
        dict(name="sgemm_512", kind="sgemm", m=512, n=512, k=512, ta=False, tb=False, beta=0.0),
        # scoring one prompt of odd length with the LM: forward only, logits out, one call after another from Python
        dict(name="lm_logits_1x333", kind="lm_forward", batch=1, seq=333),
        # the LM training step at the batch one of eight data-parallel GPUs has
        dict(name="lm_step_8x1024", kind="lm_step", batch=8, seq=1024),
        # the headline: the whole global batch on one GPU
        dict(name="lm_step_64x1024", kind="lm_step", batch=64, seq=1024),
        # one mixture-of-experts layer of the MoE LM, forward and backward, 8192 tokens
        dict(name="moe_layer_8192", kind="moe", tokens=8192, d=1024, hidden=512),
        # Mamba LM training step at the configuration's width and sequence length, two layers
        dict(name="mamba_step_2x4096", kind="mamba", batch=2, seq=4096, d=2048),
        # attention sweep, softmax attention, forward and backward, causal, the larger head size
        dict(name="flash_4096_hd128", kind="flash", batch=4, heads=16, seq=4096, hd=128, causal=True),
        # bidirectional attention of an encoder on a ragged batch length
        dict(name="flash_577_hd64", kind="flash", batch=16, heads=8, seq=577, hd=64, causal=False),
        # attention sweep, causal linear attention, a long sequence
        dict(name="linear_16384_hd64", kind="linear", batch=8, heads=16, seq=16384, hd=64, map="elu"),
        # the same on one short sequence, the other feature map and head size
        dict(name="linear_1000_hd128", kind="linear", batch=1, heads=16, seq=1000, hd=128, map="relu2"),
        # a quantised layer with a handful of tokens: the decode side of inference
        dict(name="int8_linear_16", kind="quant", fmt="int8", rows=16, inp=4096, out=4096),
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["mlp", "sgemm", "lm_forward", "lm_step", "moe", "mamba", "flash", "flash", "linear", "linear", "quant"])
    if kind == "mlp":
        dims = rng.choice(["784-256-128-10", "16-32-32-4", "64-128-128-10", "128-256-256-10", "256-512-512-256"])
        return dict(kind=kind, dims=dims, batch=_log(rng, 8, 256))
    if kind == "sgemm":
        return dict(kind=kind, m=_log(rng, 64, 4096), n=_log(rng, 64, 4096), k=_log(rng, 64, 4096), ta=rng.random() < 0.3, tb=rng.random() < 0.5,
                    beta=rng.choice([0.0, 0.0, 1.0]))
    if kind == "lm_forward":
        return dict(kind=kind, batch=_log(rng, 1, 8), seq=_log(rng, 16, 1024))
    if kind == "lm_step":
        seq = rng.choice([128, 256, 512, 1024, _log(rng, 128, 1024)])
        return dict(kind=kind, batch=_log(rng, 1, min(64, 32768 // seq)), seq=seq)
    if kind == "moe":
        d, hidden = rng.choice([(1024, 512), (1024, 512), (512, 256)])
        return dict(kind=kind, tokens=_log(rng, 256, 16384), d=d, hidden=hidden)
    if kind == "mamba":
        seq = _log(rng, 256, 8192)
        return dict(kind=kind, batch=_log(rng, 1, max(1, min(8, 8192 // seq))), seq=seq, d=rng.choice([1024, 2048]))
    if kind == "flash":
        heads, hd, seq = rng.choice([8, 16]), rng.choice([64, 128]), _log(rng, 128, 16384)
        most = max(1, min(32, int(8 * 2.0 ** 29 / (heads * hd * float(seq) * max(seq, 1024)))))
        return dict(kind=kind, batch=_log(rng, 1, most), heads=heads, seq=seq, hd=hd, causal=rng.random() < 0.7)
    if kind == "linear":
        heads, hd, seq = rng.choice([8, 16]), rng.choice([64, 128]), _log(rng, 256, 65536)
        most = max(1, min(32, 2 ** 26 // (heads * hd * seq)))
        return dict(kind=kind, batch=_log(rng, 1, most), heads=heads, seq=seq, hd=hd, map=rng.choice(["elu", "relu2"]))
    return dict(kind=kind, fmt=rng.choice(["int8", "int8", "mxfp8"]), rows=_log(rng, 1, 4096), inp=rng.choice([1024, 2048, 4096]),
                out=rng.choice([1024, 2048, 4096]))


# ----------------------------------------------------------------------------- what a program has before the call
def _gen(seed):
    torch.manual_seed(seed)                                        # weights (drawn on the host by the layers' initialisers)
    return torch.Generator(device=DEV).manual_seed(seed)


def _ids(g, vocab, *shape):
    return torch.randint(0, vocab, shape, generator=g, device=DEV)


def _trainer(model, loss_fn=None, lr=3e-4):
    return Trainer(model, Adam(model.parameters(), lr=lr), loss_fn, use_cuda_graph=True)


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    if kind == "mlp":
        dims = [int(v) for v in case["dims"].split("-")]
        model = nn.Sequential()
        for i in range(len(dims) - 1):
            model.add(nn.Linear(dims[i], dims[i + 1], init=nn.kaiming_uniform))
            if i + 2 < len(dims):
                model.add(nn.ReLU())
        model.to_device(torch.device(DEV), torch.float32)
        x = randn(case["batch"], dims[0])
        y = torch.nn.functional.one_hot(_ids(g, dims[-1], case["batch"]), dims[-1]).float()
        s = dict(trainer=_trainer(model, losses.CrossEntropyLoss(), 1e-3), x=x, y=y)
        s["trainer"].capture(x, y)
        return s
    if kind == "sgemm":
        return dict(a=randn(case["m"] * case["k"]), b=randn(case["k"] * case["n"]), c=randn(case["m"] * case["n"]), case=case)
    if kind == "lm_forward":
        model, _ = build_model("looped_lm", DEV)
        return dict(model=model.eval(), ids=_ids(g, LM.vocab, case["batch"], case["seq"]), logits=True)
    if kind in ("lm_step", "mamba"):
        if kind == "lm_step":
            model, cfg = build_model("looped_lm", DEV)
        else:
            model, cfg = build_model("mamba_lm", DEV, layers=2, vocab=VOCAB_MAMBA, d_model=case["d"], dt_rank=case["d"] // 16)
        x, y = (_ids(g, cfg.vocab, case["batch"], case["seq"]) for _ in range(2))
        s = dict(trainer=_trainer(model), x=x, y=y)
        s["trainer"].capture(x, y)
        return s
    if kind == "moe":
        layer = FineGrainedMoE(case["d"], case["hidden"], case["hidden"], 64, top_k=6, num_shared=2, act="silu", init=nn.normal_init(0.02))
        layer.to_device(torch.device(DEV), torch.bfloat16)
        x = randn(case["tokens"], case["d"]).bfloat16().requires_grad_(True)
        return dict(layer=layer, opt=Adam(layer.parameters(), lr=1e-3), x=x, dy=randn(case["tokens"], case["d"]).bfloat16())
    if kind in ("flash", "linear"):
        shape = (case["batch"], case["seq"], case["heads"], case["hd"])
        q, k, v = (randn(*shape).bfloat16().requires_grad_(True) for _ in range(3))
        return dict(q=q, k=k, v=v, do=randn(*shape).bfloat16(), causal=case.get("causal", True), map=case.get("map"), scale=case["hd"] ** -0.5)
    lin = nn.Linear(case["inp"], case["out"])
    lin.to_device(torch.device(DEV), torch.bfloat16)
    x = randn(case["rows"], case["inp"]).bfloat16()
    layer = Int8Linear.from_linear(lin) if case["fmt"] == "int8" else MxLinear(lin.weight.detach(), lin.bias, "mxfp8")
    return dict(quant=layer, x=x)


# ----------------------------------------------------------------------------- one pass
def run(s):
    if "trainer" in s:                                             # a training step: loss, gradients, updated weights
        t = s["trainer"]
        loss = t.train_step(s["x"], s["y"])
        return loss, t.optimizer.flat.grad, t.optimizer.flat.master
    if "a" in s:
        c = s["case"]
        m, n, k = c["m"], c["n"], c["k"]
        tr = lambda f: blas.Transpose.Trans if f else blas.Transpose.NoTrans
        # with beta = 1 a pass adds to what the last one left, as repeated updates of one matrix do
        return blas.sgemm(tr(c["ta"]), tr(c["tb"]), m, n, k, 1.0, s["a"], m if c["ta"] else k, s["b"], k if c["tb"] else n, c["beta"], s["c"], n)
    if "logits" in s:
        with torch.no_grad():
            return s["model"](s["ids"])
    if "layer" in s:                                               # a layer's share of a step: output, input gradient, weight gradients
        s["opt"].zero_grad()
        s["x"].grad = None
        y = s["layer"](s["x"])
        torch.autograd.backward([y, s["layer"].last_aux_loss], [s["dy"], None])
        return y, s["x"].grad, s["opt"].flat.grad
    if "quant" in s:
        return s["quant"](s["x"])
    q, k, v = s["q"], s["k"], s["v"]
    if s["map"] is None:
        o = F.flash_attention(q, k, v, s["scale"], s["causal"])
    else:
        o = linear_attention(q, k, v, scale=s["scale"], causal=True, kind=s["map"])
    return (o.detach(),) + torch.autograd.grad(o, (q, k, v), s["do"])


# ----------------------------------------------------------------------------- what the pass cannot do without
def _params(kind, case):
    if kind == "mlp":
        d = [int(v) for v in case["dims"].split("-")]
        return sum(a * b + b for a, b in zip(d, d[1:]))
    if kind in ("lm_step", "lm_forward"):
        d, block = LM.d_model, 4 * LM.d_model ** 2 + 2 * LM.d_model * LM.ff_dim
        return 2 * LM.vocab * d + LM.seq_len * d + LM.layers_per_block * block + 2 * d * d
    d, di, r, n = case["d"], 2 * case["d"], case["d"] // 16, 16
    return 2 * VOCAB_MAMBA * d + 2 * (3 * d * di + di * (r + 2 * n) + r * di)


def work(case):
    kind = case["kind"]
    step_bytes = lambda p: p * 34.0     # master, m, v read and written, gradient written and read, bf16 copy written
    if kind == "mlp":
        p = _params(kind, case)
        return dict(bytes=step_bytes(p), flops=6.0 * p * case["batch"])
    if kind == "sgemm":
        m, n, k = case["m"], case["n"], case["k"]
        return dict(bytes=4.0 * (m * k + k * n + m * n * (2 if case["beta"] else 1)), flops=2.0 * m * n * k)
    if kind in ("lm_forward", "lm_step"):
        B, S, d = case["batch"], case["seq"], LM.d_model
        apps = LM.layers_per_block * LM.loops
        per_token = 2.0 * (apps * (4 * d * d + 2 * d * LM.ff_dim) + d * LM.vocab) + apps * 2.0 * S * d
        if kind == "lm_forward":
            return dict(bytes=2.0 * _params(kind, case) + 2.0 * B * S * LM.vocab, flops=per_token * B * S)
        return dict(bytes=step_bytes(_params(kind, case)) + 16.0 * B * S, flops=3.0 * per_token * B * S)
    if kind == "moe":
        T, d, h = case["tokens"], case["d"], case["hidden"]
        w = 66 * 2 * d * h
        return dict(bytes=w * 6.0 + T * d * 2.0 * 4, flops=6.0 * T * (8 * 2 * d * h + 64 * d))
    if kind == "mamba":
        T, p = case["batch"] * case["seq"], _params(kind, case)
        used = p - VOCAB_MAMBA * case["d"]
        return dict(bytes=step_bytes(p) + 16.0 * T, flops=6.0 * used * T + 2 * 16 * 2 * case["d"] * T * 24.0)
    if kind in ("flash", "linear"):
        n = float(case["batch"] * case["heads"] * case["seq"] * case["hd"])
        byts = n * 2 * 8                                            # q, k, v, dout read; o, dq, dk, dv written
        if kind == "flash":
            return dict(bytes=byts, flops=4.0 * n * case["seq"] * 3.5 * (0.5 if case["causal"] else 1.0))
        return dict(bytes=byts, flops=n * case["hd"] * 4.0 * 3.5)
    m, n, k = case["rows"], case["out"], case["inp"]
    return dict(bytes=n * k * 1.0 + m * k * 2.0 + m * n * (4.0 if case["fmt"] == "int8" else 2.0), flops=2.0 * m * n * k)


def tolerance(case):
    return dict(TOLERANCE[case["kind"] if case["kind"] != "quant" else case["fmt"]])


# Measured on one pass each, as 2-norm of the difference over 2-norm of the result, and about four times that stated (3e-2 at
# most): MLP gradients with TF32 products against fp64 8e-3 (a few ReLUs switch); sgemm (TF32) against fp64 8e-4; LM gradients
# with bf16 against fp32 activations 2.1e-2 and logits 1.0e-2; Mamba LM 1.0e-2 and 0.9e-2; flash attention against fp64
# 2.5e-3; linear attention against fp32 on bf16 features 3.1e-3 (single elements of a ReLU^2 gradient up to 0.8 of the root mean
# square); the MoE layer in bf16 against fp32 2.0e-2 (tokens whose sixth and seventh expert tie); int8 6e-8; MXFP8 1.7e-3.
TOLERANCE = {
    "mlp": dict(rel=2e-2, max=0.99), "sgemm": dict(rel=3e-3), "lm_forward": dict(rel=3e-2, max=0.4), "lm_step": dict(rel=3e-2, max=0.99),
    "moe": dict(rel=3e-2, max=0.99), "mamba": dict(rel=3e-2, max=0.99), "flash": dict(rel=1e-2, max=0.2), "linear": dict(rel=1.2e-2, max=0.99),
    "int8": dict(rel=1e-6, max=1e-5), "mxfp8": dict(rel=7e-3),
}
