"""GPU model-level tests: the fused bf16 transformer block / LM against the same modules evaluated
with the fp32 PyTorch reference ops on CPU, learning smoke tests, CUDA-graph replay."""
import copy
import math

import pytest
import torch

from rust_neural_network_b200 import nn
from rust_neural_network_b200.loss import CrossEntropyLoss, MSELoss
from rust_neural_network_b200.models.lm import LoopedTransformerLM
from rust_neural_network_b200.models.looped_transformer import LoopedTransformer, Transformer, TransformerBlock
from rust_neural_network_b200.optim import SGD, Adam
from rust_neural_network_b200.train import SimpleDataLoader, Trainer

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return float((a - b).norm() / (b.norm() + 1e-12))


def grads_close(got, ref, rel=5e-2, floor=2e-2):
    """Per-parameter gradient check that tolerates parameters whose true gradient is ~0 (e.g. the key
    bias of softmax attention): error <= rel*|ref| + floor*(global rms of all reference grads)*sqrt(n)."""
    allref = torch.cat([r.float().reshape(-1).cpu() for r in ref])
    rms = float(allref.pow(2).mean().sqrt())
    bad = []
    for i, (g, r) in enumerate(zip(got, ref)):
        g, r = g.float().cpu(), r.float().cpu()
        err = float((g - r).norm())
        if err > rel * float(r.norm()) + floor * rms * (r.numel() ** 0.5):
            bad.append((i, tuple(r.shape), err, float(r.norm())))
    return bad


def _clone_to(module, device, dtype):
    m = copy.deepcopy(module)
    return m.to_device(device, dtype)


@pytest.mark.parametrize("B,S,d,heads,ff,causal", [(1, 1, 128, 2, 256, True), (1, 333, 128, 1, 264, True), (3, 7, 64, 1, 72, False),
                                                   (2, 130, 256, 4, 1024, False), (64, 257, 512, 8, 2048, True)])
def test_block_without_gradients_equals_the_differentiable_one(B, S, d, heads, ff, causal):
    """The one-call forward issues the kernels the differentiable function issues, on the same operands: equal bit for bit,
    before and after a weight and a bias change in place."""
    torch.manual_seed(1)
    blk = TransformerBlock(d, heads, ff, causal=causal, init=nn.normal_init(0.05)).to_device(torch.device("cuda"), torch.bfloat16)
    x = torch.randn(B, S, d, device="cuda").bfloat16()
    for _ in range(2):
        with torch.no_grad():
            y = blk(x)
            strided = blk(torch.stack([x, x], -1)[..., 0])                # not contiguous
        assert not y.requires_grad and torch.equal(y, blk(x).detach()) and torch.equal(y, strided)
        with torch.no_grad():
            blk.attn.k_proj.weight.mul_(1.5)
            blk.attn.v_proj.bias.add_(0.25)
            before = y
    assert not torch.equal(before, blk(x))


def _without_early_launches(fn):
    from rust_neural_network_b200 import _native as nv
    nv.set_pdl(False)
    try:
        r = fn()
        torch.cuda.synchronize()
        return r
    finally:
        nv.set_pdl(True)


def test_blocks_read_what_their_predecessors_wrote():
    """Blocks with biases of their own, back to back on reused workspaces and on alternating inputs, eager and as a graph:
    bit for bit what the same kernels give when each starts only after its predecessor has ended."""
    torch.manual_seed(2)
    blks = [TransformerBlock(512, 8, 1024, causal=True, init=nn.normal_init(0.05)).to_device(torch.device("cuda"), torch.bfloat16) for _ in range(4)]
    for b in blks:
        for lin in (b.attn.q_proj, b.attn.k_proj, b.attn.v_proj, b.attn.out_proj, b.ff1, b.ff2):
            lin.bias.data.normal_()
    xs = [torch.randn(2, 200, 512, device="cuda").bfloat16() for _ in range(2)]

    def forward(x):
        with torch.no_grad():
            for b in blks:
                x = b(x)
        return x

    ref = _without_early_launches(lambda: [forward(x) for x in xs])
    static = xs[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = forward(static)
    for i in range(50):
        assert torch.equal(forward(xs[i % 2]), ref[i % 2])
        static.copy_(xs[i % 2])
        graph.replay()
        assert torch.equal(y, ref[i % 2])


def test_block_without_gradients_refuses_heads_that_do_not_divide_the_width():
    blk = TransformerBlock(584, 8, 64, init=nn.normal_init(0.05)).to_device(torch.device("cuda"), torch.bfloat16)
    blk.attn.heads = 9                                                    # 584 // 9 = 64, a head size the kernels know
    x = torch.zeros(1, 4, 584, device="cuda").bfloat16()
    for grad in (True, False):
        with pytest.raises(RuntimeError), torch.set_grad_enabled(grad):
            blk(x)


def test_traced_block_runs_on_new_inputs():
    torch.manual_seed(6)
    blk = TransformerBlock(128, 2, 256, causal=True, init=nn.normal_init(0.05)).to_device(torch.device("cuda"), torch.bfloat16)
    x, x2 = (torch.randn(2, 40, 128, device="cuda").bfloat16() for _ in range(2))
    with pytest.raises(RuntimeError), torch.no_grad():                    # a trace holds no weights that want gradients
        torch.jit.trace(lambda t: blk(t) * 1.0, (x,), check_trace=False)
    for p in blk.parameters():
        p.requires_grad_(False)
    with torch.no_grad():
        traced = torch.jit.trace(lambda t: blk(t) * 1.0, (x,), check_trace=False)
        assert torch.equal(traced(x2), blk(x2))


def test_graph_keeps_its_weights_over_an_eager_forward():
    """A graph captured on shadows of the projections that are not neighbours replays the same result after a forward without
    gradients has run outside it and freed memory has been written over."""
    from rust_neural_network_b200.ops.functional import lp
    torch.manual_seed(5)
    blk = TransformerBlock(256, 4, 512, causal=True, init=nn.normal_init(0.05)).to_device(torch.device("cuda"), torch.bfloat16)
    for lin in (blk.attn.v_proj, blk.attn.q_proj, blk.attn.k_proj):
        lp(lin.weight)
    x = torch.randn(2, 64, 256, device="cuda").bfloat16()
    ref = blk(x).detach().clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = blk(x)
    with torch.no_grad():
        assert torch.equal(blk(x), ref)
    junk = [torch.full((256, 256), 9.0, device="cuda").bfloat16() for _ in range(16)]
    graph.replay()
    assert torch.equal(y, ref) and len(junk) == 16


def test_bias_free_mlp_step_reads_what_its_predecessors_wrote():
    """A captured fp32 step whose products, activation gradients and optimizer follow each other without a column sum between
    them: the weights after 100 replays carry the bits they have without early launches (contractions too short to be split)."""
    def train():
        torch.manual_seed(3)
        m = nn.Sequential()
        for i in range(3):
            m.add(nn.Linear(128, 128, bias=False))
            if i < 2:
                m.add(nn.ReLU())
        m.to_device(torch.device("cuda"), torch.float32)
        t = Trainer(m, Adam(m.parameters(), lr=1e-3), MSELoss(), use_cuda_graph=True)
        g = torch.Generator(device="cuda").manual_seed(4)
        data = [(torch.randn(32, 128, generator=g, device="cuda"), torch.randn(32, 128, generator=g, device="cuda")) for _ in range(4)]
        for i in range(100):
            t.train_step(*data[i % 4])
        return t.optimizer.flat.master.clone()

    assert torch.equal(train(), _without_early_launches(train))


@pytest.mark.parametrize("causal", [False, True])
def test_fused_block_matches_fp32_reference(causal):
    torch.manual_seed(0)
    blk = TransformerBlock(128, 2, 256, causal=causal, init=nn.normal_init(0.05))
    x = torch.randn(2, 128, 128) * 0.5
    ref_blk = copy.deepcopy(blk)
    xr = x.clone().requires_grad_(True)
    yr = ref_blk(xr)
    w = torch.randn_like(yr)
    (yr * w).sum().backward()

    g = _clone_to(blk, "cuda", torch.bfloat16)
    xg = x.cuda().bfloat16().requires_grad_(True)
    yg = g(xg)
    (yg.float() * w.cuda()).sum().backward()
    assert rel_err(yg, yr) < 2e-2
    assert rel_err(xg.grad, xr.grad) < 4e-2
    assert all(p.grad is not None for p in g.parameters())
    assert grads_close([p.grad for p in g.parameters()], [p.grad for p in ref_blk.parameters()]) == []


def test_lm_loss_matches_reference_and_learns():
    torch.manual_seed(1)
    kw = dict(vocab=512, d_model=128, heads=2, ff_dim=256, layers_per_block=2, loops=2, max_seq=128, causal=True)
    cpu = LoopedTransformerLM(**kw)
    gpu = _clone_to(cpu, "cuda", torch.bfloat16)
    ids = torch.randint(0, 512, (2, 128)); labels = torch.randint(0, 512, (2, 128))
    lc = cpu.loss(ids, labels); lg = gpu.loss(ids.cuda(), labels.cuda())
    assert abs(float(lc) - float(lg)) < 0.05
    lc.backward(); lg.backward()
    assert grads_close([p.grad for p in gpu.parameters()], [p.grad for p in cpu.parameters()], rel=0.12, floor=0.05) == []
    opt = Adam(gpu.parameters(), lr=2e-3)
    tr = Trainer(gpu, opt)
    first = float(tr.train_step(ids, labels))
    for _ in range(30):
        last = float(tr.train_step(ids, labels))
    assert last < first * 0.7


def test_cuda_graph_replay_matches_eager():
    torch.manual_seed(2)
    kw = dict(vocab=256, d_model=128, heads=2, ff_dim=256, layers_per_block=1, loops=2, max_seq=128, causal=True)
    a = LoopedTransformerLM(**kw)
    b = copy.deepcopy(a)
    a.to_device("cuda", torch.bfloat16); b.to_device("cuda", torch.bfloat16)
    ta = Trainer(a, Adam(a.parameters(), lr=1e-3), use_cuda_graph=False)
    tb = Trainer(b, Adam(b.parameters(), lr=1e-3), use_cuda_graph=True)
    data = [(torch.randint(0, 256, (2, 128)), torch.randint(0, 256, (2, 128))) for _ in range(4)]
    # capture warms up on a side stream and restores weights and optimizer state, so graph and eager agree step for step
    la = [float(ta.train_step(*d)) for d in data]
    lb = [float(tb.train_step(*d)) for d in data]
    assert all(abs(x - y) < 0.1 for x, y in zip(la, lb)), (la, lb)


def test_mlp_config1_fp32_matches_cpu_oracle():
    """MLP 784-256-128-10, CE, Adam lr 1e-3, batch 32, 100 steps: TF32 GPU path tracks the fp32 CPU oracle."""
    torch.manual_seed(3)
    def make():
        g = torch.Generator().manual_seed(7)
        return nn.Sequential(nn.Linear(784, 256, init=nn.kaiming_uniform, generator=g), nn.ReLU(),
                             nn.Linear(256, 128, init=nn.kaiming_uniform, generator=g), nn.ReLU(),
                             nn.Linear(128, 10, init=nn.kaiming_uniform, generator=g))
    cpu, gpu = make(), make().to_device("cuda")
    x = torch.randn(32, 784); y = torch.randint(0, 10, (32,))
    oc, og = Adam(cpu.parameters(), lr=1e-3), Adam(gpu.parameters(), lr=1e-3)
    lf = CrossEntropyLoss()
    lc, lg = [], []
    for _ in range(100):
        oc.zero_grad(); l = lf(cpu(x), y); l.backward(); oc.step(); lc.append(float(l))
        og.zero_grad(); l2 = lf(gpu(x.cuda()), y.cuda()); l2.backward(); og.step(); lg.append(float(l2))
    assert lc[-1] < lc[0] * 0.2
    assert max(abs(a - b) for a, b in zip(lc, lg)) < 2e-2


def test_xor_learns():
    torch.manual_seed(4)
    net = nn.Sequential(nn.Linear(2, 8), nn.Tanh(), nn.Linear(8, 1), nn.Sigmoid()).to_device("cuda")
    x = torch.tensor([[0., 0.], [0., 1.], [1., 0.], [1., 1.]]); y = torch.tensor([[0.], [1.], [1.], [0.]])
    tr = Trainer(net, Adam(net.parameters(), lr=0.05), MSELoss())
    loader = SimpleDataLoader(x, y, 4)
    for _ in range(400):
        loss = tr.train_epoch(loader)
    assert loss < 0.1


def test_transformer_and_looped_fp32_paths_run():
    torch.manual_seed(5)
    m = LoopedTransformer(16, 64, 1, 128, 8, 2).to_device("cuda")
    x = torch.randn(2, 16, 16, device="cuda")
    out, loops = m.forward_with_loops(x)
    assert out.shape == (2, 16, 8) and loops == 2
    out.sum().backward()
    t = Transformer(16, 128, 2, 128, 4, 2, causal=True).to_device("cuda", torch.bfloat16)
    y = t(torch.randn(2, 128, 16, device="cuda").bfloat16())
    assert y.shape == (2, 128, 4)
    y.float().sum().backward()
    assert all(p.grad is not None for p in t.parameters())
