"""MoE kernels: router forward/backward against torch softmax/top-k autograd, routed experts
(dispatch -> batched expert GEMMs -> combine) against the dense per-token fp32 loop, incl. gradients;
linear attention on the GPU against the O(S^2) reference."""
import pytest
import torch

from rust_neural_network_b200.models import moe as M
from rust_neural_network_b200.ops.linear_attention import linear_attention, linear_attention_ref

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return float((a - b).norm() / (b.norm() + 1e-9))


@pytest.mark.parametrize("T,E,k,renorm", [(100, 8, 2, True), (257, 64, 6, True), (64, 40, 3, False), (33, 200, 8, True)])
def test_router_forward_backward(T, E, k, renorm):
    torch.manual_seed(0)
    logits = (torch.randn(T, E, device="cuda") * 2).requires_grad_(True)
    idx, w, counts, aux = M.RouterFn.apply(logits, k, renorm, 0.01)
    lr = logits.detach().clone().requires_grad_(True)
    p = torch.softmax(lr, -1)
    wr, ir = torch.topk(p, k, dim=-1)
    if renorm:
        wr = wr / wr.sum(-1, keepdim=True)
    assert torch.equal(idx.long(), ir)
    assert torch.allclose(w, wr, atol=1e-5)
    assert torch.equal(counts.long(), torch.bincount(ir.reshape(-1), minlength=E))
    f = counts.float() / (T * k)
    auxr = E * (f * p.mean(0)).sum()
    assert torch.allclose(aux, auxr, atol=1e-5)
    g = torch.randn_like(w)
    ((w * g).sum() + 3.0 * aux).backward()
    ((wr * g).sum() + 3.0 * auxr).backward()
    assert rel_err(logits.grad, lr.grad) < 1e-3


@pytest.mark.parametrize("act", ["relu", "silu"])
def test_routed_experts_match_dense_loop(act):
    torch.manual_seed(1)
    T, d, hid, E, k = 300, 64, 128, 8, 2
    dev = "cuda"
    x = (torch.randn(T, d, device=dev) * 0.5).bfloat16().requires_grad_(True)
    W1 = torch.nn.Parameter(torch.randn(E, hid, d, device=dev) * 0.1); b1 = torch.nn.Parameter(torch.randn(E, hid, device=dev) * 0.1)
    W2 = torch.nn.Parameter(torch.randn(E, d, hid, device=dev) * 0.1); b2 = torch.nn.Parameter(torch.randn(E, d, device=dev) * 0.1)
    logits = torch.randn(T, E, device=dev)
    idx, w, _, _ = M.RouterFn.apply(logits, k, True, 0.0)
    w = w.detach().requires_grad_(True)
    out = M.MoEExpertsFn.apply(x, idx, w, W1, b1, W2, b2, act, 384, None)       # capacity large enough: nothing dropped
    xr = x.detach().float().requires_grad_(True); wr = w.detach().clone().requires_grad_(True)
    ps = [t.detach().clone().requires_grad_(True) for t in (W1, b1, W2, b2)]
    ref = M._experts_dense_autograd(xr, idx, wr, *ps, act)
    assert rel_err(out, ref) < 2e-2
    g = torch.randn_like(ref)
    (out.float() * g).sum().backward(); (ref * g).sum().backward()
    assert rel_err(x.grad, xr.grad) < 3e-2
    assert rel_err(w.grad, wr.grad) < 3e-2
    for a, b in zip((W1, b1, W2, b2), ps):
        assert rel_err(a.grad, b.grad) < 3e-2


def test_one_kernel_layer_equals_the_separate_kernels(monkeypatch):
    """The forward of the routed experts as one launch (dispatch, barriers, both grouped GEMMs, combine inside one
    persistent kernel) against the same layer as separate launches: the outputs agree to the last bit (every token's row
    goes through the same arithmetic whatever slot it lands in), the gradients up to the summation order over rows."""
    torch.manual_seed(3)
    T, d, hid, E, k = 700, 256, 512, 8, 2
    x = (torch.randn(T, d, device="cuda") * 0.5).bfloat16()
    logits = torch.randn(T, E, device="cuda")
    wv, idx = torch.topk(torch.softmax(logits, -1), k, dim=-1)
    idx = idx.int().contiguous()
    g = torch.randn(T, d, device="cuda").bfloat16()
    res = []
    for fused in (True, False):
        monkeypatch.setattr(M, "_FUSED_LAYER", fused)
        torch.manual_seed(5)
        W1 = (torch.randn(E, hid, d, device="cuda") * 0.05).bfloat16().requires_grad_(True)
        b1 = (torch.randn(E, hid, device="cuda") * 0.1).requires_grad_(True)
        W2 = (torch.randn(E, d, hid, device="cuda") * 0.05).bfloat16().requires_grad_(True)
        b2 = (torch.randn(E, d, device="cuda") * 0.1).requires_grad_(True)
        xi = x.clone().requires_grad_(True)
        wi = wv.clone().requires_grad_(True)
        for _ in range(2):                                   # twice: the second call finds the buffers as the first left them
            xi.grad = wi.grad = W1.grad = b1.grad = W2.grad = b2.grad = None
            out = M.MoEExpertsFn.apply(xi, idx, wi, W1, b1, W2, b2, "silu", 256, None)
            out.backward(g)
        res.append([t.detach().float().clone() for t in (out, xi.grad, wi.grad, W1.grad, b1.grad, W2.grad, b2.grad)])
    assert torch.equal(res[0][0], res[1][0])
    assert torch.equal(res[0][1], res[1][1])
    for a, b in zip(res[0][2:], res[1][2:]):
        assert rel_err(a, b) < 2e-3
    ref = M.moe_experts_ref(x, idx, wv, W1.detach(), b1.detach(), W2.detach(), b2.detach(), "silu")
    assert rel_err(res[0][0], ref) < 2e-2


@pytest.mark.parametrize("T,past", [(16384, True), (16383, False)])
def test_one_rank_alone_takes_the_separate_kernels_for_many_tokens(monkeypatch, T, past):
    """On both sides of the rule (16384 x 8 x 256 routed elements): output bit for bit, gradients up to the order over rows."""
    torch.manual_seed(4)
    d, hid, E, k = 256, 64, 16, 8
    assert (T * k * d >= M._ALONE_FROM) == past
    x = (torch.randn(T, d, device="cuda") * 0.5).bfloat16()
    idx = torch.topk(torch.randn(T, E, device="cuda"), k)[1].int()
    w = torch.rand(T, k, device="cuda")
    ws = [torch.nn.Parameter(torch.randn(*s, device="cuda") * 0.1) for s in ((E, hid, d), (E, hid), (E, d, hid), (E, d))]
    g = torch.randn(T, d, device="cuda").bfloat16()
    single, calls = M._fused_layer_forward, []
    monkeypatch.setattr(M, "_fused_layer_forward", lambda *a: calls.append(1) or single(*a))
    res = []
    for limit in (M._ALONE_FROM, 1 << 62):
        monkeypatch.setattr(M, "_ALONE_FROM", limit)
        xi, wi = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
        for p in ws:
            p.grad = None
        out = M.MoEExpertsFn.apply(xi, idx, wi, *ws, "silu", T * k // E + 1024 & ~127, None)
        out.backward(g)
        res.append([out.detach(), xi.grad, wi.grad] + [p.grad.clone() for p in ws])
    assert len(calls) == (1 if past else 2)
    assert torch.equal(res[0][0], res[1][0])
    for a, b in zip(res[0][1:], res[1][1:]):
        assert rel_err(a, b) < 1e-5


def test_capacity_drops_are_consistent():
    torch.manual_seed(2)
    T, d, hid, E, k = 256, 64, 64, 4, 1
    dev = "cuda"
    x = torch.randn(T, d, device=dev).bfloat16()
    W1 = torch.randn(E, hid, d, device=dev) * 0.1; b1 = torch.zeros(E, hid, device=dev)
    W2 = torch.randn(E, d, hid, device=dev) * 0.1; b2 = torch.zeros(E, d, device=dev)
    idx = torch.zeros(T, 1, dtype=torch.int32, device=dev)                  # everyone wants expert 0
    w = torch.ones(T, 1, device=dev)
    out = M.MoEExpertsFn.apply(x, idx, w, W1, b1, W2, b2, "relu", 128, None)
    kept = int((out.float().abs().sum(-1) > 0).sum())
    assert kept == 128                                                       # exactly `capacity` tokens were served


def test_moe_module_trains_bf16():
    torch.manual_seed(3)
    from rust_neural_network_b200.optim import Adam
    lm = M.MoETransformerLM(256, 128, 2, 2, 8, 2, 1, 128, 128).to_device("cuda", torch.bfloat16)
    opt = Adam(lm.parameters(), lr=2e-3)
    ids = torch.randint(0, 256, (2, 128), device="cuda"); lab = torch.randint(0, 256, (2, 128), device="cuda")
    losses = []
    for _ in range(20):
        opt.zero_grad(); l = lm.loss(ids, lab); l.backward(); opt.step(); losses.append(float(l))
    assert losses[-1] < losses[0] * 0.9


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("kind", ["elu", "relu2"])
def test_linear_attention_gpu(causal, kind):
    torch.manual_seed(4)
    q, k, v = ((torch.randn(2, 300, 2, 64, device="cuda") * 0.5).bfloat16().requires_grad_(True) for _ in range(3))
    o = linear_attention(q, k, v, 0.5, 1e-6, causal, kind)
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    r = linear_attention_ref(qr, kr, vr, 0.5, 1e-6, causal, kind)
    assert rel_err(o, r) < 8e-3                         # measured 1.6e-3 .. 3.4e-3
    g = torch.randn_like(r)
    (o.float() * g).sum().backward(); (r * g).sum().backward()
    # measured: dk, dv 3.4e-3 .. 4.5e-3 everywhere; dq 4e-3 .. 8.5e-3, and 2.0e-2 for the non-causal ELU + 1 form
    # (bf16 features near 1 in a difference of nearly equal sums)
    for name, a, b in (("dq", q, qr), ("dk", k, kr), ("dv", v, vr)):
        tol = 3e-2 if (name == "dq" and kind == "elu") else 1e-2
        assert rel_err(a.grad, b.grad) < tol, (name, rel_err(a.grad, b.grad))


@pytest.mark.parametrize("T,E,k,cap", [(700, 8, 2, 256), (64, 16, 1, 128), (3, 4, 2, 128), (900, 4, 2, 130)])
@pytest.mark.parametrize("fused", [True, False])
def test_expert_gradients_in_an_optimizers_buffer(monkeypatch, T, E, k, cap, fused):
    """Weights whose gradients live in an optimizer's buffer: the products add into it (twice here); experts without tokens, with whole and broken tiles,
    and past their capacity."""
    monkeypatch.setattr(M, "_FUSED_LAYER", fused)
    torch.manual_seed(T)
    d, hid = 64, 128
    x = (torch.randn(T, d, device="cuda") * 0.5).bfloat16().requires_grad_(True)
    idx = torch.topk(torch.randn(T, E, device="cuda") + torch.linspace(0, 3, E, device="cuda"), k)[1].int().contiguous()
    w = torch.rand(T, k, device="cuda")
    g = torch.randn(T, d, device="cuda").bfloat16()
    ws = [torch.nn.Parameter(torch.randn(*s, device="cuda") * 0.1) for s in ((E, hid, d), (E, hid), (E, d, hid), (E, d))]
    M.MoEExpertsFn.apply(x, idx, w, *ws, "silu", cap, None).backward(g)
    plain = [p.grad.clone() for p in ws]
    for p in ws:
        p._fused_grad, p.grad = True, torch.ones_like(p)
    for _ in range(2):
        M.MoEExpertsFn.apply(x, idx, w, *ws, "silu", cap, None).backward(g)
    full = bool((torch.bincount(idx.flatten().long(), minlength=E) <= cap).all())
    for p, one in zip(ws, plain):
        if full:                                             # (which of an overfull expert's tokens are dropped depends on timing)
            assert rel_err(p.grad, 1 + 2 * one) < 1e-3
        assert torch.isfinite(p.grad).all()


@pytest.mark.parametrize("rows,cols,ld", [(128, 8, 8), (300, 264, 264), (257, 40, 48), (64, 100, 100)])
def test_batched_column_sums(rows, cols, ld):
    from rust_neural_network_b200 import _native as nv
    x = torch.randn(3, rows, ld, device="cuda").bfloat16()
    valid = torch.tensor([0, 1, rows], dtype=torch.int32, device="cuda")
    out = torch.ones(3, cols, device="cuda")
    nv.check(nv.cuda().b200_colsum_batched(x.data_ptr(), out.data_ptr(), 3, rows, cols, ld, rows * ld, 1, valid.data_ptr(), nv.stream_ptr()), "colsum")
    for b, n in enumerate([0, min(rows, 128), rows]):
        want = 1 + x[b, :n, :cols].double().sum(0)
        assert float((out[b].double() - want).abs().max()) < 1e-3
