"""The extension that prepares the short GPU calls: what it refuses, views and layouts it accepts, streams and threads."""
import threading

import pytest
import torch

from rust_neural_network_b200 import _native as nv
from rust_neural_network_b200.ops import gemm as G
from rust_neural_network_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_refused_products():
    a, b = torch.randn(32, 64, device=DEV), torch.randn(16, 64, device=DEV)
    with pytest.raises(TypeError, match="operands must be"):
        G.gemm(a, b.bfloat16())
    with pytest.raises(TypeError, match="operands must be"):
        G.gemm(a.half(), b.half())
    with pytest.raises(ValueError, match="K mismatch"):
        G.gemm(a, b[:, :32])
    with pytest.raises(ValueError, match="2-D or 3-D"):
        G.gemm(a[0], b)
    with pytest.raises(ValueError, match="batch mismatch"):
        G.gemm(a.expand(2, 32, 64), b.expand(3, 16, 64))
    with pytest.raises(ValueError, match="contiguous fp32"):
        G.gemm(a, b, accumulate_into=torch.zeros(32, 16, device=DEV).bfloat16())
    with pytest.raises(ValueError, match="`out`"):
        G.gemm(a, b, out=torch.zeros(32, 15, device=DEV))
    with pytest.raises(ValueError, match="go together"):
        G.gemm(a, b, out=torch.zeros(32, 16, device=DEV), splits=2)
    with pytest.raises(ValueError, match="split-K"):
        G.gemm(torch.randn(32, 2048, device=DEV), torch.randn(16, 2048, device=DEV), splits=2, act="relu")
    with pytest.raises(TypeError, match="bias"):
        G.gemm(a, b, bias=torch.zeros(16, device=DEV).half())
    with pytest.raises(ValueError, match="row_scale"):
        G.gemm(a, b, row_scale=torch.ones(3, device=DEV))
    with pytest.raises(ValueError, match="m_valid"):
        G.gemm(a, b, m_valid=torch.ones(2, dtype=torch.int32, device=DEV))
    with pytest.raises(TypeError, match="integer"):
        G.gemm(a, b, out_dtype=torch.int32)
    with pytest.raises(ValueError, match="K-major"):
        G.gemm(torch.zeros(64, 32, dtype=torch.int8, device=DEV), torch.zeros(16, 64, dtype=torch.int8, device=DEV), a_mn=True)
    with pytest.raises(TypeError, match="bf16"):
        K.flash_fwd(*(torch.randn(1, 8, 2, 64, device=DEV) for _ in range(3)), 0.125, True)


def test_views_and_counts():
    x = torch.randn(40, 96, device=DEV).bfloat16()
    w = torch.randn(3, 24, 96, device=DEV).bfloat16()
    n = nv.launch_count()
    got = G.gemm(x[:, 1:81], w[1][:, 1:81])                          # rows off 16 bytes: padded copies
    assert nv.launch_count() == n + 1
    want = x[:, 1:81].double() @ w[1][:, 1:81].double().t()
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8
    q = torch.randn(2, 70, 3, 2, 64, device=DEV).bfloat16()
    o, lse = K.flash_fwd(q[:, :, 0], q[:, :, 1], q[:, :, 2], 0.125, True)
    ref = K.attention_ref(q[:, :, 0], q[:, :, 1], q[:, :, 2], 0.125, True)
    assert float((o.float() - ref).norm() / ref.norm()) < 1e-2 and nv.launch_count() == n + 2
    nv.check_status()


def test_calls_on_other_streams_and_threads():
    a, b = torch.randn(64, 256, device=DEV).bfloat16(), torch.randn(128, 256, device=DEV).bfloat16()
    want = G.gemm(a, b)
    torch.cuda.synchronize()
    res = []

    def work():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            r = [G.gemm(a, b) for _ in range(20)]
        s.synchronize()
        res.extend(torch.equal(x, want) for x in r)

    ts = [threading.Thread(target=work) for _ in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert len(res) == 80 and all(res)


def test_block_calls_of_one_forward_pass_equal_single_blocks():
    """The trunk looks at its blocks once for all loops; a weight that changed between two passes is seen by the second."""
    from rust_neural_network_b200.models.looped_transformer import LoopedTransformer
    torch.manual_seed(1)
    m = LoopedTransformer(64, 128, 2, 256, 64, 3, causal=True, layers_per_block=2).to_device(torch.device(DEV), torch.bfloat16)
    h = torch.randn(2, 37, 128, device=DEV).bfloat16()

    def by_blocks():
        tc, x = m.time_conditioning(h.device, h.dtype), h
        for t in range(m.num_loops):
            cond = K.binary(x, tc[t], "add")
            x = K.binary(cond, m.block(cond), "add")
        return x

    with torch.no_grad():
        first = m.trunk(h)[0]
        assert torch.equal(first, by_blocks())
        m.block.blocks[1].ff1.weight.mul_(1.5)
        second = m.trunk(h)[0]
        assert torch.equal(second, by_blocks()) and not torch.equal(first, second)
    grad = m.trunk(h)[0].detach()
    assert float((grad.float() - second.float()).norm() / second.float().norm()) < 2e-2
