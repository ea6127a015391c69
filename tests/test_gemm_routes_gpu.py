"""Products at the edges of the GEMM's tiles and routes: fp32 operands that are read transposed, narrow tiles, pairs of CTAs, sums divided
over a cluster. The oracle is the same product in fp64."""
import pytest
import torch

from rust_neural_network_b200 import _native as nv
from rust_neural_network_b200.ops import gemm as G

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(got, want, rel):
    nv.check_status()
    err = (got.double() - want).norm() / want.norm().clamp_min(1e-30)
    assert float(err) <= rel, float(err)


# TF32 keeps 10 mantissa bits of each operand: 2^-11 per factor, two factors, averaged over the sum: 2-norm below 2 * 2^-11
TF32 = 2.0 ** -10


@pytest.mark.parametrize("m,n,k", [(4, 4, 4), (32, 256, 784), (100, 52, 36), (128, 128, 32), (260, 132, 1000), (300, 1000, 64), (2048, 2044, 516)])
@pytest.mark.parametrize("a_mn,b_mn", [(True, False), (False, True), (True, True)])
def test_transposed_fp32_operands_equal_the_transposed_copy(m, n, k, a_mn, b_mn):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    a, b = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    A, B = a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b
    got = G.gemm(A, B, a_mn=a_mn, b_mn=b_mn, splits=1)
    _close(got, a.double() @ b.double().t(), TF32)
    assert torch.equal(got, G.gemm(a, b, splits=1))                 # the same products in the same order
    acc = torch.ones(m, n, device=DEV)
    G.gemm(A, B, a_mn=a_mn, b_mn=b_mn, accumulate_into=acc)
    _close(acc, a.double() @ b.double().t() + 1, TF32)


def test_fp32_operand_that_tma_cannot_read_is_transposed():
    a, b = torch.randn(40, 10, device=DEV), torch.randn(40, 24, device=DEV)       # stored [K, M], rows of 40 bytes
    _close(G.gemm(a, b, a_mn=True, b_mn=True), a.double().t() @ b.double(), TF32)
    view = torch.randn(33, 67, device=DEV)[:, 1:65]                                  # rows that start off 16 bytes
    _close(G.gemm(view, view, a_mn=True, b_mn=True), view.double().t() @ view.double(), TF32)


def test_batched_transposed_fp32():
    a, b = torch.randn(3, 36, 140, device=DEV), torch.randn(3, 36, 72, device=DEV)
    _close(G.gemm(a, b, a_mn=True, b_mn=True), a.double().transpose(1, 2) @ b.double(), TF32)


# bf16 results: half a unit of 2^-8 per element at most; the sums themselves are fp32
BF16 = 2.0 ** -8


@pytest.mark.parametrize("m,n,k", [(1, 8, 1536), (16, 512, 2048), (129, 384, 1544), (333, 512, 2048), (333, 520, 4096), (1024, 512, 2048), (1000, 509, 1600), (64, 64, 1536)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_sums_divided_over_a_cluster(m, n, k, a_mn, b_mn):
    """Around the rule's edges: 24 K blocks, ranks without a block (K = 1544, 1600), ragged rows and columns, 8, 4 and 1 CTAs a tile."""
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    a, b = torch.randn(m, k, device=DEV, generator=g).bfloat16(), torch.randn(n, k, device=DEV, generator=g).bfloat16()
    A, B = a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b
    want = a.double() @ b.double().t()
    got = G.gemm(A, B, a_mn=a_mn, b_mn=b_mn)
    _close(got, want, BF16)
    assert torch.equal(got, G.gemm(A, B, a_mn=a_mn, b_mn=b_mn))         # summed in rank order
    f = torch.empty(m, n, device=DEV)
    G.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32, out=f)
    _close(f, want, 1e-5)
    if not (a_mn or b_mn):
        bias, res = torch.randn(n, device=DEV, generator=g), torch.randn(m, n, device=DEV, generator=g).bfloat16()
        got, pre = G.gemm(a, b, bias=bias, act="relu", residual=res, want_aux=True, alpha=0.5)
        v = 0.5 * want + bias.double()
        _close(pre, v, BF16)
        _close(got, v.clamp_min(0) + res.double(), BF16)
        saved = torch.randn(m, n, device=DEV, generator=g).bfloat16()
        _close(G.gemm(a, b, aux_in=saved, dact="relu"), want * (saved > 0).double(), BF16)
        acc = torch.ones(m, n, device=DEV)
        G.gemm(a, b, accumulate_into=acc, splits=0)
        _close(acc, want + 1, 1e-5)


@pytest.mark.parametrize("m,n,k,stride", [(333, 512, 512, 512), (333, 512, 512, 520), (40, 136, 64, 140), (2048, 512, 128, 512), (300, 2000, 96, 2000)])
def test_residual_fetched_ahead(m, n, k, stride):
    """64- and 128-wide tiles; a residual whose rows are 16-byte pieces, lie apart, or are read one by one."""
    g = torch.Generator(device=DEV).manual_seed(m + n)
    a, b = torch.randn(m, k, device=DEV, generator=g).bfloat16(), torch.randn(n, k, device=DEV, generator=g).bfloat16()
    res = torch.randn(m, stride, device=DEV, generator=g).bfloat16()[:, :n]
    want = a.double() @ b.double().t() + res.double()
    for bn in (0, 64, 128, 256):
        _close(G.gemm(a, b, residual=res, bn=bn), want, BF16)


@pytest.mark.parametrize("dtype", [torch.int8, torch.float8_e4m3fn])
@pytest.mark.parametrize("bn", [0, 64, 128, 256, 512])
@pytest.mark.parametrize("m,n,k", [(1, 24, 128), (300, 200, 144), (513, 776, 2064)])
def test_8bit_tiles(dtype, bn, m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m + n)
    if dtype == torch.int8:
        a, b = (torch.randint(-127, 128, s, device=DEV, generator=g).to(torch.int8) for s in ((m, k), (n, k)))
    else:
        a, b = (torch.randn(s, device=DEV, generator=g).to(dtype) for s in ((m, k), (n, k)))
    rs, cs = torch.rand(m, device=DEV, generator=g) + 0.5, torch.rand(n, device=DEV, generator=g) + 0.5
    want = a.double() @ b.double().t()
    got = G.gemm(a, b, row_scale=rs, col_scale=cs, out_dtype=torch.float32, bn=bn)
    # e4m3 products are summed with fewer bits than fp32 (about 2^-13 of the largest), integers exactly
    _close(got, want * rs.double()[:, None] * cs.double(), 1e-6 if dtype == torch.int8 else 2e-3)
    if dtype == torch.int8:
        assert torch.equal(G.gemm(a, b, out_dtype=torch.int32, bn=bn).double(), want)


@pytest.mark.parametrize("m,n,k", [(256, 256, 32), (511, 777, 100), (2048, 1500, 64), (4096, 4096, 36)])
def test_fp32_pairs_and_narrow_tiles_agree(m, n, k):
    """The rule for fp32 tiles moves between 64, 128 and pairs of 256: the same sum in the same order on each."""
    a, b = torch.randn(m, k, device=DEV), torch.randn(n, k, device=DEV)
    want = a.double() @ b.double().t()
    one = G.gemm(a, b, bn=128, splits=1)
    _close(one, want, TF32)
    for bn in (64, 256):
        got = torch.empty(m, n, device=DEV)
        rec = G.gemm(a, b, out=got, splits=1, _prepare=True)
        nv.check(nv.cuda().b200_gemm_launch(bytes(rec[0]), bn, 148, nv.stream_ptr()), "launch")
        assert torch.equal(got, one)
