// The host side of the calls that take less time on the GPU than Python takes to prepare them: checks, result tensors, launch records and
// launches of matrix products, softmax and linear attention, and the quantised layers, for CUDA tensors. The Python functions of the same names
// (ops/gemm.py, ops/kernels.py, ops/linear_attention.py, ops/quant_kernels.py, ops/mx.py) hold the contract and the CPU path and pass CUDA tensors on
// to these; autograd stays there.
#include <torch/extension.h>

#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <optional>
#include <vector>

#include "../attention/linattn_sm100.h"
#include "../gemm/gemm_mx_sm100.h"
#include "../gemm/gemm_sm100.h"

extern "C" int b200_quant_rows(const void* x, int is_bf16, long long rows, int cols, long long ldx, void* q, long long ldq, float* scales, int mode,
                               cudaStream_t st);

namespace {

using at::Tensor;
using Opt = std::optional<Tensor>;
namespace py = pybind11;

long long g_launches = 0;              // kernels launched from here (the caller's thread holds the interpreter lock)

[[noreturn]] void value_error(const std::string& m) { throw py::value_error(m); }
[[noreturn]] void type_error(const std::string& m) { throw py::type_error(m); }

void check(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string(what) + " failed with code " + std::to_string(rc));
}

cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

constexpr int MAX_DEVICES = 64;

int device_slot(const at::Device& d) {
  const int i = d.has_index() ? d.index() : 0;
  if (i < 0 || i >= MAX_DEVICES) throw std::runtime_error("device index out of range");
  return i;
}

int num_sms(const at::Device& d) {
  static int sms[MAX_DEVICES] = {};
  const int i = device_slot(d);
  if (!sms[i] && cudaDeviceGetAttribute(&sms[i], cudaDevAttrMultiProcessorCount, i) != cudaSuccess) throw std::runtime_error("no such device");
  return sms[i];
}

// the per-device word that kernels report expired waits in; `_native.status_word` owns it for the life of the process
uint32_t* status(const at::Device& d) {
  static uint32_t* words[MAX_DEVICES] = {};
  const int i = device_slot(d);
  if (!words[i]) {
    const py::object f = py::module_::import("rust_neural_network_b200._native").attr("status_ptr");
    words[i] = reinterpret_cast<uint32_t*>(f(py::module_::import("torch").attr("device")("cuda", i)).cast<uintptr_t>());
  }
  return words[i];
}

bool has(const Opt& t) { return t.has_value() && t->defined(); }
template <typename T = void>
T* ptr(const Opt& t) { return has(t) ? reinterpret_cast<T*>(t->data_ptr()) : nullptr; }
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

// ---------------------------------------------------------------------------------------------------- products
// Can TMA read this 2-D or 3-D operand where it is? Unit inner stride, other strides and base in multiples of 16 bytes.
bool readable(const Tensor& t) {
  const int64_t q = 16 / t.element_size(), n = t.dim();
  return t.stride(n - 1) == 1 && t.stride(n - 2) % q == 0 && aligned16(t.data_ptr()) && t.stride(n - 2) >= t.size(n - 1) &&
         (n == 2 || t.size(0) == 1 || t.stride(0) % q == 0);
}

struct Operand { Tensor t; int64_t batch, rows, cols, ld, stride; };

// `t` itself, or a copy whose rows are padded to multiples of 16 bytes
Operand operand(const Tensor& t) {
  if (t.dim() != 2 && t.dim() != 3) value_error("gemm operands must be 2-D or 3-D");
  if (t.dim() == 2 && readable(t)) return {t, 1, t.size(0), t.size(1), t.stride(0), t.size(0) * t.stride(0)};
  Tensor u = t.dim() == 2 ? t.unsqueeze(0) : t;
  if (!readable(u)) {
    const int64_t q = 16 / t.element_size(), inner = cdiv(u.size(2), q) * q;
    Tensor v = at::zeros({u.size(0), u.size(1), inner}, u.options()).narrow(2, 0, u.size(2));
    v.copy_(u);
    u = v;
  }
  return {u, u.size(0), u.size(1), u.size(2), u.stride(1), u.stride(0)};
}

int kind_of(const Tensor& a, const Tensor& b) {
  const auto x = a.scalar_type(), y = b.scalar_type();
  if (x == at::kBFloat16 && y == at::kBFloat16) return b200::GEMM_BF16;
  if (x == at::kFloat && y == at::kFloat) return b200::GEMM_F32;
  if (x == at::kChar && y == at::kChar) return b200::GEMM_S8S8;
  if (x == at::kByte && y == at::kChar) return b200::GEMM_U8S8;
  if (x == at::kFloat8_e4m3fn && y == at::kFloat8_e4m3fn) return b200::GEMM_E4M3;
  type_error(std::string("gemm operands must be bf16 x bf16, fp32 x fp32, int8 x int8, uint8 x int8 or e4m3 x e4m3 (got ") + c10::toString(x) + ", " +
             c10::toString(y) + ")");
}

struct Product {
  b200::GemmArgs args = {};
  int bn = 0;
  Tensor res, aux;
  std::vector<Tensor> keep;            // what the record points at
};

// `out_code`: mode of the result, or -1 for the operands' own; `exact`: the record is run by another kernel, which divides no sum
Product prepare(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const Opt& bias, int act, const Opt& residual_, const Opt& aux_in_, int dact,
                bool want_aux, double alpha, int out_code, const Opt& accumulate_into, int64_t splits, int bn, const Opt& alpha_t_, const Opt& row_scale_,
                const Opt& col_scale_, const Opt& out_, const Opt& m_valid, const Opt& k_valid, bool exact) {
  using namespace b200;
  const int kind = kind_of(a, b);
  const bool is_f32 = kind == GEMM_F32, lowp = kind >= GEMM_S8S8;
  if (lowp && (a_mn || b_mn)) value_error("8-bit GEMM operands must be K-major");
  const bool squeeze = a.dim() == 2;
  const Operand x = operand(a), y = operand(b);
  if (x.batch != y.batch) value_error("batch mismatch");
  const int64_t batch = x.batch, M = a_mn ? x.cols : x.rows, K = a_mn ? x.rows : x.cols, N = b_mn ? y.cols : y.rows, Kb = b_mn ? y.rows : y.cols;
  if (K != Kb) value_error("gemm K mismatch: " + std::to_string(K) + " vs " + std::to_string(Kb));
  const at::Device dev = a.device();
  const int sms = num_sms(dev);

  int mode;
  Tensor out;
  bool may_divide = false;
  if (has(accumulate_into)) {
    out = *accumulate_into;
    if (out.scalar_type() != at::kFloat || !out.is_contiguous()) value_error("accumulate_into must be a contiguous fp32 tensor");
    mode = OUT_F32_ATOMIC;
  } else {
    mode = out_code >= 0 ? out_code : is_f32 ? OUT_F32 : OUT_BF16;
    if (mode == OUT_I32 && kind != GEMM_S8S8 && kind != GEMM_U8S8) type_error("an int32 result needs integer operands");
    if (has(out_)) {
      out = *out_;
      const auto want = mode == OUT_I32 ? at::kInt : mode == OUT_F32 ? at::kFloat : at::kBFloat16;
      if (out.scalar_type() != want || out.stride(-1) != 1 || out.numel() != batch * M * N)
        value_error("`out` must have the result's dtype, size and a unit inner stride");
      if (splits > 1) value_error("`out` and split-K do not go together (split-K accumulates into a zeroed fp32 buffer)");
      may_divide = splits == 0;
      splits = 1;
    }
  }
  const bool linear = act == ACT_NONE && !has(aux_in_) && !want_aux;
  // The launcher chooses the tiles (bn = 0) and may divide a sum over the CTAs of a cluster (0 splits). Here: into how many parts that
  // are added in memory an fp32 result's contraction is split, on the tiles that go with it.
  const bool one_cta = exact || (splits == 1 && !may_divide);
  const int64_t num_kb = cdiv(K, is_f32 ? 32 : lowp ? 128 : 64);
  if (splits == 0) {
    splits = 1;
    if ((mode == OUT_F32 || mode == OUT_F32_ATOMIC) && num_kb >= (lowp ? 64 : 16) && linear) {
      const int64_t row_tiles = cdiv(M, 128) * batch, t256 = row_tiles * cdiv(N, 256);
      // Few tiles and a long K (weight gradients): split-K fills the machine either way, and the wider tile moves a third less
      // operand traffic from L2 per FLOP (measured 167 -> 113 us on 2048 x 512 x 65536).
      int sbn = bn;
      if (!sbn) {
        if (!is_f32 && !lowp && N >= 256 && (t256 >= sms || K >= 16 * 64 * std::max<int64_t>(1, sms / std::max<int64_t>(t256, 1)))) sbn = 256;
        else sbn = N <= 64 && !is_f32 && !lowp ? 64 : 128;
      }
      const int64_t tiles = row_tiles * cdiv(N, sbn);
      if (tiles > 0 && tiles < sms / 2) splits = std::max<int64_t>(1, std::min(sms / tiles, num_kb / 8));
      if (splits > 1 || sbn == 256) bn = sbn;
    }
  }
  if (splits > 1) {
    const int64_t kb = std::max<int64_t>(1, num_kb);
    splits = cdiv(kb, cdiv(kb, splits));
  }
  if (splits > 1) {
    if (mode == OUT_BF16 || !linear) value_error("split-K needs an fp32 output and a linear epilogue");
    mode = OUT_F32_ATOMIC;
  }
  if (!out.defined()) {
    const auto opts = a.options().dtype(mode == OUT_I32 ? at::kInt : mode != OUT_BF16 ? at::kFloat : at::kBFloat16);
    const std::vector<int64_t> shape = squeeze ? std::vector<int64_t>{M, N} : std::vector<int64_t>{batch, M, N};
    out = mode == OUT_F32_ATOMIC ? at::zeros(shape, opts) : at::empty(shape, opts);
  }
  int64_t ldc, stride_c;
  Tensor out3 = out;
  if (out.dim() == 2 && batch == 1 && out.size(0) == M && out.size(1) == N) {
    ldc = out.stride(0);
    stride_c = M * ldc;
  } else {
    if (out.dim() != 3) out3 = out.view({batch, M, N});
    ldc = out3.stride(1);
    stride_c = batch > 1 ? out3.stride(0) : M * ldc;
  }
  Tensor aux;
  if (want_aux) aux = squeeze ? at::empty({M, N}, a.options().dtype(at::kBFloat16)) : at::empty({batch, M, N}, a.options().dtype(at::kBFloat16));
  Opt aux_in = aux_in_, residual = residual_, row_scale = row_scale_, col_scale = col_scale_, alpha_t = alpha_t_;
  if (has(aux_in)) {
    aux_in = aux_in->contiguous().view({batch, M, N});
    if (aux_in->scalar_type() != at::kBFloat16) type_error("aux_in must be bf16");
  }
  if (has(residual)) {
    residual = residual->reshape({batch, M, N});
    if (residual->scalar_type() != at::kBFloat16) residual = residual->to(at::kBFloat16);
    if (residual->stride(-1) != 1) residual = residual->contiguous();
  }
  if (has(bias) && bias->scalar_type() != at::kFloat && bias->scalar_type() != at::kBFloat16) type_error("bias must be fp32 or bf16");
  if ((want_aux || has(aux_in)) && ldc != N) value_error("aux tensors need a dense output (ldc == N)");
  if (has(row_scale)) {
    row_scale = row_scale->to(at::kFloat).contiguous();
    if (row_scale->numel() != batch * M) value_error("row_scale needs one value per row of A");
  }
  if (has(col_scale)) {
    col_scale = col_scale->to(at::kFloat).contiguous();
    if (col_scale->numel() != N) value_error("col_scale needs one value per row of B");
  }
  for (const auto* v : {&m_valid, &k_valid})
    if (has(*v) && ((*v)->scalar_type() != at::kInt || (*v)->numel() != batch || !(*v)->is_cuda()))
      value_error(std::string(v == &m_valid ? "m_valid" : "k_valid") + " must be an int32 device tensor with one entry per batch");
  if (has(alpha_t) && alpha_t->scalar_type() != at::kFloat) alpha_t = alpha_t->to(at::kFloat);

  Product r;
  GemmArgs& g = r.args;
  GemmParams& p = g.p;
  p.M = g.M = (int)M; p.N = g.N = (int)N; p.K = g.K = (int)K; p.batch = g.batch = (int)batch;
  p.splits = one_cta || splits > 1 ? (int)splits : 0;
  p.C = out3.data_ptr(); p.ldc = ldc; p.strideC = stride_c;
  if (has(bias)) {
    p.bias = bias->data_ptr(); p.bias_f32 = bias->scalar_type() == at::kFloat;
    p.bias_vec_ok = aligned16(p.bias) && N % 4 == 0 && bias->is_contiguous();
    p.strideBias = bias->dim() == 2 ? N : 0;                       // [batch, N]: one vector per batch
  }
  if (has(residual)) {
    p.residual = residual->data_ptr(); p.ldr = residual->stride(1); p.strideR = residual->stride(0);
    p.res_vec_ok = p.ldr % 8 == 0 && aligned16(p.residual) && (batch == 1 || p.strideR % 8 == 0);
  }
  p.aux_out = aux.defined() ? aux.data_ptr() : nullptr; p.aux_in = ptr(aux_in);
  p.alpha = (float)alpha; p.alpha_ptr = ptr<float>(alpha_t); p.act = act; p.dact = dact; p.out_mode = mode;
  const int es = mode != OUT_BF16 ? 4 : 2;
  p.vec_ok = ldc * es % 16 == 0 && aligned16(p.C) && (batch == 1 || stride_c * es % 16 == 0) && ((!want_aux && !has(aux_in)) || N % 8 == 0);
  p.row_scale = ptr<float>(row_scale); p.col_scale = ptr<float>(col_scale); p.status = status(dev);
  p.m_valid = ptr<int>(m_valid); p.k_valid = ptr<int>(k_valid);
  g.A = x.t.data_ptr(); g.lda = x.ld; g.strideA = x.stride; g.a_mn = a_mn;
  g.B = y.t.data_ptr(); g.ldb = y.ld; g.strideB = y.stride; g.b_mn = b_mn;
  g.dtype = kind;
  r.bn = bn;
  r.res = squeeze && out.dim() == 3 ? out3.select(0, 0) : out;
  r.aux = aux;
  r.keep = {x.t, y.t, out3};
  for (const Opt* t : std::initializer_list<const Opt*>{&bias, &residual, &aux_in, &row_scale, &col_scale, &alpha_t, &m_valid, &k_valid})
    if (has(*t)) r.keep.push_back(**t);
  return r;
}

py::object gemm(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const Opt& bias, int act, const Opt& residual, const Opt& aux_in, int dact,
                bool want_aux, double alpha, int out_code, const Opt& accumulate_into, int64_t splits, int bn, const Opt& alpha_t, const Opt& row_scale,
                const Opt& col_scale, const Opt& out, const Opt& m_valid, const Opt& k_valid) {
  const Product r = prepare(a, b, a_mn, b_mn, bias, act, residual, aux_in, dact, want_aux, alpha, out_code, accumulate_into, splits, bn, alpha_t, row_scale,
                            col_scale, out, m_valid, k_valid, false);
  check(b200_gemm_launch(&r.args, r.bn, num_sms(a.device()), stream()), "b200_gemm_launch");
  ++g_launches;
  const Tensor& res = has(accumulate_into) ? *accumulate_into : r.res;
  if (want_aux) return py::make_tuple(res, r.aux);
  return py::cast(res);
}

// a fused kernel runs this product itself: the filled launch record, the tile width, the results and everything that the record points at
py::tuple gemm_record(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const Opt& bias, int act, const Opt& residual, const Opt& aux_in, int dact,
                      bool want_aux, double alpha, int out_code, const Opt& accumulate_into, int64_t splits, int bn, const Opt& alpha_t,
                      const Opt& row_scale, const Opt& col_scale, const Opt& out, const Opt& m_valid, const Opt& k_valid) {
  const Product r = prepare(a, b, a_mn, b_mn, bias, act, residual, aux_in, dact, want_aux, alpha, out_code, accumulate_into, splits, bn, alpha_t, row_scale,
                            col_scale, out, m_valid, k_valid, true);
  return py::make_tuple(py::bytes(reinterpret_cast<const char*>(&r.args), sizeof(r.args)), r.bn, r.res,
                        r.aux.defined() ? py::cast(r.aux) : py::object(py::none()), r.keep);
}

// ---------------------------------------------------------------------------------------------------- attention
b200::AttnTensor attn(const Tensor& t) { return {t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)}; }
bool attn_ok(const Tensor& t) {
  return t.stride(3) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0 && aligned16(t.data_ptr());
}
Tensor attn_ready(const Tensor& t) { return attn_ok(t) ? t : t.contiguous(); }

std::pair<Tensor, Tensor> flash_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, double scale, bool causal) {
  if (q_.scalar_type() != at::kBFloat16) type_error("flash attention kernels take bf16");
  const Tensor q = attn_ready(q_), k = attn_ready(k_), v = attn_ready(v_);
  const int64_t B = q.size(0), Sq = q.size(1), H = q.size(2), hd = q.size(3);
  Tensor o = at::empty({B, Sq, H, hd}, q.options()), lse = at::empty({B, H, Sq}, q.options().dtype(at::kFloat));
  b200::FlashArgs a = {};
  a.q = attn(q); a.k = attn(k); a.v = attn(v); a.o = attn(o);
  a.lse = lse.data_ptr<float>();
  a.B = (int)B; a.H = (int)H; a.Sq = (int)Sq; a.Skv = (int)k.size(1); a.hd = (int)hd;
  a.scale = (float)scale; a.causal = causal; a.status = status(q.device());
  check(b200_flash_fwd(&a, stream()), "flash_fwd");
  ++g_launches;
  return {o, lse};
}

std::tuple<Tensor, Tensor, Tensor> flash_bwd(const Tensor& dout_, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                                             double scale, bool causal, const Opt& dq_, const Opt& dk_, const Opt& dv_) {
  const int64_t B = q.size(0), Sq = q.size(1), H = q.size(2), hd = q.size(3), Skv = k.size(1);
  const Tensor dout = attn_ready(dout_);
  const auto bf = q.options().dtype(at::kBFloat16), f32 = q.options().dtype(at::kFloat);
  Tensor dq = has(dq_) ? *dq_ : at::empty({B, Sq, H, hd}, bf), dk = has(dk_) ? *dk_ : at::empty({B, Skv, H, hd}, bf),
         dv = has(dv_) ? *dv_ : at::empty({B, Skv, H, hd}, bf);
  Tensor delta = at::empty({B, H, Sq}, f32), accum;
  if (Skv > 128) accum = at::empty({B, H, cdiv(Sq, 32) * 32, hd}, f32);       // the kernel's own layout; one key block adds nothing up and writes dq itself
  b200::FlashArgs a = {};
  a.q = attn(q); a.k = attn(k); a.v = attn(v); a.o = attn(o);
  a.dout = attn(dout); a.dq = attn(dq); a.dk = attn(dk); a.dv = attn(dv);
  a.lse = lse.data_ptr<float>(); a.delta = delta.data_ptr<float>(); a.dq_accum = accum.defined() ? accum.data_ptr<float>() : nullptr;
  a.B = (int)B; a.H = (int)H; a.Sq = (int)Sq; a.Skv = (int)Skv; a.hd = (int)hd;
  a.scale = (float)scale; a.causal = causal; a.status = status(q.device());
  check(b200_flash_bwd(&a, stream()), "flash_bwd");
  g_launches += Skv > 128 ? 3 : 2;
  return {dq, dk, dv};
}

constexpr int64_t LA_CHUNK = 128;

b200::LinAttnArgs la_args(const Tensor& q, const Tensor& k, const Tensor& v, double scale, double eps, int kind, int64_t n_seg) {
  b200::LinAttnArgs a = {};
  a.q = attn(q); a.k = attn(k); a.v = attn(v);
  a.B = (int)q.size(0); a.S = (int)q.size(1); a.H = (int)q.size(2); a.hd = (int)q.size(3);
  a.scale = (float)scale; a.eps = (float)eps; a.kind = kind; a.status = status(q.device());
  a.n_seg = (int)n_seg; a.seg_chunks = (int)cdiv(cdiv(q.size(1), LA_CHUNK), n_seg);
  return a;
}

// (q, k, v as the kernels read them, O, denominators, the segments' states or nothing, the remainder of O or nothing)
py::tuple linattn_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, double scale, double eps, int kind, bool keep_remainder, int64_t n_seg) {
  const Tensor q = attn_ready(q_), k = attn_ready(k_), v = attn_ready(v_);
  const int64_t B = q.size(0), S = q.size(1), H = q.size(2), d = q.size(3);
  const auto bf = q.options(), f32 = q.options().dtype(at::kFloat);
  Tensor o = at::empty({B, S, H, d}, bf), den = at::empty({B, H, S}, f32);
  Tensor o_lo = keep_remainder ? at::empty_like(o) : at::empty({0}), seg = n_seg > 1 ? at::empty({B * H, n_seg, d * d + d}, f32) : at::empty({0});
  b200::LinAttnArgs a = la_args(q, k, v, scale, eps, kind, n_seg);
  a.o = attn(o); a.den = den.data_ptr<float>();
  if (keep_remainder) a.o_lo = attn(o_lo);
  if (n_seg > 1) a.seg = seg.data_ptr<float>();
  check(b200_linattn(&a, 0, stream()), "linattn");
  g_launches += n_seg == 1 ? 1 : 3;
  return py::make_tuple(q, k, v, o, den, seg, o_lo);
}

// the whole backward; `s_in`: what the forward started its segments (or its one walk) from, or nothing
std::tuple<Tensor, Tensor, Tensor> linattn_bwd(const Tensor& dout_, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& den,
                                               const Tensor& s_in, const Tensor& o_lo, double scale, double eps, int kind) {
  const int64_t B = q.size(0), S = q.size(1), H = q.size(2), d = q.size(3), n_seg = s_in.numel() && s_in.dim() == 3 ? s_in.size(1) : 1;
  const Tensor dout = attn_ok(dout_) && dout_.scalar_type() == at::kBFloat16 ? dout_ : dout_.to(at::kBFloat16).contiguous();
  Tensor dq = at::empty_like(o), dk = at::empty_like(o), dv = at::empty_like(o);
  Tensor g = at::empty({B, S, H, d}, q.options()), dden = at::empty({B, H, S}, den.options()), dseg;
  b200::LinAttnArgs a = la_args(q, k, v, scale, eps, kind, n_seg);
  a.o = attn(o); a.den = den.data_ptr<float>(); a.dout = attn(dout); a.dq = attn(dq); a.dk = attn(dk); a.dv = attn(dv);
  a.g = attn(g); a.dden = dden.data_ptr<float>();
  if (o_lo.numel()) a.o_lo = attn(o_lo);
  if (n_seg > 1) {
    dseg = at::empty_like(s_in);
    a.seg = s_in.data_ptr<float>(); a.dseg = dseg.data_ptr<float>();
  } else if (s_in.numel()) {
    a.s_in = s_in.data_ptr<float>();
  }
  check(b200_linattn(&a, 4, stream()), "linattn");
  g_launches += n_seg == 1 ? 3 : 5;
  return {dq, dk, dv};
}

// ---------------------------------------------------------------------------------------------------- quantised operands
Tensor rows_of(const Tensor& x) {
  Tensor y = x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16 ? x : x.to(at::kFloat);
  return y.stride(-1) == 1 ? y : y.contiguous();
}

std::pair<Tensor, Tensor> quant_rows(const Tensor& x_, int mode) {
  const Tensor x = rows_of(x_);
  const int64_t rows = x.size(0), cols = x.size(1);
  Tensor q = at::empty({rows, cols}, x.options().dtype(mode == 0 ? at::kChar : at::kFloat8_e4m3fn)), s = at::empty({rows}, x.options().dtype(at::kFloat));
  check(b200_quant_rows(x.data_ptr(), x.scalar_type() == at::kBFloat16, rows, (int)cols, x.stride(0), q.data_ptr(), cols, s.data_ptr<float>(), mode, stream()),
        "quant_rows");
  ++g_launches;
  return {q, s};
}

std::pair<Tensor, Tensor> mx_quant(const Tensor& x_, int kind, double tensor_scale, int64_t sf_bytes) {
  const Tensor x = rows_of(x_);
  const int64_t rows = x.size(0), K = x.size(1);
  const auto u8 = x.options().dtype(at::kByte);
  Tensor data = at::empty({rows, kind == 0 ? K : K / 2}, u8), sf = at::empty({sf_bytes}, u8);
  check(b200_mx_quant(x.data_ptr(), x.scalar_type() == at::kBFloat16, x.stride(0), rows, (int)K, kind, (float)tensor_scale, data.data_ptr(), sf.data_ptr(),
                      stream()), "mx_quant");
  ++g_launches;
  return {data, sf};
}

Tensor gemm_mx(const Tensor& a, const Tensor& sfa, const Tensor& b, const Tensor& sfb, int64_t M, int64_t N, int64_t K, int kind, double alpha, bool f32,
               const Opt& bias_) {
  Tensor out = at::empty({M, N}, a.options().dtype(f32 ? at::kFloat : at::kBFloat16));
  Opt bias = bias_;
  if (has(bias)) {
    if (bias->scalar_type() != at::kBFloat16 || bias->dim() != 1 || bias->size(0) != N) value_error("bias must be a bf16 vector of N elements");
    if (!bias->is_contiguous() || !aligned16(bias->data_ptr())) bias = bias->clone(at::MemoryFormat::Contiguous);
  }
  b200::MxGemmArgs g = {};
  g.A = a.data_ptr(); g.B = b.data_ptr(); g.sfa = sfa.data_ptr(); g.sfb = sfb.data_ptr();
  g.C = out.data_ptr(); g.ldc = N;
  g.M = (int)M; g.N = (int)N; g.K = (int)K;
  g.out_f32 = f32; g.alpha = (float)alpha; g.kind = kind; g.bias = ptr(bias); g.status = status(a.device());
  check(b200_gemm_mx(&g, num_sms(a.device()), stream()), "gemm_mx");
  ++g_launches;
  return out;
}

}  // namespace

PYBIND11_MODULE(_b200nn_entry, m) {
  m.def("gemm", &gemm);
  m.def("gemm_record", &gemm_record);
  m.def("flash_fwd", &flash_fwd);
  m.def("flash_bwd", &flash_bwd);
  m.def("linattn_fwd", &linattn_fwd);
  m.def("linattn_bwd", &linattn_bwd);
  m.def("quant_rows", &quant_rows);
  m.def("mx_quant", &mx_quant);
  m.def("gemm_mx", &gemm_mx);
  m.def("launches", [] { return g_launches; });
  m.def("reset_launches", [] { g_launches = 0; });
}
