// Host side of the tensor-level entry points (ops.py) in C++: argument checks, output allocation with PyTorch's caching
// allocator, the argument block and the call into libqlin_b200.so on the tensors' device and current stream.
//
// A deploy-time Linear is two kernels of a few microseconds each when a handful of tokens go through it.  Building the two
// argument blocks field by field through ctypes, entering device contexts and looking up streams in Python cost about
// 72 us a call at 1 x 4096 x 14336, four times what the GPU needed; with the same steps here a call takes 22 us, of which
// the two kernels are 19.
//
// No kernel, no fallback and no state of its own: everything a call keeps is one status word per device, which lives as
// long as the process.
#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/stl.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

#include <mutex>
#include <optional>
#include <stdexcept>
#include <string>
#include <variant>
#include <vector>

#include "../../../include/qlin_b200.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;
using Scalar = std::variant<Tensor, double>;

[[noreturn]] void raise(const std::string& msg) { throw std::runtime_error(msg); }

void check(int rc, const char* what) {
  if (rc != QLIN_OK) raise(std::string(what) + " failed with status " + std::to_string(rc) + ": " + qlin_last_error_string());
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kChar:
      return QLIN_DT_I8;
    case at::kByte:
      return QLIN_DT_U8;
    case at::kInt:
      return QLIN_DT_I32;
    case at::kFloat:
      return QLIN_DT_F32;
    case at::kHalf:
      return QLIN_DT_F16;
    case at::kBFloat16:
      return QLIN_DT_BF16;
    case at::kFloat8_e4m3fn:
      return QLIN_DT_F8E4M3;
    case at::kFloat8_e5m2:
      return QLIN_DT_F8E5M2;
    default:
      return QLIN_DT_NONE;
  }
}

at::ScalarType scalar_type(int code) {
  switch (code) {
    case QLIN_DT_I32:
      return at::kInt;
    case QLIN_DT_F32:
      return at::kFloat;
    case QLIN_DT_F16:
      return at::kHalf;
    case QLIN_DT_BF16:
      return at::kBFloat16;
    default:
      raise("unsupported output dtype");
  }
}

bool is_float(at::ScalarType t) { return t == at::kFloat || t == at::kHalf || t == at::kBFloat16; }

// All given tensors are on one CUDA device, which is returned.
at::Device require_cuda(std::initializer_list<const Tensor*> tensors) {
  std::optional<at::Device> dev;
  for (const Tensor* t : tensors) {
    if (t == nullptr || !t->defined()) continue;
    if (!t->is_cuda()) raise("qlin_b200 ops run on CUDA tensors only (there is no CPU path)");
    if (!dev) {
      dev = t->device();
    } else if (t->device() != *dev) {
      raise("tensors on different devices: " + dev->str() + " and " + t->device().str());
    }
  }
  if (!dev) raise("no tensor given");
  return *dev;
}

const Tensor* ptr_of(const OptTensor& t) { return t ? &*t : nullptr; }
void* data(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

Tensor empty(at::IntArrayRef sizes, at::ScalarType t, at::Device dev) { return at::empty(sizes, at::TensorOptions().dtype(t).device(dev)); }

// fp32, one-dimensional, contiguous (undefined stays undefined).
Tensor f32(const OptTensor& t) {
  if (!t) return Tensor();
  if (t->scalar_type() == at::kFloat && t->is_contiguous()) return *t;
  return t->reshape({-1}).to(at::kFloat).contiguous();
}

// K-contiguous 2-D view or copy whose row stride and base are 16-byte aligned.
Tensor pad_k(const Tensor& t) {
  const int64_t es = t.element_size();
  if (t.stride(1) == 1 && (t.stride(0) * es) % 16 == 0 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && t.stride(0) >= t.size(1)) return t;
  const int64_t k = t.size(1), kp = (k * es + 15) / 16 * 16 / es;
  Tensor buf = at::zeros({t.size(0), kp}, t.options());
  Tensor view = buf.narrow(1, 0, k);
  view.copy_(t);
  return view;
}

// Status word of a device, created on first use and never released (kernels in flight may write it until the process ends).
Tensor status_word(int index) {
  static std::mutex* mutex = new std::mutex;
  static std::vector<Tensor>* words = new std::vector<Tensor>(64);
  if (index < 0 || index >= 64) raise("device ordinal out of range");
  std::lock_guard<std::mutex> lock(*mutex);
  Tensor& w = (*words)[index];
  if (!w.defined()) w = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(index))));
  return w;
}

void* stream_of(at::Device dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

// ------------------------------------------------------------------------------------------------ GEMM
struct Chain {  // chunk function, epilogue and rounding dtypes of a GEMM call
  int64_t chunk_k;
  int trun_bits, max_acc_bits, trunc_then_acc, clamp_dl16, epilogue, prod_round, scale_round, mid_round, acc_round;
};

struct Scatter {
  std::vector<int64_t> bases;
  int64_t rows = 0, row0 = 0, ld = 0;
};

// A quantiser call whose launch was left to the GEMM that reads its codes.
struct QuantCall {
  qlin_quant_args args = {};
  qlin_scalar_src src[4] = {};
  bool any_src = false;
  std::vector<Tensor> keep;  // tensors the argument block points into
};

Tensor gemm_impl(const Tensor& a_in, const Tensor& b_in, const OptTensor& c_in, const OptTensor& out_in, const Chain& ch, const OptTensor& row_scale,
                 const OptTensor& col_scale, const OptTensor& bias, const Scatter* scatter, int64_t max_ctas, int out_code, const QuantCall* quant = nullptr) {
  const at::Device dev = require_cuda({&a_in, &b_in, ptr_of(c_in), ptr_of(out_in), ptr_of(row_scale), ptr_of(col_scale), ptr_of(bias)});
  if (a_in.dim() != 2 || b_in.dim() != 2 || a_in.size(1) != b_in.size(1)) raise("incompatible shapes: a [M,K] and b [N,K] are wanted");
  const at::ScalarType kt = a_in.scalar_type();
  if (kt != b_in.scalar_type() || (kt != at::kChar && kt != at::kFloat8_e4m3fn && kt != at::kFloat8_e5m2))
    raise("operands must both be int8, float8_e4m3fn or float8_e5m2");
  const bool f8 = kt != at::kChar;
  const int64_t M = a_in.size(0), K = a_in.size(1), N = b_in.size(0);
  const at::ScalarType raw = f8 ? at::kFloat : at::kInt;
  const at::ScalarType ot = ch.epilogue == QLIN_EPI_RAW ? raw : (out_code == QLIN_DT_NONE ? at::kFloat : scalar_type(out_code));
  const c10::cuda::CUDAGuard guard(dev);
  int64_t ldd = N;
  Tensor out;
  if (scatter != nullptr) {
    if (out_in || c_in) raise("scatter excludes out and c");
    ldd = scatter->ld > 0 ? scatter->ld : N;
  } else if (!out_in) {
    out = empty({M, N}, ot, dev);
  } else {
    out = *out_in;
    if (out.scalar_type() != ot || out.dim() != 2 || out.size(0) != M || out.size(1) != N || out.stride(1) != 1) raise("out has the wrong dtype, shape or layout");
    ldd = out.stride(0);
  }
  if (M == 0 || N == 0) return out;
  if (K == 0) raise("K must be positive");
  const Tensor a = pad_k(a_in), b = pad_k(b_in);
  Tensor c;
  if (c_in) {
    if (c_in->scalar_type() != raw || c_in->dim() != 2 || c_in->size(0) != M || c_in->size(1) != N) raise("c must be an [M,N] tensor of the accumulator dtype");
    c = c_in->stride(1) != 1 ? c_in->contiguous() : *c_in;
  }
  const Tensor rs = f32(row_scale), cs = f32(col_scale), bs = f32(bias);
  if (rs.defined() && rs.numel() != 1 && rs.numel() != M) raise("row_scale must have 1 or M elements");
  if (cs.defined() && cs.numel() != 1 && cs.numel() != N) raise("col_scale must have 1 or N elements");
  if (bs.defined() && bs.numel() != N) raise("bias must have N elements");
  qlin_gemm_args g = {};
  g.a = data(a);
  g.b = data(b);
  g.c = data(c);
  g.d = data(out);
  g.row_scale = static_cast<const float*>(data(rs));
  g.col_scale = static_cast<const float*>(data(cs));
  g.bias = static_cast<const float*>(data(bs));
  g.status = static_cast<int32_t*>(status_word(dev.index()).data_ptr());
  g.lda = a.stride(0);
  g.ldb = b.stride(0);
  g.ldc = c.defined() ? c.stride(0) : 0;
  g.ldd = ldd;
  g.M = static_cast<int32_t>(M);
  g.N = static_cast<int32_t>(N);
  g.K = static_cast<int32_t>(K);
  g.kind = dtype_code(kt);
  g.chunk_k = static_cast<int32_t>(ch.chunk_k);
  g.trun_bits = ch.trun_bits;
  g.max_acc_bits = ch.max_acc_bits;
  g.trunc_then_acc = ch.trunc_then_acc;
  g.clamp_dl16 = ch.clamp_dl16;
  g.epilogue = ch.epilogue;
  g.row_scale_stride = rs.defined() && rs.numel() != 1 ? 1 : 0;
  g.col_scale_stride = cs.defined() && cs.numel() != 1 ? 1 : 0;
  g.prod_round = ch.prod_round;
  g.scale_round = ch.scale_round;
  g.mid_round = ch.mid_round;
  g.acc_round = ch.acc_round;
  g.out_dtype = dtype_code(ot);
  g.max_ctas = static_cast<int32_t>(max_ctas);
  if (scatter != nullptr) {
    if (scatter->bases.size() > 8) raise("at most 8 scatter destinations");
    for (size_t i = 0; i < scatter->bases.size(); ++i) g.scatter_d[i] = reinterpret_cast<void*>(scatter->bases[i]);
    g.scatter_rows = static_cast<int32_t>(scatter->rows);
    g.scatter_row0 = static_cast<int32_t>(scatter->row0);
  }
  if (quant != nullptr) {
    check(qlin_quant_gemm(&quant->args, quant->any_src ? quant->src : nullptr, &g, stream_of(dev)), "qlin_quant_gemm");
  } else {
    check(qlin_gemm(&g, stream_of(dev)), "qlin_gemm");
  }
  return out;
}

OptTensor gemm(const Tensor& a, const Tensor& b, const OptTensor& c, const OptTensor& out, int64_t chunk_k, int trun_bits, int max_acc_bits, bool trunc_then_acc,
               bool clamp_dl16, int epilogue, const OptTensor& row_scale, const OptTensor& col_scale, const OptTensor& bias, int prod_round,
               int scale_round, int mid_round, int acc_round, int64_t max_ctas, int out_code, const std::vector<int64_t>& scatter_bases,
               int64_t scatter_rows, int64_t scatter_row0, int64_t scatter_ld) {
  const Chain ch{chunk_k, trun_bits, max_acc_bits, trunc_then_acc, clamp_dl16, epilogue, prod_round, scale_round, mid_round, acc_round};
  Scatter sc;
  const bool scattered = scatter_rows > 0;
  if (scattered) sc = Scatter{scatter_bases, scatter_rows, scatter_row0, scatter_ld};
  Tensor r = gemm_impl(a, b, c, out, ch, row_scale, col_scale, bias, scattered ? &sc : nullptr, max_ctas, out_code);
  return r.defined() ? OptTensor(r) : std::nullopt;
}

// ------------------------------------------------------------------------------------------------ row quantiser
struct QuantOpts {
  int mode, native_chain, smooth_mul, clamp_codes, levels, dl8_flush, f8_e5m2;
  float shift, add2, dyn_eps;
};

bool is_static(int mode) {
  return mode == QLIN_Q_I8_STATIC || mode == QLIN_Q_I8_STATIC_CLAMP_FIRST || mode == QLIN_Q_I8_STATIC_ROUND_FIRST || mode == QLIN_Q_I8_AFFINE_RCP;
}

// A scalar of the quantiser: a number, or a one-element tensor.  Tensors on the device are left there in the static modes.
float scalar(const Scalar& s, at::Device dev, bool may_stay, qlin_scalar_src& src, bool& any) {
  if (const double* d = std::get_if<double>(&s)) return static_cast<float>(*d);
  const Tensor& t = std::get<Tensor>(s);
  const at::ScalarType st = t.scalar_type();
  if (may_stay && t.device() == dev && t.numel() == 1 && (is_float(st) || st == at::kInt)) {
    src.ptr = t.data_ptr();
    src.dtype = dtype_code(st);
    any = true;
    return 0.0f;
  }
  return static_cast<float>(t.item().toDouble());
}

void act_quant_impl(const Tensor& x_in, const QuantOpts& o, const OptTensor& smooth, const OptTensor& smooth_rcp, const OptTensor& scale_in,
                    const Scalar* scalars, bool want_codes, bool want_dq, Tensor& codes, Tensor& scale, Tensor& dq, QuantCall* later = nullptr) {
  const at::Device dev = require_cuda({&x_in, ptr_of(smooth), ptr_of(scale_in)});
  if (x_in.dim() != 2) raise("act_quant takes a 2-D tensor");
  if (!is_float(x_in.scalar_type())) raise("unsupported activation dtype");
  const c10::cuda::CUDAGuard guard(dev);
  const Tensor x = x_in.stride(1) != 1 ? x_in.contiguous() : x_in;
  const int64_t rows = x.size(0), cols = x.size(1);
  at::ScalarType ct = at::kChar;
  if (o.mode == QLIN_Q_F8_DYN || (o.mode == QLIN_Q_F8_TENSOR && !o.f8_e5m2)) {
    ct = at::kFloat8_e4m3fn;
  } else if (o.mode == QLIN_Q_F8_TENSOR) {
    ct = at::kFloat8_e5m2;
  }
  // codes that a GEMM reads next get rows of a multiple of 16 bytes
  const int64_t ldq = later != nullptr ? (cols + 15) / 16 * 16 : cols;
  if (want_codes) codes = ldq == cols ? empty({rows, cols}, ct, dev) : empty({rows, ldq}, ct, dev).narrow(1, 0, cols);
  if (want_dq) dq = empty({rows, cols}, x.scalar_type(), dev);
  scale = empty({rows}, at::kFloat, dev);
  const Tensor sm = f32(smooth);
  if (sm.defined() && sm.numel() != cols) raise("smooth must have one entry per column");
  const Tensor rsm = sm.defined() && !o.smooth_mul ? f32(smooth_rcp) : Tensor();
  const Tensor si = f32(scale_in);
  if (rows == 0 || cols == 0) return;
  QuantCall now;
  QuantCall& call = later != nullptr ? *later : now;
  qlin_quant_args& q = call.args;
  q.x = data(x);
  q.smooth = static_cast<const float*>(data(sm));
  q.smooth_rcp = static_cast<const float*>(data(rsm));
  q.scale_in = static_cast<const float*>(data(si));
  q.codes = data(codes);
  q.scale_out = static_cast<float*>(data(scale));
  q.dq_out = data(dq);
  q.status = static_cast<int32_t*>(status_word(dev.index()).data_ptr());
  q.ldx = x.stride(0);
  q.ldq = ldq;
  q.lddq = cols;
  q.rows = static_cast<int32_t>(rows);
  q.cols = static_cast<int32_t>(cols);
  q.x_dtype = dtype_code(x.scalar_type());
  q.mode = o.mode;
  q.native_chain = o.native_chain;
  q.smooth_mul = o.smooth_mul;
  q.clamp_codes = o.clamp_codes;
  q.qmax_levels = o.levels;
  q.dl8_flush = o.dl8_flush;
  q.scale_in_stride = si.defined() && si.numel() != 1 ? 1 : 0;
  const bool st = is_static(o.mode);
  q.scale0 = scalar(scalars[0], dev, st, call.src[0], call.any_src);
  q.zp0 = scalar(scalars[1], dev, st, call.src[1], call.any_src);
  q.lo = scalar(scalars[2], dev, st, call.src[2], call.any_src);
  q.hi = scalar(scalars[3], dev, st, call.src[3], call.any_src);
  q.shift = o.shift;
  q.add2 = o.add2;
  q.dyn_eps = o.dyn_eps;
  q.f8_format = o.f8_e5m2;
  if (later != nullptr) {
    later->keep = {x, sm, rsm, si};
    return;
  }
  check(call.any_src ? qlin_act_quant_static(&q, call.src, stream_of(dev)) : qlin_act_quant(&q, stream_of(dev)), "qlin_act_quant");
}

OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }

std::tuple<OptTensor, Tensor, OptTensor> act_quant(const Tensor& x, int mode, const OptTensor& smooth, const OptTensor& smooth_rcp, bool smooth_mul,
                                                   int native_chain, bool clamp_codes, int levels, bool want_codes, bool want_dq, const OptTensor& scale_in,
                                                   bool dl8_flush, const Scalar& scale0, const Scalar& zp0, const Scalar& lo, const Scalar& hi, double shift,
                                                   double add2, double dyn_eps, bool f8_e5m2) {
  const QuantOpts o{mode,      native_chain, smooth_mul, clamp_codes, levels, dl8_flush, f8_e5m2, static_cast<float>(shift), static_cast<float>(add2),
                    static_cast<float>(dyn_eps)};
  const Scalar scalars[4] = {scale0, zp0, lo, hi};
  Tensor codes, scale, dq;
  act_quant_impl(x, o, smooth, smooth_rcp, scale_in, scalars, want_codes, want_dq, codes, scale, dq);
  return {opt(codes), scale, opt(dq)};
}

// Quantises the rows of x [.., K] and multiplies them with weight [N, K]: the two launches of a deploy-time Linear in one
// call.  row_scale: the scales to dequantise with (none: the ones the quantiser found per row).
Tensor quant_gemm(const Tensor& x, int mode, const OptTensor& smooth, const OptTensor& smooth_rcp, int native_chain, int levels, bool dl8_flush,
                  const Scalar& scale0, const Scalar& zp0, const Scalar& lo, const Scalar& hi, double shift, double add2, const Tensor& weight,
                  const OptTensor& row_scale, const OptTensor& col_scale, const OptTensor& bias, int64_t chunk_k, int trun_bits, int max_acc_bits,
                  bool clamp_dl16, int epilogue, int prod_round, int scale_round, int mid_round, int acc_round, int64_t max_ctas, int out_code) {
  const QuantOpts o{mode, native_chain, 0, 0, levels, dl8_flush, 0, static_cast<float>(shift), static_cast<float>(add2), 1e-5f};
  const Scalar scalars[4] = {scale0, zp0, lo, hi};
  Tensor codes, scale, dq;
  const Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
  QuantCall quant;
  act_quant_impl(x2, o, smooth, smooth_rcp, std::nullopt, scalars, true, false, codes, scale, dq, &quant);
  const Chain ch{chunk_k, trun_bits, max_acc_bits, 1, clamp_dl16, epilogue, prod_round, scale_round, mid_round, acc_round};
  Tensor out = gemm_impl(codes, weight, std::nullopt, std::nullopt, ch, row_scale ? row_scale : OptTensor(scale), col_scale, bias, nullptr, max_ctas, out_code, &quant);
  if (x.dim() == 2) return out;
  std::vector<int64_t> shape = x.sizes().vec();
  shape.back() = weight.size(0);
  return out.reshape(shape);
}

// ------------------------------------------------------------------------------------------------ per-tensor FP8
// Partial maxima of |x| over a dense tensor.
Tensor absmax_parts(const Tensor& x_in) {
  const at::Device dev = require_cuda({&x_in});
  if (!is_float(x_in.scalar_type())) raise("unsupported dtype");
  const c10::cuda::CUDAGuard guard(dev);
  const Tensor x = x_in.contiguous();
  const Tensor parts = empty({qlin_absmax_parts_count(x.numel())}, at::kFloat, dev);
  check(qlin_absmax_parts(data(x), x.numel(), dtype_code(x.scalar_type()), static_cast<float*>(data(parts)), stream_of(dev)), "qlin_absmax_parts");
  return parts;
}

// Codes [rows, cols] and / or [cols, rows] with rows of a multiple of 16 bytes, the scale [1] and, optionally, the column sums.
std::tuple<OptTensor, OptTensor, Tensor, OptTensor> f8_tensor_quant(const Tensor& x_in, const Tensor& parts, bool e5m2, double eps, bool dl8_flush,
                                                                    bool want_codes, bool want_t, bool want_colsum) {
  const at::Device dev = require_cuda({&x_in, &parts});
  if (x_in.dim() != 2) raise("f8_tensor_quant takes a 2-D tensor");
  if (!is_float(x_in.scalar_type())) raise("unsupported activation dtype");
  const c10::cuda::CUDAGuard guard(dev);
  const Tensor x = x_in.contiguous();
  const int64_t rows = x.size(0), cols = x.size(1);
  const at::ScalarType ct = e5m2 ? at::kFloat8_e5m2 : at::kFloat8_e4m3fn;
  Tensor codes, codes_t, colsum, ws;
  const int64_t ldq = (cols + 15) / 16 * 16, ldt = (rows + 15) / 16 * 16;
  if (want_codes) codes = ldq == cols ? empty({rows, cols}, ct, dev) : empty({rows, ldq}, ct, dev).narrow(1, 0, cols);
  if (want_t) codes_t = ldt == rows ? empty({cols, rows}, ct, dev) : empty({cols, ldt}, ct, dev).narrow(1, 0, rows);
  if (want_colsum) {
    colsum = empty({cols}, at::kFloat, dev);
    ws = empty({std::max<int64_t>(1, qlin_f8_tensor_colsum_workspace_bytes(static_cast<int32_t>(rows), static_cast<int32_t>(cols)) / 4)}, at::kFloat, dev);
  }
  const Tensor scale = empty({1}, at::kFloat, dev);
  qlin_f8_tensor_args a = {};
  a.x = data(x);
  a.amax_parts = static_cast<const float*>(data(parts));
  a.nparts = static_cast<int32_t>(parts.numel());
  a.codes = data(codes);
  a.codes_t = data(codes_t);
  a.scale_out = static_cast<float*>(data(scale));
  a.colsum = static_cast<float*>(data(colsum));
  a.workspace = static_cast<float*>(data(ws));
  a.ldx = cols;
  a.ldq = ldq;
  a.ldt = ldt;
  a.rows = static_cast<int32_t>(rows);
  a.cols = static_cast<int32_t>(cols);
  a.x_dtype = dtype_code(x.scalar_type());
  a.f8_format = e5m2;
  a.dl8_flush = dl8_flush;
  a.f8_max = e5m2 ? 57344.0f : 448.0f;
  a.eps = static_cast<float>(eps);
  check(qlin_f8_tensor_quant(&a, stream_of(dev)), "qlin_f8_tensor_quant");
  return {opt(codes), opt(codes_t), scale, opt(colsum)};
}

// ------------------------------------------------------------------------------------------------ PACT+
Tensor clip_f32(const Tensor& t, at::Device dev) {
  Tensor d = t.detach();
  if (d.dim() == 1 && d.numel() == 1 && d.scalar_type() == at::kFloat && d.device() == dev) return d;
  d = d.reshape({-1}).narrow(0, 0, 1);
  if (d.scalar_type() != at::kFloat || d.device() != dev) d = d.to(at::TensorOptions().device(dev).dtype(at::kFloat));
  return d.contiguous();
}

qlin_pact2_args pact_args(const Tensor& x, const Tensor& out, const Tensor& cv, const Tensor& cvn, int num_bits, bool align_zero, int variant) {
  qlin_pact2_args p = {};
  p.x = data(x);
  p.out = data(out);
  p.clip_val = static_cast<const float*>(data(cv));
  p.clip_valn = static_cast<const float*>(data(cvn));
  p.numel = x.numel();
  p.dtype = dtype_code(x.scalar_type());
  p.num_bits = num_bits;
  p.align_zero = align_zero;
  p.variant = variant;
  return p;
}

Tensor pact2_fwd(const Tensor& x_in, const Tensor& clip_val, const OptTensor& clip_valn, int num_bits, bool align_zero, int variant) {
  const at::Device dev = require_cuda({&x_in});
  if (!is_float(x_in.scalar_type())) raise("unsupported dtype");
  const c10::cuda::CUDAGuard guard(dev);
  const Tensor x = x_in.detach().contiguous();
  const Tensor out = at::empty_like(x);
  const Tensor cv = clip_f32(clip_val, dev), cvn = clip_valn ? clip_f32(*clip_valn, dev) : Tensor();
  const qlin_pact2_args p = pact_args(x, out, cv, cvn, num_bits, align_zero, variant);
  check(qlin_pact2_fwd(&p, stream_of(dev)), "qlin_pact2_fwd");
  return out;
}

std::tuple<Tensor, Tensor> pact2_bwd(const Tensor& x_in, const Tensor& grad_out, const Tensor& clip_val, const OptTensor& clip_valn, int num_bits,
                                     bool align_zero, int variant) {
  const at::Device dev = require_cuda({&x_in, &grad_out});
  if (!is_float(x_in.scalar_type())) raise("unsupported dtype");
  const c10::cuda::CUDAGuard guard(dev);
  const Tensor x = x_in.detach().contiguous();
  Tensor g = grad_out.detach().contiguous();
  if (g.scalar_type() != x.scalar_type()) g = g.to(x.scalar_type());
  const Tensor gx = at::empty_like(x);
  const Tensor cv = clip_f32(clip_val, dev), cvn = clip_valn ? clip_f32(*clip_valn, dev) : Tensor();
  const int64_t ws_floats = std::max<int64_t>(1, static_cast<int64_t>(qlin_pact2_bwd_workspace_bytes(x.numel()) / 4));
  const Tensor ws = empty({ws_floats}, at::kFloat, dev), grads = empty({2}, at::kFloat, dev);
  qlin_pact2_args p = pact_args(x, gx, cv, cvn, num_bits, align_zero, variant);
  p.grad_out = data(g);
  p.grad_clip = static_cast<float*>(data(grads));
  p.workspace = data(ws);
  check(qlin_pact2_bwd(&p, stream_of(dev)), "qlin_pact2_bwd");
  return {gx, grads};
}

// ------------------------------------------------------------------------------------------------ per-channel weight quantiser
std::tuple<OptTensor, OptTensor, Tensor> weight_fq_perch(const Tensor& w_in, int num_bits, int mode, const OptTensor& clip, const OptTensor& smooth,
                                                         bool native_mul, int clip_dtype, bool want_dq, bool want_codes, double c0, double c1) {
  const at::Device dev = require_cuda({&w_in, ptr_of(clip), ptr_of(smooth)});
  const c10::cuda::CUDAGuard guard(dev);
  Tensor w = w_in.dim() != 2 ? w_in.reshape({w_in.size(0), -1}) : w_in;
  if (!is_float(w.scalar_type())) raise("unsupported weight dtype");
  if (w.stride(1) != 1) w = w.contiguous();
  const int64_t rows = w.size(0), cols = w.size(1);
  Tensor clip_io;
  if (mode == QLIN_W_GIVEN) {
    if (!clip || clip->numel() != rows) raise("W_GIVEN needs one clip value per row");
    clip_io = f32(clip->detach().reshape({-1})).clone();
  } else {
    clip_io = empty({rows}, at::kFloat, dev);
  }
  Tensor dq, codes;
  if (want_dq) dq = empty({rows, cols}, w.scalar_type(), dev);
  if (want_codes) codes = empty({rows, cols}, at::kChar, dev);
  const Tensor sm = f32(smooth);
  if (rows == 0 || cols == 0) return {opt(dq), opt(codes), clip_io};
  qlin_wfq_args a = {};
  a.w = data(w);
  a.smooth = static_cast<const float*>(data(sm));
  a.dq_out = data(dq);
  a.codes = data(codes);
  a.clip_io = static_cast<float*>(data(clip_io));
  a.ldw = w.stride(0);
  a.ldo = a.ldq = cols;
  a.rows = static_cast<int32_t>(rows);
  a.cols = static_cast<int32_t>(cols);
  a.dtype = dtype_code(w.scalar_type());
  a.num_bits = num_bits;
  a.mode = mode;
  a.native_mul = native_mul;
  a.clip_dtype = clip_dtype;
  a.c0 = static_cast<float>(c0);
  a.c1 = static_cast<float>(c1);
  check(qlin_weight_fq_perch(&a, stream_of(dev)), "qlin_weight_fq_perch");
  return {opt(dq), opt(codes), clip_io};
}

// ------------------------------------------------------------------------------------------------ QAT Linear
// out = x w^T + bias for fake-quantised fp32 operands on the tensor cores (qlin_qat_*), with its gradients.
struct QatShape {
  int64_t tokens, in, out;
};

// The operands' arguments of one pass; `floats` is [out + 2]: scales, the step and its clip value.
qlin_qat_args qat_args(const Tensor& x, const Tensor& w, const Tensor& floats, const Tensor& flags, const QatShape& n) {
  qlin_qat_args a = {};
  a.x = static_cast<const float*>(data(x));
  a.w = static_cast<const float*>(data(w));
  a.scale = static_cast<float*>(data(floats));
  a.step = a.scale + n.out;
  a.clip_kept = a.step + 1;
  a.flags = static_cast<int32_t*>(data(flags));
  a.status = static_cast<int32_t*>(status_word(x.device().index()).data_ptr());
  a.tokens = static_cast<int32_t>(n.tokens);
  a.in = static_cast<int32_t>(n.in);
  a.out = static_cast<int32_t>(n.out);
  return a;
}

// What the kernels can read: fp32 memory on the device that holds the values as they are, and nothing at work that has to see operators.
bool plain(const Tensor& g, const at::Device& dev) {
  const c10::DispatchKeySet seen({c10::DispatchKey::Python, c10::DispatchKey::Functionalize, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                  c10::DispatchKey::Batched, c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
  return g.device() == dev && g.layout() == at::kStrided && g.scalar_type() == at::kFloat && g.has_storage() && !g.key_set().has_any(seen) &&
         !c10::impl::TorchDispatchModeTLS::any_modes_set() && !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

// The same, dense and aligned, for operands: hooks on saved tensors may bring them back with other strides, from another address or device.
bool plain_operand(const Tensor& t, const at::Device& dev) {
  return plain(t, dev) && t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

class QatProduct : public torch::autograd::Function<QatProduct> {
 public:
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& bias, const Tensor& clip_x,
                        const OptTensor& clipn_x, const Tensor& clip_w, int64_t bits_x, int64_t bits_w, int64_t variant) {
    const at::Device dev = x.device();
    const c10::cuda::CUDAGuard guard(dev);
    const QatShape n{x.numel() / x.size(-1), x.size(-1), w.size(0)};
    const Tensor floats = empty({n.out + 2}, at::kFloat, dev), flags = empty({qlin_qat_flag_count()}, at::kInt, dev);
    const Tensor xc = empty({n.tokens, n.in}, at::kBFloat16, dev), wc = empty({n.out, n.in}, at::kBFloat16, dev);
    std::vector<int64_t> shape = x.sizes().vec();
    shape.back() = n.out;
    const Tensor out = empty(shape, at::kFloat, dev);
    const Tensor bs = bias ? bias->detach().contiguous() : Tensor(), cv = clip_f32(clip_x, dev), cvn = clipn_x ? clip_f32(*clipn_x, dev) : Tensor();
    const Tensor cw = clip_w.detach().contiguous();
    qlin_qat_args a = qat_args(x, w, floats, flags, n);
    a.bias = static_cast<const float*>(data(bs));
    a.clip_x = static_cast<const float*>(data(cv));
    a.clipn_x = static_cast<const float*>(data(cvn));
    a.clip_w = static_cast<const float*>(data(cw));
    a.x_codes = data(xc);
    a.w_codes = data(wc);
    a.d = static_cast<float*>(data(out));
    a.num_bits_x = static_cast<int32_t>(bits_x);
    a.num_bits_w = static_cast<int32_t>(bits_w);
    a.variant = static_cast<int32_t>(variant);
    check(qlin_qat_codes(&a, 0, stream_of(dev)), "qlin_qat_codes");
    check(qlin_qat_product(&a, 0, stream_of(dev)), "qlin_qat_product");
    // the step and scales are kept, not the clip values they came from: a later forward pass may have replaced those
    ctx->save_for_backward({x, w, floats});
    ctx->saved_data["bits"] = std::vector<int64_t>{bits_x, bits_w, variant};
    ctx->saved_data["bias"] = bias.has_value();
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const torch::autograd::variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &floats = saved[2];
    const QatShape n{x.numel() / x.size(-1), x.size(-1), w.size(0)};
    const bool want_x = ctx->needs_input_grad(0), want_w = ctx->needs_input_grad(1);
    const bool want_b = ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(2);
    Tensor gx, gw, gb;
    const Tensor& go = grads[0];
    if (go.defined()) {
      const Tensor g = go.reshape({n.tokens, n.out});
      const at::Device dev = go.device();
      // gradients that are differentiated again, that are batched, or that a mode or a subclass follows
      if (at::GradMode::is_enabled() || !plain(g, dev) || !plain_operand(x, dev) || !plain_operand(w, dev) || !plain_operand(floats, dev)) {
        if (want_x) gx = g.matmul(w).reshape(x.sizes());
        if (want_w) gw = g.t().matmul(x.reshape({n.tokens, n.in}));
      } else if (want_x || want_w) {
        const c10::cuda::CUDAGuard guard(dev);
        const Tensor gc = g.contiguous(), flags = empty({qlin_qat_flag_count()}, at::kInt, dev);
        const std::vector<int64_t> bits = ctx->saved_data["bits"].toIntVector();
        const Tensor planes = empty({3, n.tokens, n.out}, at::kBFloat16, dev), rcp = empty({n.out}, at::kFloat, dev);
        // both operands' codes are made, and checked, whichever gradient is wanted
        Tensor xc = empty({n.tokens, n.in}, at::kBFloat16, dev), wc = empty({n.in, n.out}, at::kBFloat16, dev);
        qlin_qat_args a = qat_args(x, w, floats, flags, n);
        a.g = static_cast<const float*>(data(gc));
        a.x_codes = data(xc);
        a.w_codes = data(wc);
        a.g_planes = data(planes);
        a.rcp = static_cast<float*>(data(rcp));
        a.num_bits_x = static_cast<int32_t>(bits[0]);
        a.num_bits_w = static_cast<int32_t>(bits[1]);
        a.variant = static_cast<int32_t>(bits[2]);
        Tensor ws;
        if (want_b) {
          gb = empty({n.out}, at::kFloat, dev);
          ws = empty({qlin_qat_colsum_workspace_bytes(a.tokens, a.out) / 4}, at::kFloat, dev);
          a.colsum = static_cast<float*>(data(gb));
          a.workspace = static_cast<float*>(data(ws));
        }
        check(qlin_qat_codes(&a, 1, stream_of(dev)), "qlin_qat_codes");
        check(qlin_qat_split(&a, stream_of(dev)), "qlin_qat_split");
        if (want_w) {
          gw = empty({n.out, n.in}, at::kFloat, dev);
          a.d = static_cast<float*>(data(gw));
          check(qlin_qat_product(&a, 2, stream_of(dev)), "qlin_qat_product");
        }
        xc.reset();
        if (want_x) {
          gx = empty(x.sizes(), at::kFloat, dev);
          a.d = static_cast<float*>(data(gx));
          a.x_codes = nullptr;
          check(qlin_qat_product(&a, 1, stream_of(dev)), "qlin_qat_product");
        }
      }
      if (want_b && !gb.defined()) gb = g.sum(0);
    }
    return {gx, gw, gb, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// Calls with fewer multiply-adds than this, or with a side shorter than 128, stay with the library.  Device time of forward and
// backward, library -> tensor cores: 256 x 768 x 768 (2^27.2) 65 -> 67 us, 700 x 768 x 768 (2^28.6) 95 -> 73, 256 x 768 x 3072
// (2^29.2) 159 -> 101, 4096 x 768 x 768 364 -> 135.
constexpr double kQatMinWork = 268435456.0;
constexpr int64_t kQatMinSide = 128;

// Whether qat_linear takes these operands: fp32 in fp32 arithmetic (no TF32, no autocast), dense, aligned, and large enough.
bool qat_takes(const Tensor& x, const Tensor& w, const OptTensor& bias, const Tensor& clip_w) {
  if (!x.is_cuda() || x.scalar_type() != at::kFloat || w.scalar_type() != at::kFloat || w.device() != x.device() || w.dim() != 2 || x.dim() < 1) return false;
  if (x.size(-1) != w.size(1) || !x.is_contiguous() || !w.is_contiguous() || x.layout() != at::kStrided || w.layout() != at::kStrided) return false;
  if (bias && (bias->scalar_type() != at::kFloat || bias->device() != x.device() || bias->dim() != 1 || bias->size(0) != w.size(0))) return false;
  if (clip_w.scalar_type() != at::kFloat || clip_w.device() != x.device() || clip_w.numel() != w.size(0)) return false;
  const int64_t in = w.size(1), out = w.size(0);
  if (in < kQatMinSide || out < kQatMinSide || x.numel() < kQatMinSide * in || in % 8 != 0 || out % 8 != 0 || x.numel() / in > 0x7fffffff - 256 || in > 0x7fffff00 || out > qlin_qat_max_out()) return false;
  if (!plain_operand(x, x.device()) || !plain_operand(w, x.device()) || (bias && !plain(*bias, x.device()))) return false;
  if (at::autocast::is_autocast_enabled(at::kCUDA)) return false;
  const at::Float32Precision prec = at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL);
  if (prec != at::Float32Precision::NONE && prec != at::Float32Precision::IEEE) return false;
  return static_cast<double>(x.numel()) * static_cast<double>(out) >= kQatMinWork;
}

Tensor qat_linear(const Tensor& x, const Tensor& w, const OptTensor& bias, const Tensor& clip_x, const OptTensor& clipn_x, const Tensor& clip_w, int64_t bits_x,
                  int64_t bits_w, int64_t variant) {
  return QatProduct::apply(x, w, bias, clip_x.detach(), clipn_x ? OptTensor(clipn_x->detach()) : std::nullopt, clip_w, bits_x, bits_w, variant);
}

}  // namespace

PYBIND11_MODULE(_qlin_host, m) {
  using rel = py::call_guard<py::gil_scoped_release>;
  m.def("status_word", &status_word, rel());
  m.def("gemm", &gemm, rel());
  m.def("act_quant", &act_quant, rel());
  m.def("quant_gemm", &quant_gemm, rel());
  m.def("absmax_parts", &absmax_parts, rel());
  m.def("f8_tensor_quant", &f8_tensor_quant, rel());
  m.def("weight_fq_perch", &weight_fq_perch, rel());
  m.def("pact2_fwd", &pact2_fwd, rel());
  m.def("pact2_bwd", &pact2_bwd, rel());
  m.def("qat_takes", &qat_takes, rel());
  m.def("qat_linear", &qat_linear, rel());
}
