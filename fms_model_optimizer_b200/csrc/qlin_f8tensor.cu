// qlin_f8_tensor_quant: one FP8 scale for a whole tensor (the per-tensor branch of the FP8 Linear), with the codes written
// row-major, transposed, or both from one read of the tensor, and optionally the column sums of the codes.
//
// Two launches: qlin_absmax_parts reduces |x| to at most kAbsParts partial maxima, and every block of the quantise kernel
// reduces those to the tensor's maximum before its first tile (no one-block kernel in between).  A backward pass needs the
// codes of the gradient both ways, those of x and W transposed, and the column sums of the gradient's codes; both GEMM
// operands are K-major.
//
// Bound by HBM and, at a few tiles a block, by the latency of a tile: s bytes read and one or two bytes written per element.  The
// resident blocks walk over 128 x 64 tiles; a thread quantises two 16-element slices and loads each slice of its next tile as soon
// as it has used this one's (the first tile's before the maximum is known); the transposed copy goes through a swizzled
// shared tile of 4-byte words, read back as 8 rows x 4 columns per thread and turned with byte permutes, so both outputs are
// written in runs of 64 and 128 bytes.
//
// Codes, or codes both ways, L2 flushed, before (half as many blocks again as fit, no load ahead, four-way conflicts in the
// stores to shared memory) and after: 4096 x 4096 bf16 22.5 -> 18.4 and 24.6 -> 20.5 us, 8192 x 8192 bf16 63.5 -> 43.0 and
// 79.9 -> 53.3 (5.0 TB/s), fp32 71.7 -> 65.6 and 88.1 -> 77.9.
#include <type_traits>

#include <cuda_fp8.h>

#include "qlin_internal.h"
#include "qlin_rows.cuh"

namespace qlin {

constexpr int kAbsThreads = 512;
constexpr int kAbsParts = 296;  // two blocks per SM
constexpr int kF8Threads = 256;
constexpr int kF8TileM = 128, kF8TileN = 64;

template <typename XT>
__global__ void __launch_bounds__(kAbsThreads) absmax_parts_kernel(const XT* x, int64_t numel, float* parts) {
  __shared__ float red[32];
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  const int64_t nvec = vec ? numel >> 4 : 0;
  const int64_t first = static_cast<int64_t>(blockIdx.x) * kAbsThreads + threadIdx.x, stride = static_cast<int64_t>(gridDim.x) * kAbsThreads;
  float am = 0.0f;
  int64_t i = first;
  for (; i + stride < nvec; i += 2 * stride) {  // two slices in flight
    float a[16], b[16];
    load16(x + i * 16, a);
    load16(x + (i + stride) * 16, b);
#pragma unroll
    for (int j = 0; j < 16; ++j) am = fmaxf(am, fmaxf(fabsf(a[j]), fabsf(b[j])));
  }
  if (i < nvec) {
    float a[16];
    load16(x + i * 16, a);
#pragma unroll
    for (int j = 0; j < 16; ++j) am = fmaxf(am, fabsf(a[j]));
  }
  for (i = nvec * 16 + first; i < numel; i += stride) am = fmaxf(am, fabsf(load1(x + i)));
  am = block_reduce<OpMax>(am, red, 0.0f);
  if (threadIdx.x == 0) parts[blockIdx.x] = am;
}

struct F8TensorParams {
  const void* x;
  const float* parts;
  uint8_t* codes;
  uint8_t* codes_t;
  float* scale_out;
  float* colsum_ws;  // [row tiles][cols]
  int64_t ldx, ldq, ldt;
  int32_t rows, cols, nparts, e5m2, dl8_flush;
  float f8_max, eps;
};

// fp32 -> fp8 as torch converts: e4m3 NaN above 464, e5m2 infinity from 61440.
__device__ __forceinline__ uint8_t f8_scalar(float v, bool e5m2) {
  if (e5m2) {
    if (v != v) return 0x7F;
    return static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_NOSAT, __NV_E5M2));
  }
  if (!(fabsf(v) <= 464.0f)) return static_cast<uint8_t>(0x7F | (signbit(v) ? 0x80 : 0));
  return static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
}
__device__ __forceinline__ uint32_t f8_pair(float lo, float hi, bool e5m2) {
  uint16_t r;
  if (e5m2) {
    asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  } else {
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  }
  return r;
}

// Sixteen values -> sixteen codes.  `fast`: the scale lies in [1e-15, 1e15], so no quotient exceeds the format's largest value
// by more than the rounding of the scale (448 -> 450, 57344 -> 57600; both convert to the largest value, saturating or not).
// bf16: x * RN(1 / s) rounded to bf16 is the rounded quotient (see qlin_quant.cu).  fp32: the exact quotient from three fused
// operations, with the sign of a zero put back.  fp16 rows, whose scale may be a coarse subnormal, convert one by one.
template <typename XT>
__device__ __forceinline__ void f8_codes16(const float (&v)[16], float s, float rs, bool fast, bool e5m2, bool flush, uint32_t (&w)[4]) {
  constexpr bool kBf16 = std::is_same<XT, __nv_bfloat16>::value, kF32 = std::is_same<XT, float>::value;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    if ((kBf16 || kF32) && fast) {
      float t[4];
#pragma unroll
      for (int k = 0; k < 4; k += 2) {
        const float a = v[4 * g + k], b = v[4 * g + k + 1];
        if (kBf16) {
          const __nv_bfloat162 h = __float22bfloat162_rn(__fmul2_rn(make_float2(a, b), make_float2(rs, rs)));
          const uint32_t hw = *reinterpret_cast<const uint32_t*>(&h);
          t[k] = __uint_as_float(hw << 16);
          t[k + 1] = __uint_as_float(hw & 0xFFFF0000u);
        } else {
          const float qa = __fmul_rn(a, rs), qb = __fmul_rn(b, rs);
          t[k] = copysignf(__fmaf_rn(__fmaf_rn(-s, qa, a), rs, qa), a);
          t[k + 1] = copysignf(__fmaf_rn(__fmaf_rn(-s, qb, b), rs, qb), b);
        }
      }
      w[g] = f8_pair(t[0], t[1], e5m2) | (f8_pair(t[2], t[3], e5m2) << 16);
    } else {
      w[g] = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        w[g] |= static_cast<uint32_t>(f8_scalar(Elem<XT>::rnd(__fdiv_rn(v[4 * g + k], s)), e5m2)) << (8 * k);
    }
    if (flush) {  // values below 0.0087890625 become 0: e4m3 codes up to 4 (4 * 2^-9), e5m2 codes up to 32 (2^-7)
      const uint32_t top = e5m2 ? 32u : 4u;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (((w[g] >> (8 * k)) & 0x7Fu) <= top) w[g] &= ~(0xFFu << (8 * k));
    }
  }
}

// 4 x 4 bytes: word i holds row i; out[k] holds column k.
__device__ __forceinline__ void transpose4(const uint32_t (&a)[4], uint32_t (&out)[4]) {
  const uint32_t t0 = __byte_perm(a[0], a[1], 0x5140), t1 = __byte_perm(a[2], a[3], 0x5140);
  const uint32_t t2 = __byte_perm(a[0], a[1], 0x7362), t3 = __byte_perm(a[2], a[3], 0x7362);
  out[0] = __byte_perm(t0, t1, 0x5410);
  out[1] = __byte_perm(t0, t1, 0x7632);
  out[2] = __byte_perm(t2, t3, 0x5410);
  out[3] = __byte_perm(t2, t3, 0x7632);
}

// Sixteen elements as they lie in memory.
template <typename XT>
struct F8Raw {
  static constexpr int kWords = 4 * static_cast<int>(sizeof(XT));
  uint32_t w[kWords];
};
__device__ __forceinline__ uint32_t f8_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t f8_bits(__half v) { return __half_as_ushort(v); }
__device__ __forceinline__ uint32_t f8_bits(__nv_bfloat16 v) { return __bfloat16_as_ushort(v); }

// Columns col .. col + 15 of `row`, zeros outside the tensor.
template <typename XT>
__device__ __forceinline__ void f8_fetch(const F8TensorParams& p, bool vec, int row, int col, F8Raw<XT>& raw) {
  constexpr int kPer = 4 / static_cast<int>(sizeof(XT));  // elements a word
  const XT* src = reinterpret_cast<const XT*>(p.x) + static_cast<int64_t>(row) * p.ldx + col;
  if (row < p.rows && vec && col + 16 <= p.cols) {
#pragma unroll
    for (int i = 0; i < F8Raw<XT>::kWords / 4; ++i) {
      const uint4 q = reinterpret_cast<const uint4*>(src)[i];
      raw.w[4 * i] = q.x, raw.w[4 * i + 1] = q.y, raw.w[4 * i + 2] = q.z, raw.w[4 * i + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < F8Raw<XT>::kWords; ++i) raw.w[i] = 0u;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (row < p.rows && col + j < p.cols) raw.w[j / kPer] |= f8_bits(src[j]) << (16 * (j % kPer));
  }
}
__device__ __forceinline__ void f8_widen(const F8Raw<float>& r, float (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r.w[j]);
}
__device__ __forceinline__ void f8_widen(const F8Raw<__half>& r, float (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&r.w[j]));
    v[2 * j] = f.x, v[2 * j + 1] = f.y;
  }
}
__device__ __forceinline__ void f8_widen(const F8Raw<__nv_bfloat16>& r, float (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) v[2 * j] = __uint_as_float(r.w[j] << 16), v[2 * j + 1] = __uint_as_float(r.w[j] & 0xFFFF0000u);
}

// Resident blocks an SM; a block walks over its tiles, and each slice of the next one is loaded as soon as this tile's is used up.
template <typename XT>
constexpr int f8_resident() { return sizeof(XT) == 4 ? 3 : 4; }

template <typename XT>
__global__ void __launch_bounds__(kF8Threads, f8_resident<XT>()) f8_tensor_quant_kernel(const F8TensorParams p) {
  __shared__ uint32_t tile[kF8TileM * (kF8TileN / 4)];  // word (row, c4) at row * 16 + (c4 ^ (row / 8) ^ (row / 2 % 4)): stores without conflicts, loads two-way
  __shared__ float red[32];
  const int tiles_n = (p.cols + kF8TileN - 1) / kF8TileN, tiles_m = (p.rows + kF8TileM - 1) / kF8TileM;
  const int64_t tiles = static_cast<int64_t>(tiles_m) * tiles_n;
  const bool vec_x = (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0 && (p.ldx * static_cast<int64_t>(sizeof(XT))) % 16 == 0;
  F8Raw<XT> raw[2];
  const auto fetch = [&](int64_t t, int h) {
    const int id = threadIdx.x + h * kF8Threads;
    f8_fetch(p, vec_x, static_cast<int>(t / tiles_n) * kF8TileM + (id >> 2), static_cast<int>(t % tiles_n) * kF8TileN + (id & 3) * 16, raw[h]);
  };
  fetch(blockIdx.x, 0);  // under way while the maximum is found; the grid has no more blocks than tiles
  fetch(blockIdx.x, 1);
  float am = 0.0f;
  for (int i = threadIdx.x; i < p.nparts; i += kF8Threads) am = fmaxf(am, p.parts[i]);
  am = block_reduce<OpMax>(am, red, 0.0f);
  const float s = fmaxf(Elem<XT>::rnd(__fdiv_rn(am, p.f8_max)), Elem<XT>::rnd(p.eps));
  if (blockIdx.x == 0 && threadIdx.x == 0 && p.scale_out != nullptr) *p.scale_out = s;
  const float rs = rcp_for_div(s);
  const bool fast = rs == rs;
  const bool e5m2 = p.e5m2 != 0, flush = p.dl8_flush != 0;
  const bool vec_q = (reinterpret_cast<uintptr_t>(p.codes) & 15u) == 0 && p.ldq % 16 == 0;
  const bool turn = p.codes_t != nullptr || p.colsum_ws != nullptr;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int tm = static_cast<int>(t / tiles_n), tn = static_cast<int>(t % tiles_n);
    const int row0 = tm * kF8TileM, col0 = tn * kF8TileN;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int id = threadIdx.x + h * kF8Threads;
      const int r = id >> 2, row = row0 + r, col = col0 + (id & 3) * 16;
      float v[16];
      f8_widen(raw[h], v);
      if (t + gridDim.x < tiles) fetch(t + gridDim.x, h);
      uint32_t w[4];
      f8_codes16<XT>(v, s, rs, fast, e5m2, flush, w);
      if (row >= p.rows || col >= p.cols) {  // padding of the transposed rows: zeros (a zero scale makes NaN of 0 / s)
#pragma unroll
        for (int g = 0; g < 4; ++g) w[g] = 0u;
      }
      if (p.codes != nullptr && row < p.rows && col < p.cols) {
        uint8_t* dst = p.codes + static_cast<int64_t>(row) * p.ldq + col;
        if (vec_q && col + 16 <= p.cols) {
          *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (col + j < p.cols) dst[j] = static_cast<uint8_t>(w[j >> 2] >> (8 * (j & 3)));
        }
      }
      if (turn) {
#pragma unroll
        for (int g = 0; g < 4; ++g) tile[r * 16 + ((((id & 3) * 4) + g) ^ (r >> 3) ^ ((r >> 1) & 3))] = w[g];
      }
    }
    if (!turn) continue;
    __syncthreads();
    const int rg = threadIdx.x & 15, c4 = threadIdx.x >> 4;  // eight rows, four columns
    uint32_t a[4], b[4], lo[4], hi[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = tile[(rg * 8 + i) * 16 + (c4 ^ rg ^ (i >> 1))];
      b[i] = tile[(rg * 8 + 4 + i) * 16 + (c4 ^ rg ^ (2 + (i >> 1)))];
    }
    transpose4(a, lo);
    transpose4(b, hi);
    if (p.codes_t != nullptr && row0 + rg * 8 < p.ldt) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int col = col0 + c4 * 4 + k;
        if (col < p.cols) *reinterpret_cast<uint2*>(p.codes_t + static_cast<int64_t>(col) * p.ldt + row0 + rg * 8) = make_uint2(lo[k], hi[k]);
      }
    }
    if (p.colsum_ws != nullptr) {  // e5m2: a code is the upper byte of an fp16 number
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t word = i == 0 ? lo[k] : hi[k];
          const uint32_t h0 = __byte_perm(word, 0u, 0x1404), h1 = __byte_perm(word, 0u, 0x3424);
          const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&h0)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&h1));
          sum += (f0.x + f0.y) + (f1.x + f1.y);
        }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const int col = col0 + c4 * 4 + k;
        if (rg == 0 && col < p.cols) p.colsum_ws[static_cast<int64_t>(tm) * p.cols + col] = sum;
      }
    }
    __syncthreads();
  }
}

// Adds the row tiles' column sums in order.
__global__ void __launch_bounds__(256) f8_colsum_finish_kernel(const float* ws, int tiles_m, int cols, float* colsum) {
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= cols) return;
  float sum = 0.0f;
  for (int i = 0; i < tiles_m; ++i) sum += ws[static_cast<int64_t>(i) * cols + c];
  colsum[c] = sum;
}

static int abs_parts(int64_t numel) {
  const int64_t want = (numel + kAbsThreads * 16 - 1) / (kAbsThreads * 16);
  return static_cast<int>(want < 1 ? 1 : (want > kAbsParts ? kAbsParts : want));
}

template <typename XT>
static int launch_f8_tensor(const F8TensorParams& p, cudaStream_t stream) {
  const int64_t tiles = static_cast<int64_t>((p.rows + kF8TileM - 1) / kF8TileM) * ((p.cols + kF8TileN - 1) / kF8TileN);
  const int64_t cap = static_cast<int64_t>(sm_count()) * f8_resident<XT>();
  f8_tensor_quant_kernel<XT><<<static_cast<int>(tiles < cap ? tiles : cap), kF8Threads, 0, stream>>>(p);
  QLIN_CHECK_LAUNCH("qlin_f8_tensor_quant");
  return QLIN_OK;
}

}  // namespace qlin

using namespace qlin;

extern "C" int32_t qlin_absmax_parts_count(int64_t numel) { return abs_parts(numel); }

extern "C" int qlin_absmax_parts(const void* x, int64_t numel, int32_t dtype, float* parts, void* stream) {
  if (numel < 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_absmax_parts: negative numel");
  if ((x == nullptr && numel > 0) || parts == nullptr) return fail(QLIN_ERR_NULL, "qlin_absmax_parts: x or parts is NULL");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int grid = abs_parts(numel);
  switch (dtype) {
    case QLIN_DT_F32:
      absmax_parts_kernel<float><<<grid, kAbsThreads, 0, s>>>(static_cast<const float*>(x), numel, parts);
      break;
    case QLIN_DT_F16:
      absmax_parts_kernel<__half><<<grid, kAbsThreads, 0, s>>>(static_cast<const __half*>(x), numel, parts);
      break;
    case QLIN_DT_BF16:
      absmax_parts_kernel<__nv_bfloat16><<<grid, kAbsThreads, 0, s>>>(static_cast<const __nv_bfloat16*>(x), numel, parts);
      break;
    default:
      return fail(QLIN_ERR_BAD_DTYPE, "qlin_absmax_parts: dtype must be F32, F16 or BF16");
  }
  QLIN_CHECK_LAUNCH("qlin_absmax_parts");
  return QLIN_OK;
}

extern "C" int64_t qlin_f8_tensor_colsum_workspace_bytes(int32_t rows, int32_t cols) {
  return static_cast<int64_t>((rows + kF8TileM - 1) / kF8TileM) * cols * static_cast<int64_t>(sizeof(float));
}

extern "C" int qlin_f8_tensor_quant(const qlin_f8_tensor_args* a, void* stream) {
  if (a == nullptr) return fail(QLIN_ERR_NULL, "qlin_f8_tensor_quant: args is NULL");
  if (a->rows < 0 || a->cols < 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_f8_tensor_quant: negative dimension");
  if (a->amax_parts == nullptr || a->nparts < 1) return fail(QLIN_ERR_NULL, "qlin_f8_tensor_quant: amax_parts is NULL");
  if (a->codes == nullptr && a->codes_t == nullptr && a->colsum == nullptr) return fail(QLIN_ERR_NULL, "qlin_f8_tensor_quant: no output requested");
  if (!(a->f8_max > 0.0f)) return fail(QLIN_ERR_UNSUPPORTED, "qlin_f8_tensor_quant: f8_max must be positive");
  if (a->rows == 0 || a->cols == 0) return QLIN_OK;
  if (a->x == nullptr) return fail(QLIN_ERR_NULL, "qlin_f8_tensor_quant: x is NULL");
  if (a->ldx < a->cols || (a->codes != nullptr && a->ldq < a->cols)) return fail(QLIN_ERR_BAD_SHAPE, "qlin_f8_tensor_quant: leading dimension smaller than the row length");
  if (a->codes_t != nullptr && (a->ldt < a->rows || a->ldt % 16 != 0 || !aligned16(a->codes_t)))
    return fail(QLIN_ERR_BAD_ALIGN, "qlin_f8_tensor_quant: codes_t must be 16-byte aligned with ldt >= rows a multiple of 16");
  if (a->colsum != nullptr && (a->f8_format != 1 || a->workspace == nullptr))
    return fail(QLIN_ERR_UNSUPPORTED, "qlin_f8_tensor_quant: column sums need e5m2 codes and a workspace");
  F8TensorParams p;
  p.x = a->x;
  p.parts = a->amax_parts;
  p.nparts = a->nparts;
  p.codes = static_cast<uint8_t*>(a->codes);
  p.codes_t = static_cast<uint8_t*>(a->codes_t);
  p.scale_out = a->scale_out;
  p.colsum_ws = a->colsum != nullptr ? a->workspace : nullptr;
  p.ldx = a->ldx;
  p.ldq = a->ldq;
  p.ldt = a->ldt;
  p.rows = a->rows;
  p.cols = a->cols;
  p.e5m2 = a->f8_format == 1;
  p.dl8_flush = a->dl8_flush;
  p.f8_max = a->f8_max;
  p.eps = a->eps;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int rc;
  switch (a->x_dtype) {
    case QLIN_DT_F32:
      rc = launch_f8_tensor<float>(p, s);
      break;
    case QLIN_DT_F16:
      rc = launch_f8_tensor<__half>(p, s);
      break;
    case QLIN_DT_BF16:
      rc = launch_f8_tensor<__nv_bfloat16>(p, s);
      break;
    default:
      return fail(QLIN_ERR_BAD_DTYPE, "qlin_f8_tensor_quant: x_dtype must be F32, F16 or BF16");
  }
  if (rc != QLIN_OK || a->colsum == nullptr) return rc;
  f8_colsum_finish_kernel<<<(a->cols + 255) / 256, 256, 0, s>>>(a->workspace, (a->rows + kF8TileM - 1) / kF8TileM, a->cols, a->colsum);
  QLIN_CHECK_LAUNCH("qlin_f8_tensor_quant(column sums)");
  return QLIN_OK;
}
