// The product of a fake-quantised activation and a fake-quantised weight (QLinear of QAT), forward and backward, on the int8
// tensor cores instead of an fp32 SIMT GEMM, with 64-bit accuracy up to the result's rounding.
//
// Both factors are whole numbers times scales: qx = (q + z) * step with q in [0, 255], qw = c * w_scale[n] with |c| <= 127.
//   forward   out[m,n] = step * w_scale[n] * (sum_k (q - h) c + (z + h) sum_k c) + bias[n], h = 2^(bits - 1): one int8 GEMM,
//             exact sums.
//   backward  gx[m,k] = sum_n (g[m,n] w_scale[n]) c[n,k] and gw[n,k] = step * sum_m g[m,n] (q + z)[m,k]: the fp32 factor is
//             written as a 31-bit fixed-point number per row (column) of g with a power-of-two scale, split into four
//             signed bytes, and the four byte planes run as one int8 GEMM with four times the rows; the int32 sums of the
//             planes are combined in fp64.  An element within 2^-6 of its row's maximum is represented exactly, any
//             other to 2^-31 of that maximum, and no sum is rounded, so the result is closer to the 64-bit product than
//             an fp32 GEMM's.  A row that holds an infinity or NaN gives NaN.
//
// 4096 x 768 x 3072, forward and backward with the quantizers: 1160 us with the fp32 library GEMMs (1063 of them), now 227 us
// on the GPU: three int8 GEMMs 98, planes and their statistics 63, combinations 17, codes and folded bias 13, the rest
// the quantizers.  Relative error against 64 bits: output 6e-8 (was 5e-7), gradients 4e-8 (was 1e-6).
//
// The kernels here are the ones around the GEMMs, all HBM / L2-bound: codes from fake-quantised values (row-major and
// transposed), the folded bias, row and column planes of g, and the combination of the planes' sums.
#include "qlin_internal.h"
#include "qlin_rows.cuh"

namespace qlin {

constexpr int kFmThreads = 256;

// Turns 4 x 4 bytes: word i holds row i; out[k] holds column k.
__device__ __forceinline__ void turn4(const uint32_t (&a)[4], uint32_t (&out)[4]) {
  const uint32_t t0 = __byte_perm(a[0], a[1], 0x5140), t1 = __byte_perm(a[2], a[3], 0x5140);
  const uint32_t t2 = __byte_perm(a[0], a[1], 0x7362), t3 = __byte_perm(a[2], a[3], 0x7362);
  out[0] = __byte_perm(t0, t1, 0x5410);
  out[1] = __byte_perm(t0, t1, 0x7632);
  out[2] = __byte_perm(t2, t3, 0x5410);
  out[3] = __byte_perm(t2, t3, 0x7632);
}

// value = (q + z) * step of a PACT+ quantiser, from its clip values, in the order the quantiser derives them (fp32).
struct ActScalars {
  float step;
  double z;
  double half;  // codes are stored as q - half, signed bytes around the middle of the range
};
__device__ __forceinline__ ActScalars act_scalars(const qlin_fq_act& a) {
  const float cv = *a.clip_val;
  ActScalars s;
  s.half = static_cast<double>(1 << (a.num_bits - 1));
  if (a.variant == QLIN_PACT_TWO_SIDED) {
    const float cvn = *a.clip_valn;
    const float scale = __fmul_rn(__fdiv_rn(1.0f, __fsub_rn(cv, cvn)), static_cast<float>((1 << a.num_bits) - 1));
    float zp = __fmul_rn(cvn, scale);
    if (a.align_zero) zp = rintf(zp);
    s.step = __fdiv_rn(1.0f, scale);
    s.z = zp;
  } else if (a.variant == QLIN_PACT_ONE_SIDED) {
    s.step = __fdiv_rn(1.0f, __fmul_rn(__fdiv_rn(1.0f, cv), static_cast<float>((1 << a.num_bits) - 1)));
    s.z = 0.0;
  } else {
    const float n = static_cast<float>((1 << a.num_bits) - (a.align_zero ? 2 : 1));
    s.step = __fdiv_rn(1.0f, __fmul_rn(__fdiv_rn(1.0f, __fmul_rn(2.0f, cv)), n));
    s.z = -static_cast<double>(cv) / static_cast<double>(s.step);
  }
  return s;
}
__device__ __forceinline__ float weight_scale(float clip, int num_bits) {
  return __fdiv_rn(__fmul_rn(clip, 2.0f), static_cast<float>((1 << num_bits) - 2));
}

// Codes of a fake-quantised tensor: q - half (activations) or c (weights, one scale per row), row-major and transposed.
// 128 x 64 tiles; out-of-range parts of the transposed rows are zeros.
template <bool WEIGHT>
__global__ void __launch_bounds__(kFmThreads) fq_codes_kernel(const float* v, int rows, int cols, const qlin_fq_act act, const float* w_clip, int w_bits,
                                                             uint8_t* codes, uint8_t* codes_t, int64_t ldt) {
  __shared__ uint32_t tile[128 * 16];
  double inv = 0.0, z = 0.0;
  if (!WEIGHT) {
    const ActScalars s = act_scalars(act);
    inv = 1.0 / static_cast<double>(s.step);
    z = s.z + s.half;
  }
  const int tiles_n = (cols + 63) / 64, tiles_m = (rows + 127) / 128;
  const int64_t tiles = static_cast<int64_t>(tiles_m) * tiles_n;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int row0 = static_cast<int>(t / tiles_n) * 128, col0 = static_cast<int>(t % tiles_n) * 64;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int id = threadIdx.x + h * kFmThreads;
      const int r = id >> 2, row = row0 + r, col = col0 + (id & 3) * 16;
      uint32_t w[4] = {0, 0, 0, 0};
      if (row < rows && col < cols) {  // cols is a multiple of 16
        float x[16];
        load16(v + static_cast<int64_t>(row) * cols + col, x);
        if (WEIGHT) inv = 1.0 / static_cast<double>(weight_scale(w_clip[row], w_bits));
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int c = __double2int_rn(static_cast<double>(x[j]) * inv - z);
          w[j >> 2] |= (static_cast<uint32_t>(c) & 0xFFu) << (8 * (j & 3));
        }
        *reinterpret_cast<uint4*>(codes + static_cast<int64_t>(row) * cols + col) = make_uint4(w[0], w[1], w[2], w[3]);
      }
#pragma unroll
      for (int g = 0; g < 4; ++g) tile[r * 16 + ((((id & 3) * 4) + g) ^ (r >> 3))] = w[g];
    }
    __syncthreads();
    const int rg = threadIdx.x & 15, c4 = threadIdx.x >> 4;
    uint32_t a[4], b[4], lo[4], hi[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = tile[(rg * 8 + i) * 16 + (c4 ^ rg)];
      b[i] = tile[(rg * 8 + 4 + i) * 16 + (c4 ^ rg)];
    }
    turn4(a, lo);
    turn4(b, hi);
    if (row0 + rg * 8 < ldt) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int col = col0 + c4 * 4 + k;
        if (col < cols) *reinterpret_cast<uint2*>(codes_t + static_cast<int64_t>(col) * ldt + row0 + rg * 8) = make_uint2(lo[k], hi[k]);
      }
    }
    __syncthreads();
  }
}

// One warp per weight row: w_scale[n], and bias[n] + step * w_scale[n] * (z + half) * sum_k c[n,k], formed in fp64.
// scal = {step, z + half} in fp64 for the backward pass, step_out the same step in fp32 (NaN where the quantiser's is unusable).
__global__ void __launch_bounds__(kFmThreads) fq_fold_kernel(const int8_t* codes, int n, int k, const qlin_fq_act act, const float* w_clip, int w_bits,
                                                            const float* bias, float* w_scale, float* bias_out, float* step_out, double* scal) {
  const ActScalars s = act_scalars(act);
  const bool usable = fabsf(s.step) > 0.0f && fabsf(s.step) < __int_as_float(0x7f800000);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *step_out = usable ? s.step : __int_as_float(0x7fc00000);
    scal[0] = usable ? static_cast<double>(s.step) : static_cast<double>(__int_as_float(0x7fc00000));
    scal[1] = s.z + s.half;
  }
  const int row = blockIdx.x * (kFmThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n) return;
  int sum = 0;
  const int4* src = reinterpret_cast<const int4*>(codes + static_cast<int64_t>(row) * k);
  for (int i = lane; i < k / 16; i += 32) {
    const int4 q = src[i];
    sum = __dp4a(q.x, 0x01010101, sum);
    sum = __dp4a(q.y, 0x01010101, sum);
    sum = __dp4a(q.z, 0x01010101, sum);
    sum = __dp4a(q.w, 0x01010101, sum);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) {
    const float ws = weight_scale(w_clip[row], w_bits);
    w_scale[row] = ws;
    const double fold = static_cast<double>(s.step) * static_cast<double>(ws) * (s.z + s.half) * static_cast<double>(sum);
    bias_out[row] = static_cast<float>((bias != nullptr ? static_cast<double>(bias[row]) : 0.0) + fold);
  }
}

// Power-of-two scale of a fixed-point row from the bits of its largest |value|: value * 2^e is below 2^30.  *back = 2^-e, or NaN
// for a row that holds an infinity or NaN.  A row of zeros gets 1.
__device__ __forceinline__ double plane_scale(uint32_t amax_bits, double* back) {
  if (amax_bits >= 0x7f800000u) {
    *back = static_cast<double>(__int_as_float(0x7fc00000));
    return 0.0;
  }
  const float m = __uint_as_float(amax_bits);
  const int e = m > 0.0f ? 29 - ilogbf(m) : 0;
  *back = scalbn(1.0, -e);
  return scalbn(1.0, e);
}
// |t| <= 2^30 -> four signed bytes, the lowest in the lowest byte: t = b0 + 2^8 b1 + 2^16 b2 + 2^24 b3.
__device__ __forceinline__ uint32_t plane_bytes(int t) { return (static_cast<uint32_t>(t) + 0x00808080u) ^ 0x00808080u; }

// One block per row of g: planes[b][m][n] = byte b of rint(g[m,n] * w_scale[n] * 2^e_m); back[m] = 2^-e_m.
__global__ void __launch_bounds__(kFmThreads) fq_row_planes_kernel(const float* g, const float* w_scale, int rows, int cols, uint8_t* planes, double* back) {
  __shared__ uint32_t red[kFmThreads / 32];
  const int n4 = cols >> 2;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const float4* src = reinterpret_cast<const float4*>(g + static_cast<int64_t>(row) * cols);
    const float4* ws4 = reinterpret_cast<const float4*>(w_scale);
    uint32_t am = 0;  // bits of |.|: an infinity or NaN is larger than every number
    for (int i = threadIdx.x; i < n4; i += kFmThreads) {
      const float4 v = src[i], w = ws4[i];
      am = max(max(am, __float_as_uint(fabsf(v.x * w.x))), __float_as_uint(fabsf(v.y * w.y)));
      am = max(max(am, __float_as_uint(fabsf(v.z * w.z))), __float_as_uint(fabsf(v.w * w.w)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) am = max(am, __shfl_xor_sync(0xffffffffu, am, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = am;
    __syncthreads();
    am = red[0];
#pragma unroll
    for (int i = 1; i < kFmThreads / 32; ++i) am = max(am, red[i]);
    __syncthreads();
    double inv_back;
    const double up = plane_scale(am, &inv_back);
    if (threadIdx.x == 0) back[row] = inv_back;
    const int64_t plane = static_cast<int64_t>(rows) * cols;
    for (int i = threadIdx.x; i < n4; i += kFmThreads) {
      const float4 v = src[i], w = ws4[i];
      const uint32_t t[4] = {plane_bytes(__double2int_rn(static_cast<double>(v.x) * w.x * up)), plane_bytes(__double2int_rn(static_cast<double>(v.y) * w.y * up)),
                             plane_bytes(__double2int_rn(static_cast<double>(v.z) * w.z * up)), plane_bytes(__double2int_rn(static_cast<double>(v.w) * w.w * up))};
      uint32_t out[4];
      turn4(t, out);
#pragma unroll
      for (int b = 0; b < 4; ++b) *reinterpret_cast<uint32_t*>(planes + b * plane + static_cast<int64_t>(row) * cols + 4 * i) = out[b];
    }
  }
}

// Column statistics of g over slices of rows: bits of max |g| and the fp64 sum.  A block: 128 columns x one slice.
__global__ void __launch_bounds__(kFmThreads) fq_col_stats_kernel(const float* g, int rows, int cols, int rows_per_slice, uint32_t* amax, double* sums) {
  __shared__ uint32_t s_max[8][128];
  __shared__ double s_sum[8][128];
  const int c4 = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int col = blockIdx.x * 128 + 4 * c4;
  const int r0 = blockIdx.y * rows_per_slice, r1 = min(rows, r0 + rows_per_slice);
  uint32_t m[4] = {0, 0, 0, 0};
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  if (col < cols) {
    for (int r = r0 + rl; r < r1; r += 8) {
      const float4 v = *reinterpret_cast<const float4*>(g + static_cast<int64_t>(r) * cols + col);
      m[0] = max(m[0], __float_as_uint(fabsf(v.x)));
      m[1] = max(m[1], __float_as_uint(fabsf(v.y)));
      m[2] = max(m[2], __float_as_uint(fabsf(v.z)));
      m[3] = max(m[3], __float_as_uint(fabsf(v.w)));
      s[0] += v.x;
      s[1] += v.y;
      s[2] += v.z;
      s[3] += v.w;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    s_max[rl][4 * c4 + j] = m[j];
    s_sum[rl][4 * c4 + j] = s[j];
  }
  __syncthreads();
  const int c = blockIdx.x * 128 + threadIdx.x;
  if (threadIdx.x < 128 && c < cols) {
    uint32_t mm = 0;
    double ss = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      mm = max(mm, s_max[i][threadIdx.x]);
      ss += s_sum[i][threadIdx.x];
    }
    amax[static_cast<int64_t>(blockIdx.y) * cols + c] = mm;
    sums[static_cast<int64_t>(blockIdx.y) * cols + c] = ss;
  }
}
// Folds the slices (in order): amax[0][c], the column's sum in fp64 and fp32 (the bias gradient).
__global__ void __launch_bounds__(kFmThreads) fq_col_finish_kernel(uint32_t* amax, const double* sums, int slices, int cols, double* sum, float* grad_bias) {
  const int c = blockIdx.x * kFmThreads + threadIdx.x;
  if (c >= cols) return;
  uint32_t m = 0;
  double s = 0.0;
  for (int i = 0; i < slices; ++i) {
    m = max(m, amax[static_cast<int64_t>(i) * cols + c]);
    s += sums[static_cast<int64_t>(i) * cols + c];
  }
  amax[c] = m;
  sum[c] = s;
  if (grad_bias != nullptr) grad_bias[c] = static_cast<float>(s);
}

// planes[b][n][m] = byte b of rint(g[m,n] * 2^e_n), rows of ldt bytes (zeros beyond `rows`); back[n] = 2^-e_n.  A block: 128
// rows x 32 columns of g through shared memory.
__global__ void __launch_bounds__(kFmThreads) fq_col_planes_kernel(const float* g, int rows, int cols, const uint32_t* amax, uint8_t* planes, int64_t ldt, double* back) {
  __shared__ uint32_t tile[128][33];
  const int row0 = blockIdx.y * 128, col0 = blockIdx.x * 32;
  const int lc = threadIdx.x & 31, col = col0 + lc;
  double up = 0.0, bk = 1.0;
  if (col < cols) up = plane_scale(amax[col], &bk);
  if (blockIdx.y == 0 && threadIdx.x < 32 && col < cols) back[col] = bk;
#pragma unroll 4
  for (int r = threadIdx.x >> 5; r < 128; r += 8) {
    const int row = row0 + r;
    float v = 0.0f;
    if (row < rows && col < cols) v = g[static_cast<int64_t>(row) * cols + col];
    tile[r][lc] = plane_bytes(__double2int_rn(static_cast<double>(v) * up));
  }
  __syncthreads();
  const int m4 = threadIdx.x & 31;
  if (row0 + 4 * m4 >= ldt) return;
  const int64_t plane = static_cast<int64_t>(cols) * ldt;
#pragma unroll
  for (int c = threadIdx.x >> 5; c < 32; c += 8) {
    if (col0 + c >= cols) break;
    const uint32_t t[4] = {tile[4 * m4][c], tile[4 * m4 + 1][c], tile[4 * m4 + 2][c], tile[4 * m4 + 3][c]};
    uint32_t out[4];
    turn4(t, out);
#pragma unroll
    for (int b = 0; b < 4; ++b) *reinterpret_cast<uint32_t*>(planes + b * plane + static_cast<int64_t>(col0 + c) * ldt + row0 + 4 * m4) = out[b];
  }
}

// out[r,c] = ((sum of the planes' products) * back[r] + add[r] * scal[1]) * scal[0]; add / scal may be NULL (0 and 1).
__global__ void __launch_bounds__(kFmThreads) fq_combine_kernel(const int32_t* acc, int rows, int cols, const double* back, const double* add, const double* scal, float* out) {
  const int n4 = cols >> 2;
  const int64_t total = static_cast<int64_t>(rows) * n4, plane = static_cast<int64_t>(rows) * n4;
  const int4* a = reinterpret_cast<const int4*>(acc);
  const double mul = scal != nullptr ? scal[0] : 1.0, off = scal != nullptr ? scal[1] : 0.0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * kFmThreads + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * kFmThreads) {
    const int r = static_cast<int>(i / n4);
    const int4 p0 = a[i], p1 = a[i + plane], p2 = a[i + 2 * plane], p3 = a[i + 3 * plane];
    const double bk = back[r], ad = add != nullptr ? add[r] * off : 0.0;
    // every partial value is a whole number below 2^53: exact
    auto one = [&](int x0, int x1, int x2, int x3) {
      const double d = ((static_cast<double>(x3) * 256.0 + x2) * 256.0 + x1) * 256.0 + x0;
      return static_cast<float>((d * bk + ad) * mul);
    };
    reinterpret_cast<float4*>(out)[i] = make_float4(one(p0.x, p1.x, p2.x, p3.x), one(p0.y, p1.y, p2.y, p3.y), one(p0.z, p1.z, p2.z, p3.z), one(p0.w, p1.w, p2.w, p3.w));
  }
}

static int cap_grid(int64_t want, int per_sm) {
  const int64_t cap = static_cast<int64_t>(sm_count()) * per_sm;
  return static_cast<int>(want < 1 ? 1 : (want < cap ? want : cap));
}
static int col_slices(int rows, int cols) {
  const int blocks = (cols + 127) / 128;
  int slices = (sm_count() * 4 + blocks - 1) / blocks;
  const int most = (rows + 31) / 32;
  if (slices > most) slices = most;
  return slices < 1 ? 1 : slices;
}

}  // namespace qlin

using namespace qlin;

extern "C" int qlin_fq_codes(const qlin_fq_codes_args* a, void* stream) {
  if (a == nullptr) return fail(QLIN_ERR_NULL, "qlin_fq_codes: args is NULL");
  if (a->rows < 1 || a->cols < 1 || a->cols % 16 != 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_fq_codes: cols must be a positive multiple of 16");
  if (a->v == nullptr || a->codes == nullptr || a->codes_t == nullptr) return fail(QLIN_ERR_NULL, "qlin_fq_codes: v, codes or codes_t is NULL");
  if (!aligned16(a->v) || !aligned16(a->codes) || !aligned16(a->codes_t) || a->ldt % 16 != 0 || a->ldt < a->rows)
    return fail(QLIN_ERR_BAD_ALIGN, "qlin_fq_codes: 16-byte aligned buffers and ldt >= rows, a multiple of 16, are wanted");
  const bool weight = a->w_clip != nullptr;
  if (!weight && a->act.clip_val == nullptr) return fail(QLIN_ERR_NULL, "qlin_fq_codes: neither activation nor weight clip values");
  if (!weight && (a->act.num_bits < 2 || a->act.num_bits > 8 || (a->act.variant == QLIN_PACT_TWO_SIDED && a->act.clip_valn == nullptr)))
    return fail(QLIN_ERR_UNSUPPORTED, "qlin_fq_codes: 2 to 8 bits, and clip_valn with the two-sided quantiser, are wanted");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int64_t tiles = static_cast<int64_t>((a->rows + 127) / 128) * ((a->cols + 63) / 64);
  const int grid = cap_grid(tiles, 6);
  if (weight) {
    fq_codes_kernel<true><<<grid, kFmThreads, 0, s>>>(a->v, a->rows, a->cols, a->act, a->w_clip, a->w_bits, static_cast<uint8_t*>(a->codes),
                                                     static_cast<uint8_t*>(a->codes_t), a->ldt);
  } else {
    fq_codes_kernel<false><<<grid, kFmThreads, 0, s>>>(a->v, a->rows, a->cols, a->act, nullptr, 0, static_cast<uint8_t*>(a->codes),
                                                      static_cast<uint8_t*>(a->codes_t), a->ldt);
  }
  QLIN_CHECK_LAUNCH("qlin_fq_codes");
  return QLIN_OK;
}

extern "C" int qlin_fq_fold(const int8_t* codes, int32_t n, int32_t k, const qlin_fq_act* act, const float* w_clip, int32_t w_bits, const float* bias,
                            float* w_scale, float* bias_out, float* step_out, double* scal, void* stream) {
  if (codes == nullptr || act == nullptr || w_clip == nullptr || w_scale == nullptr || bias_out == nullptr || step_out == nullptr || scal == nullptr)
    return fail(QLIN_ERR_NULL, "qlin_fq_fold: NULL argument");
  if (n < 1 || k < 1 || k % 16 != 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_fq_fold: k must be a positive multiple of 16");
  fq_fold_kernel<<<(n + kFmThreads / 32 - 1) / (kFmThreads / 32), kFmThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(codes, n, k, *act, w_clip, w_bits, bias, w_scale,
                                                                                                                          bias_out, step_out, scal);
  QLIN_CHECK_LAUNCH("qlin_fq_fold");
  return QLIN_OK;
}

extern "C" int qlin_fq_row_planes(const float* g, const float* w_scale, int32_t rows, int32_t cols, void* planes, double* back, void* stream) {
  if (g == nullptr || w_scale == nullptr || planes == nullptr || back == nullptr) return fail(QLIN_ERR_NULL, "qlin_fq_row_planes: NULL argument");
  if (rows < 1 || cols < 1 || cols % 16 != 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_fq_row_planes: cols must be a positive multiple of 16");
  if (!aligned16(g) || !aligned16(w_scale) || !aligned16(planes)) return fail(QLIN_ERR_BAD_ALIGN, "qlin_fq_row_planes: 16-byte aligned buffers are wanted");
  fq_row_planes_kernel<<<cap_grid(rows, 8), kFmThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(g, w_scale, rows, cols, static_cast<uint8_t*>(planes), back);
  QLIN_CHECK_LAUNCH("qlin_fq_row_planes");
  return QLIN_OK;
}

extern "C" int64_t qlin_fq_col_workspace_bytes(int32_t rows, int32_t cols) {
  return rows < 1 || cols < 1 ? 0 : static_cast<int64_t>(col_slices(rows, cols)) * cols * static_cast<int64_t>(sizeof(double) + sizeof(uint32_t));
}

extern "C" int qlin_fq_col_planes(const float* g, int32_t rows, int32_t cols, void* workspace, void* planes, int64_t ldt, double* back, double* colsum,
                                  float* grad_bias, void* stream) {
  if (g == nullptr || workspace == nullptr || colsum == nullptr) return fail(QLIN_ERR_NULL, "qlin_fq_col_planes: NULL argument");
  if (rows < 1 || cols < 1 || cols % 16 != 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_fq_col_planes: cols must be a positive multiple of 16");
  if (planes != nullptr && (back == nullptr || ldt < rows || ldt % 16 != 0 || !aligned16(planes)))
    return fail(QLIN_ERR_BAD_ALIGN, "qlin_fq_col_planes: planes need back, 16-byte alignment and ldt >= rows, a multiple of 16");
  if (!aligned16(g) || !aligned16(workspace)) return fail(QLIN_ERR_BAD_ALIGN, "qlin_fq_col_planes: 16-byte aligned buffers are wanted");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int slices = col_slices(rows, cols), per = (rows + slices - 1) / slices;
  const int used = (rows + per - 1) / per;
  double* sums = static_cast<double*>(workspace);
  uint32_t* amax = reinterpret_cast<uint32_t*>(sums + static_cast<int64_t>(slices) * cols);
  fq_col_stats_kernel<<<dim3((cols + 127) / 128, used), kFmThreads, 0, s>>>(g, rows, cols, per, amax, sums);
  fq_col_finish_kernel<<<(cols + kFmThreads - 1) / kFmThreads, kFmThreads, 0, s>>>(amax, sums, used, cols, colsum, grad_bias);
  if (planes != nullptr)
    fq_col_planes_kernel<<<dim3((cols + 31) / 32, (rows + 127) / 128), kFmThreads, 0, s>>>(g, rows, cols, amax, static_cast<uint8_t*>(planes), ldt, back);
  QLIN_CHECK_LAUNCH("qlin_fq_col_planes");
  return QLIN_OK;
}

extern "C" int qlin_fq_combine(const int32_t* acc, int32_t rows, int32_t cols, const double* back, const double* add, const double* scal, float* out, void* stream) {
  if (acc == nullptr || back == nullptr || out == nullptr) return fail(QLIN_ERR_NULL, "qlin_fq_combine: NULL argument");
  if (rows < 1 || cols < 1 || cols % 4 != 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_fq_combine: cols must be a positive multiple of 4");
  if (!aligned16(acc) || !aligned16(out)) return fail(QLIN_ERR_BAD_ALIGN, "qlin_fq_combine: 16-byte aligned buffers are wanted");
  const int64_t want = (static_cast<int64_t>(rows) * (cols / 4) + kFmThreads - 1) / kFmThreads;
  fq_combine_kernel<<<cap_grid(want, 8), kFmThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(acc, rows, cols, back, add, scal, out);
  QLIN_CHECK_LAUNCH("qlin_fq_combine");
  return QLIN_OK;
}
