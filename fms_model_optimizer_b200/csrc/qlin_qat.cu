// The fp32 product of a QAT Linear and its gradients on bf16 tensor cores, at fp32 accuracy.
//
//   out[t,n] = sum_k x[t,k] w[n,k] + b[n],   gx[t,k] = sum_n g[t,n] w[n,k],   gw[n,k] = sum_t g[t,n] x[t,k]
//
// x and w are fake-quantised: x = c step and w = d s[n] with whole numbers c, d of at most 8 bits and a sign, which bf16 holds
// exactly (up to 256, so the codes 256 and -1 that some clip pairs reach fit, and so does a NaN).  With the zero point taken
// off beforehand there is no offset that could cancel.  The gradient is any fp32 number: g s[n] (times a power of two that keeps
// small parts in range), rounded once, is the sum of three bf16 numbers (8 + 8 + 8 bits, each rounded from what the ones before
// left over).  So the forward product is one bf16 GEMM whose sums are whole numbers, and each gradient is three, with every
// product exact and the sums in fp32.
//
// The tensor core truncates as it adds, which shows after a few hundred terms.  So no accumulator of a gradient lives longer
// than 64 values of K (192 products, three parts each): the epilogue warps read it and add it to running sums in registers, rounded to nearest, while the tensor core
// fills the other accumulator.  Relative error (2-norm) against 64 bits, tokens x in x out, of the output, gx and gw, and of
// the fp32 library product in brackets: 4096 x 768 x 3072 5.7e-8, 1.5e-7, 1.6e-7 (4.9e-7, 9.9e-7, 1.1e-6); 64 x 768 x 768
// 5.6e-8, 9.6e-8, 6.5e-8 (2.3e-7, 2.3e-7, 1.5e-7); 16384 x 1024 x 1024 5.4e-8, 1.0e-7, 3.0e-7 (5.7e-7, 5.7e-7, 2.3e-6).  With
// accumulators of 256 terms the gradients are at 5.8e-7, in some shapes behind the library.
//
// What bounds it: the product itself, whose stages (three parts of the gradient and one of codes, 56 to 64 KB for 768 to 1536
// tensor cycles) are limited by what three of them keep in flight from L2; then the split of the gradient (HBM).  Forward and
// backward of 4096 x 768 x 3072: 1124 us of device time with the library's fp32 GEMMs, 212 with this.
//
// What the argument rests on is checked where the operands are made: a value that is not bit for bit what the quantizer makes of a
// whole number (another quantizer's output, a hook's), a scale out of range, an infinity or NaN in the gradient, a gradient element
// so large that a sum of its products with codes could leave fp32's range (which the product with the operand itself need not), or a
// tiny one beside a scale at which its lost digits could show raises a flag on the device.  Every block of a product reads its
// flags first, and with one up the product is computed in fp32 from the operands themselves.
#include <cmath>

#include <cuda.h>
#include <cuda_bf16.h>

#include "qlin_internal.h"
#include "qlin_ptx.cuh"
#include "qlin_rows.cuh"

namespace qlin {

// ------------------------------------------------------------------------------------------------ operands
constexpr float kMaxCode = 256.0f;                // whole numbers up to here are bf16 numbers
// A gradient enters as t = g s 2^kShift, and the products take the power of two out again.  Let 2^e be at least the longer contraction.
// Above: |t| up to 2^(kSumExp - e), so that a sum of 2^e products with codes of up to 2^8 stays below 2^126.  Below: from 2^-100 on
// the third part is a normal bf16 number.  A smaller t loses at most 2^-124, its sums 2^(e - 115), gx 2^(e - 115 - kShift) and gw
// that times step / s: below half of the smallest fp32 number, which no result can show, while step / s is at most
// 2^(kShift - 36 - e).  So tiny elements (the tails of a GELU's or a softmax's gradient) cost nothing, and only a tiny element
// in a column whose step / s is above that raises the flag.  At e = 12: |g s| up to 2^34, step / s up to 2^24.
constexpr int kShift = 72;
constexpr int kSumExp = 118;
constexpr float kTiny = 7.888609052210118e-31f;   // 2^-100
constexpr float kShiftUp = 4722366482869645213696.0f, kShiftDown = 1.0f / kShiftUp;  // 2^72, 2^-72
constexpr float kApart = 8.8817841970012523e-16f;  // 2^-50
constexpr int kPrepThreads = 256;
constexpr int kQatFlagSlots = 1184;  // flags of each kernel that makes an operand

struct QatCodesParams {
  const float* x;       // [rows, cols], dense
  __nv_bfloat16* codes; // [rows, ldo], or [cols, ldo] when transposed
  const float* clip;    // activations: clip_val [1]; weights: one per row
  const float* clipn;   // two-sided activations: clip_valn [1]
  float* scale;         // activations: step [1]; weights: s [rows]
  float* clip_kept;     // symmetric activations: the clip value of the forward pass [1]
  int32_t* flags;       // one per block
  int64_t ldo;
  int32_t rows, cols, num_bits, variant, transposed, given;  // given: `scale` holds the step or scales of the forward pass
};

// The step of the activation quantizers, in the order qlin_pact2_fwd derives it.
__device__ __forceinline__ float act_step(const QatCodesParams& p) {
  const float cv = *p.clip;
  float range, n;
  if (p.variant == QLIN_PACT_TWO_SIDED) {
    range = __fsub_rn(cv, *p.clipn);
    n = static_cast<float>((1 << p.num_bits) - 1);
  } else if (p.variant == QLIN_PACT_ONE_SIDED) {
    range = cv;
    n = static_cast<float>((1 << p.num_bits) - 1);
  } else {
    range = __fmul_rn(2.0f, cv);
    n = static_cast<float>((1 << p.num_bits) - 2);
  }
  return __fdiv_rn(1.0f, __fmul_rn(__fdiv_rn(1.0f, range), n));
}

__device__ __forceinline__ bool scale_ok(float s) {
  const float a = fabsf(s);
  return a > 1e-18f && a < 1e18f;
}

// The whole number of steps in x; `bad` is raised where x is not the fp32 product of one (NaN passes as NaN).
__device__ __forceinline__ float code_of(float x, float step, float rstep, bool& bad) {
  const float c = rintf(div_exact(x, step, rstep));
  bad |= !(x == __fmul_rn(c, step) && fabsf(c) <= kMaxCode) && x == x;
  return c;
}

// The symmetric quantizer's values are not products but k * step - clip with k = 0 .. 2 half, up to 2^-15 of a step off the
// multiple k - half of the step that they stand for.  So `bad` is raised where x is not that expression of a whole number.
__device__ __forceinline__ float code_of_sym(float x, float step, float rstep, float clip, float half, bool& bad) {
  const float k = rintf(div_exact(__fadd_rn(x, clip), step, rstep));
  const float c = k - half;
  bad |= !(x == __fsub_rn(__fmul_rn(k, step), clip) && fabsf(c) <= kMaxCode) && x == x;
  return c;
}

__device__ __forceinline__ uint32_t pack_codes(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Activations: flat over the rows, eight columns a thread and step (cols is a multiple of 8).
__global__ void __launch_bounds__(kPrepThreads) qat_act_codes_kernel(const QatCodesParams p) {
  const float step = p.given ? *p.scale : act_step(p), rstep = rcp_for_div(step);
  bool bad = !scale_ok(step);
  const bool sym = p.variant == QLIN_PACT_SYMMETRIC;
  const float clip = !sym ? 0.0f : (p.given ? *p.clip_kept : *p.clip), half = static_cast<float>((1 << (p.num_bits - 1)) - 1);
  const auto code = [&](float v) { return sym ? code_of_sym(v, step, rstep, clip, half, bad) : code_of(v, step, rstep, bad); };
  const int per_row = p.cols / 8;
  const int64_t total = static_cast<int64_t>(p.rows) * per_row;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * kPrepThreads + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * kPrepThreads) {
    const float4 a = reinterpret_cast<const float4*>(p.x)[2 * i], b = reinterpret_cast<const float4*>(p.x)[2 * i + 1];
    uint4 o;
    o.x = pack_codes(code(a.x), code(a.y));
    o.y = pack_codes(code(a.z), code(a.w));
    o.z = pack_codes(code(b.x), code(b.y));
    o.w = pack_codes(code(b.z), code(b.w));
    reinterpret_cast<uint4*>(p.codes)[i] = o;
  }
  const int any = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    p.flags[blockIdx.x] = any;
    if (blockIdx.x == 0 && !p.given) {
      *p.scale = step;
      if (sym) *p.clip_kept = clip;
    }
  }
}

// Weights: one scale per row, tiles of 64 x 64 so that the codes can be written transposed.
__global__ void __launch_bounds__(kPrepThreads) qat_weight_codes_kernel(const QatCodesParams p) {
  __shared__ __nv_bfloat16 tile[64][66];
  const int tiles_c = (p.cols + 63) / 64, tiles = ((p.rows + 63) / 64) * tiles_c;
  bool bad = false;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int r0 = t / tiles_c * 64, c0 = t % tiles_c * 64;
    const int c = (threadIdx.x & 15) * 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = k * 16 + (threadIdx.x >> 4), row = r0 + r;
      if (row < p.rows && c0 + c < p.cols) {  // cols is a multiple of 8
        const float s = p.given ? p.scale[row] : __fdiv_rn(__fmul_rn(p.clip[row], 2.0f), static_cast<float>((1 << p.num_bits) - 2));
        const float4 v = *reinterpret_cast<const float4*>(p.x + static_cast<int64_t>(row) * p.cols + c0 + c);
        const bool zero = s == 0.0f;  // a row of zeros: any scale will do
        const float sp = zero ? 1.0f : s, rs = rcp_for_div(sp);
        if (!zero) bad |= !scale_ok(s);
        const uint32_t lo = pack_codes(code_of(v.x, sp, rs, bad), code_of(v.y, sp, rs, bad));
        const uint32_t hi = pack_codes(code_of(v.z, sp, rs, bad), code_of(v.w, sp, rs, bad));
        if (zero) bad |= !(v.x == 0.0f && v.y == 0.0f && v.z == 0.0f && v.w == 0.0f);
        if (p.transposed) {
          *reinterpret_cast<uint32_t*>(&tile[r][c]) = lo;
          *reinterpret_cast<uint32_t*>(&tile[r][c + 2]) = hi;
        } else {
          *reinterpret_cast<uint2*>(p.codes + static_cast<int64_t>(row) * p.ldo + c0 + c) = make_uint2(lo, hi);
        }
        if (c0 + c == 0 && !p.given) p.scale[row] = sp;
      }
    }
    if (p.transposed) {
      __syncthreads();
      // a warp writes 64 consecutive rows of one column: two codes a lane
      const int lane = threadIdx.x & 31;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int cc = k * 8 + (threadIdx.x >> 5), r = 2 * lane;
        if (c0 + cc < p.cols && r0 + r < p.rows) {  // rows is a multiple of 8
          __nv_bfloat162 v;
          v.x = tile[r][cc];
          v.y = tile[r + 1][cc];
          *reinterpret_cast<__nv_bfloat162*>(p.codes + static_cast<int64_t>(c0 + cc) * p.ldo + r0 + r) = v;
        }
      }
      __syncthreads();
    }
  }
  const int any = __syncthreads_or(bad);
  if (threadIdx.x == 0) p.flags[blockIdx.x] = any;
}

struct QatSplitParams {
  const float* g;         // [rows, cols], dense
  const float* scale;     // [cols]
  __nv_bfloat16* planes;  // [3][rows][cols]
  int32_t* flags;
  float* sums;            // optional [row blocks][cols]: each block's column sums
  float* rcp;             // [cols]: 1 / s
  int32_t rows, cols, block_rows;
  const float* step;      // optional [1]: without it no tiny element is left out
  float huge, far;        // the largest |t|; the largest step / s at which tiny elements go unseen
};
constexpr int kSplitThreads = 128;  // eight columns a thread

// g s[n] 2^kShift as three bf16 numbers, and the column sums of g.  Bound by HBM: 4 bytes read and 6 written an element.
__global__ void __launch_bounds__(kSplitThreads) qat_split_kernel(const QatSplitParams p) {
  const int strips = (p.cols + 8 * kSplitThreads - 1) / (8 * kSplitThreads);
  const int c = (static_cast<int>(blockIdx.x % strips) * kSplitThreads + static_cast<int>(threadIdx.x)) * 8;
  const int rb = blockIdx.x / strips;
  const int row1 = min(p.rows, (rb + 1) * p.block_rows);
  const int64_t plane = static_cast<int64_t>(p.rows) * p.cols / 8;
  const bool vec = (reinterpret_cast<uintptr_t>(p.g) & 15u) == 0;
  bool bad = false;
  if (c < p.cols) {  // cols is a multiple of 8
    const float4 sa = *reinterpret_cast<const float4*>(p.scale + c), sb = *reinterpret_cast<const float4*>(p.scale + c + 4);
    float s[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
    uint32_t far = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      bad |= !scale_ok(s[j]);  // also for products that the weight's codes are no part of
      if (rb == 0) p.rcp[c + j] = __fdiv_rn(1.0f, s[j]);  // made here so that it undoes the very scale that the planes carry
      if (p.step == nullptr || !(fabsf(*p.step) <= p.far * fabsf(s[j]))) far |= 1u << j;
      s[j] *= kShiftUp;
    }
    float sum[8] = {};
#pragma unroll 4
    for (int row = rb * p.block_rows; row < row1; ++row) {
      const int64_t at = static_cast<int64_t>(row) * p.cols + c;
      float v[8];
      if (vec) {
        const float4 a = *reinterpret_cast<const float4*>(p.g + at), b = *reinterpret_cast<const float4*>(p.g + at + 4);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
      } else {  // a gradient that starts anywhere
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = p.g[at + j];
      }
      uint32_t o[3][4];
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        float2 t = __fmul2_rn(make_float2(v[j], v[j + 1]), make_float2(s[j], s[j + 1]));
        // not finite or too large (a NaN fails every comparison), or too small where that shows; an exact zero is fine
        bad |= !(fabsf(t.x) <= p.huge) || ((far >> j & 1) && fabsf(t.x) < kTiny && v[j] != 0.0f);
        bad |= !(fabsf(t.y) <= p.huge) || ((far >> (j + 1) & 1) && fabsf(t.y) < kTiny && v[j + 1] != 0.0f);
        sum[j] += v[j];
        sum[j + 1] += v[j + 1];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const uint32_t h = pack_codes(t.x, t.y);
          o[q][j / 2] = h;
          t = __fadd2_rn(t, make_float2(-__uint_as_float(h << 16), -__uint_as_float(h & 0xFFFF0000u)));
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) reinterpret_cast<uint4*>(p.planes)[q * plane + at / 8] = make_uint4(o[q][0], o[q][1], o[q][2], o[q][3]);
    }
    if (p.sums != nullptr) {
      float4* dst = reinterpret_cast<float4*>(p.sums + static_cast<int64_t>(rb) * p.cols + c);
      dst[0] = make_float4(sum[0], sum[1], sum[2], sum[3]);
      dst[1] = make_float4(sum[4], sum[5], sum[6], sum[7]);
    }
  }
  const int any = __syncthreads_or(bad);
  if (threadIdx.x == 0) p.flags[blockIdx.x] = any;
}

// Adds the row blocks' column sums: 32 columns a block, eight threads a column, in a fixed order.
__global__ void __launch_bounds__(256) qat_colsum_kernel(const float* sums, int blocks, int cols, float* out) {
  __shared__ float part[8][33];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), g = threadIdx.x >> 5;
  float a = 0.0f;
  if (c < cols)
#pragma unroll 8
    for (int b = g; b < blocks; b += 8) a += sums[static_cast<int64_t>(b) * cols + c];
  part[g][threadIdx.x & 31] = a;
  __syncthreads();
  if (g == 0 && c < cols) {
#pragma unroll
    for (int k = 1; k < 8; ++k) a += part[k][threadIdx.x & 31];
    out[c] = a;
  }
}

// ------------------------------------------------------------------------------------------------ fp32 product on a flag
// D[M,N] = sum_k A[m,k] B[n,k] + bias[n] from the fp32 operands, one FMA a term in the order of k.  Each operand is dense along K or along
// its rows, and the dense side is a multiple of 8.
struct QatFp32Params {
  const float* a;
  const float* b;
  int64_t a_m, a_k, b_n, b_k;  // element strides
  int32_t a_vec;               // a starts on a 16-byte boundary
  int32_t wide;                // tiles of 128 columns
};
constexpr int kFpM = 128, kFpK = 16, kFpThreads = 256;
constexpr int fp_row(int k, int width) { return k * (width + 4); }  // 16-byte rows
constexpr int fp_buffer_floats(int nt) { return fp_row(kFpK, kFpM) + fp_row(kFpK, 64 * nt); }

// Bound by the FMA pipe and by what shared memory returns (8 x 8 outputs a thread take four 16-byte reads for 32 packed FMAs; with 8 x 4
// it is three for 16).  Tiles of 128 x 64 NT, two buffers, the next 16 values of k on their way from global memory while these are
// multiplied.  Forward and backward with a flag up, a kernel of 64 x 64 tiles behind the tensor cores' product -> this in its place
// (library): one infinity in the gradient, 4096 x 768 x 3072 2992 -> 1234 us (1185), 2048 x 4096 x 4096 10790 -> 3420 (3735); activations
// with codes past 256 10380 -> 3550 (3735), the forward pass of that alone 4720 -> 1850 (1240).
// Not inlined: beside it the tensor cores' path would spill.
template <int NT>
__device__ __noinline__ void qat_fp32_product(const QatFp32Params f, float* d, const float* bias, int M, int N, int K) {
  extern __shared__ __align__(1024) uint8_t smem_bytes[];
  float* smem = reinterpret_cast<float*>(smem_bytes);
  constexpr int kN = 64 * NT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ty = (warp & 3) * 32 + (lane >> 3) * 4, tx = (warp >> 2) * 32 * NT + (lane & 7) * 4;  // rows ty .. + 3 and 16 on, columns tx .. + 3 and 32 on
  const int num_n = (N + kN - 1) / kN, tiles = (M + kFpM - 1) / kFpM * num_n, num_k = (K + kFpK - 1) / kFpK;
  const bool a_along_k = f.a_k == 1, b_along_k = f.b_k == 1;
  // a thread brings four values along the dense side from one row, or one k, of each 64 rows
  const int ar = a_along_k ? tid >> 2 : (tid & 15) * 4, ak = a_along_k ? (tid & 3) * 4 : tid >> 4;
  const int br = b_along_k ? tid >> 2 : (tid & 15) * 4, bk = b_along_k ? (tid & 3) * 4 : tid >> 4;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int m0 = t / num_n * kFpM, n0 = t % num_n * kN;
    float4 ra[2], rb[NT];
    const auto fetch = [&](int k0) {  // four along the dense side are all inside or all outside
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int m = m0 + ar + 64 * c;
        ra[c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (m < M && k0 + ak < K) {
          const float* src = f.a + m * f.a_m + (k0 + ak) * f.a_k;
          ra[c] = f.a_vec ? *reinterpret_cast<const float4*>(src) : make_float4(src[0], src[1], src[2], src[3]);
        }
      }
#pragma unroll
      for (int c = 0; c < NT; ++c) {
        const int n = n0 + br + 64 * c;
        rb[c] = n < N && k0 + bk < K ? *reinterpret_cast<const float4*>(f.b + n * f.b_n + (k0 + bk) * f.b_k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    };
    const auto put = [](float* dst, int width, bool along_k, int k, int r, float4 v) {
      if (along_k) {
        dst[fp_row(k, width) + r] = v.x;
        dst[fp_row(k + 1, width) + r] = v.y;
        dst[fp_row(k + 2, width) + r] = v.z;
        dst[fp_row(k + 3, width) + r] = v.w;
      } else {
        *reinterpret_cast<float4*>(dst + fp_row(k, width) + r) = v;
      }
    };
    const auto keep = [&](int buf) {
      float* sa = smem + buf * fp_buffer_floats(NT);
#pragma unroll
      for (int c = 0; c < 2; ++c) put(sa, kFpM, a_along_k, ak, ar + 64 * c, ra[c]);
#pragma unroll
      for (int c = 0; c < NT; ++c) put(sa + fp_row(kFpK, kFpM), kN, b_along_k, bk, br + 64 * c, rb[c]);
    };
    float2 acc[8][2 * NT];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 2 * NT; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
    fetch(0);
    keep(0);
    asm volatile("bar.sync 3, 256;" ::: "memory");
#pragma unroll 1
    for (int kb = 0; kb < num_k; ++kb) {
      const bool more = kb + 1 < num_k;
      if (more) fetch((kb + 1) * kFpK);
      const float* sa = smem + (kb & 1) * fp_buffer_floats(NT);
      const float* sb = sa + fp_row(kFpK, kFpM);
#pragma unroll
      for (int k = 0; k < kFpK; ++k) {
        float av[8];
        float2 bv[2 * NT];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 u = *reinterpret_cast<const float4*>(sa + fp_row(k, kFpM) + ty + 16 * h);
          av[4 * h] = u.x, av[4 * h + 1] = u.y, av[4 * h + 2] = u.z, av[4 * h + 3] = u.w;
        }
#pragma unroll
        for (int h = 0; h < NT; ++h) {
          const float4 u = *reinterpret_cast<const float4*>(sb + fp_row(k, kN) + tx + 32 * h);
          bv[2 * h] = make_float2(u.x, u.y), bv[2 * h + 1] = make_float2(u.z, u.w);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 2 * NT; ++j) acc[i][j] = __ffma2_rn(make_float2(av[i], av[i]), bv[j], acc[i][j]);
      }
      if (more) keep((kb + 1) & 1);
      asm volatile("bar.sync 3, 256;" ::: "memory");
    }
#pragma unroll
    for (int h = 0; h < NT; ++h) {
      const int n = n0 + tx + 32 * h;
      if (n >= N) continue;  // N is a multiple of 8
      const float4 c = bias == nullptr ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : make_float4(bias[n], bias[n + 1], bias[n + 2], bias[n + 3]);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty + (i >> 2) * 16 + (i & 3);
        float4 o = make_float4(acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x, acc[i][2 * h + 1].y);
        if (bias != nullptr) o = make_float4(__fadd_rn(o.x, c.x), __fadd_rn(o.y, c.y), __fadd_rn(o.z, c.z), __fadd_rn(o.w, c.w));
        if (m < M) *reinterpret_cast<float4*>(d + static_cast<int64_t>(m) * N + n) = o;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ product
// D[M,N] = (sum over planes and K of A_plane[m,k] B[n,k]) * row[m] * col[n] * scalar * down + bias[n] in fp32, one CTA pair per
// 256 x BN tile.  A stage holds 64 K values of all planes of A and of B, so B is loaded once for the three planes.  An operand is
// K-major ([rows, K] in memory: boxes of 64 K values x rows) or MN-major ([K, rows]: boxes of 64 rows x 64 K values).
struct QatGemmParams {
  float* d;
  const float* row;
  const float* col;
  const float* scalar;
  const float* bias;
  int32_t* status;
  float down;  // a power of two
  int32_t M, N, K, planes, a_mn, b_mn, promote;  // promote: stages per accumulator
  int32_t num_m, num_n;
  const int32_t* flags;  // three groups of kQatFlagSlots; the first n of each belong to this product's operands
  int32_t flag_n[3];
  QatFp32Params f;
};

struct QatAux {
  uint64_t full[4];
  uint64_t empty[4];
  uint64_t tfull[2];
  uint64_t tempty[2];
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
  float cs[256];
  float bias[256];
};

template <int BN_>
struct QatCfg {
  static constexpr int BN = BN_;
  static constexpr int STAGES = 3;
  static constexpr int EPI_WARPS = 8;
  static constexpr int PRODUCER_WARP = EPI_WARPS;
  static constexpr int MMA_WARP = EPI_WARPS + 1;
  static constexpr int THREADS = (EPI_WARPS + 2) * 32;
  static constexpr int PLANE_BYTES = 128 * 128;    // 128 rows x 64 bf16
  static constexpr int B_BYTES = BN / 2 * 128;
  static constexpr int STAGE_BYTES = 3 * PLANE_BYTES + B_BYTES;
  static constexpr int COLS = BN / 2;              // columns of an epilogue warp
  static constexpr int OUT_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int AUX_OFFSET = OUT_OFFSET + EPI_WARPS * 4096;
  static constexpr int SMEM_BYTES = AUX_OFFSET + static_cast<int>(sizeof(QatAux));
};
static_assert(QatCfg<256>::SMEM_BYTES <= 232448, "shared memory budget");
static_assert(2 * fp_buffer_floats(2) * 4 <= QatCfg<128>::OUT_OFFSET && kFpThreads == QatCfg<128>::EPI_WARPS * 32, "the fp32 product runs in the epilogue warps");

__device__ __forceinline__ void qat_load(uint32_t bar, void* dst, const void* tmap, int32_t x, int32_t y, int32_t z) {
  asm volatile(
      "{\n\t"
      ".reg .pred pe;\n\t"
      "elect.sync _|pe, 0xffffffff;\n\t"
      "@pe cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {%3, %4, %5}], [%0];\n\t"
      "}" ::"r"(bar),
      "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void qat_expect(uint32_t bar, uint32_t bytes) {
  asm volatile(
      "{\n\t"
      ".reg .pred pe;\n\t"
      "elect.sync _|pe, 0xffffffff;\n\t"
      "@pe mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;\n\t"
      "}" ::"r"(bar),
      "r"(bytes)
      : "memory");
}
// Leader only: the four K = 16 steps of 64 K values of one plane.  astep, bstep: descriptor units (16 bytes) between steps.
__device__ __forceinline__ void qat_mma4(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint64_t astep, uint64_t bstep, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred pe, pa, pt;\n\t"
      ".reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
      "elect.sync _|pe, 0xffffffff;\n\t"
      "setp.ne.b32 pa, %4, 0;\n\t"
      "setp.ne.b32 pt, %3, 0;\n\t"
      "add.s64 a1, %1, %5;\n\t"
      "add.s64 b1, %2, %6;\n\t"
      "add.s64 a2, a1, %5;\n\t"
      "add.s64 b2, b1, %6;\n\t"
      "add.s64 a3, a2, %5;\n\t"
      "add.s64 b3, b2, %6;\n\t"
      "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, pa;\n\t"
      "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], a1, b1, %3, pt;\n\t"
      "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], a2, b2, %3, pt;\n\t"
      "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], a3, b3, %3, pt;\n\t"
      "}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "l"(astep), "l"(bstep)
      : "memory");
}
// Descriptor of an MN-major tile: chunks of 64 rows (128 bytes), each 64 K values deep and 8 KB from the next; groups of
// eight K values are 1024 bytes apart.
__device__ __forceinline__ uint64_t make_smem_desc_mn(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(8192 >> 4) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

template <int BN>
__global__ void __launch_bounds__(QatCfg<BN>::THREADS, 1)
qat_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ CUtensorMap tmap_d,
                const QatGemmParams p) {
  using C = QatCfg<BN>;
  extern __shared__ __align__(1024) uint8_t smem[];
  QatAux* aux = reinterpret_cast<QatAux*>(smem + C::AUX_OFFSET);
  volatile int* abort_flag = &aux->abort_flag;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const bool aligned = (smem_u32(smem) & 1023u) == 0;
  int up = 0;  // the flags are complete: the kernels that raise them ended before this one began
#pragma unroll
  for (int g = 0; g < 3; ++g)
#pragma unroll
    for (int i = 0; i < (kQatFlagSlots + C::THREADS - 1) / C::THREADS; ++i) {
      const int at = i * C::THREADS + static_cast<int>(threadIdx.x);
      if (at < p.flag_n[g]) up |= p.flags[g * kQatFlagSlots + at];
    }

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&aux->full[s], 1);
      mbar_init(&aux->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&aux->tfull[b], 1);
      mbar_init(&aux->tempty[b], 2 * C::EPI_WARPS);
    }
    mbar_init(&aux->drain, 1);
    aux->abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == C::MMA_WARP) {
    tmem_alloc_pair(&aux->tmem_base, 512);
    tmem_relinquish_pair();
  }
  if (warp == C::PRODUCER_WARP && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_d);
  }
  tc_fence_before();
  const bool again = __syncthreads_or(up) != 0;  // the same in every block
  cluster_arrive_wait();  // both CTAs' barriers exist before either touches the other's
  tc_fence_after();
  const uint32_t tmem_base = aux->tmem_base;

  const int num_tiles = p.num_m * p.num_n;
  const int num_kb = (p.K + 63) / 64;
  bool timed_out = false;

  if (again) {
    if (warp < C::EPI_WARPS) {
      if (p.f.wide) {
        qat_fp32_product<2>(p.f, p.d, p.bias, p.M, p.N, p.K);
      } else {
        qat_fp32_product<1>(p.f, p.d, p.bias, p.M, p.N, p.K);
      }
    }
  } else if (!aligned) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, static_cast<int32_t>(QLIN_ERR_BAD_ALIGN));
  } else if (warp == C::PRODUCER_WARP) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    uint32_t s = 0, ph = 0;
    bool ok = true;
    const uint32_t bytes = 2u * (static_cast<uint32_t>(p.planes) * C::PLANE_BYTES + C::B_BYTES);
    for (int t = pair; t < num_tiles && ok; t += num_pairs) {
      const int m0 = (t % p.num_m) * 256 + static_cast<int>(rank) * 128;
      const int n0 = (t / p.num_m) * BN + static_cast<int>(rank) * (BN / 2);
      for (int kb = 0; kb < num_kb; ++kb) {
        ok = warp_mbar_wait(&aux->empty[s], ph ^ 1u, abort_flag);
        if (!ok) break;
        uint8_t* st = smem + s * C::STAGE_BYTES;
        const uint32_t bar = map_to_cta(&aux->full[s], 0);
        if (leader) qat_expect(bar, bytes);
        for (int q = 0; q < p.planes; ++q) {
          uint8_t* dst = st + q * C::PLANE_BYTES;
          if (p.a_mn) {
            qat_load(bar, dst, &tmap_a, m0, kb * 64, q);
            qat_load(bar, dst + 8192, &tmap_a, m0 + 64, kb * 64, q);
          } else {
            qat_load(bar, dst, &tmap_a, kb * 64, m0, q);
          }
        }
        uint8_t* dst = st + 3 * C::PLANE_BYTES;
        if (p.b_mn) {
          for (int c = 0; c < BN / 128; ++c) qat_load(bar, dst + c * 8192, &tmap_b, n0 + c * 64, kb * 64, 0);
        } else {
          qat_load(bar, dst, &tmap_b, kb * 64, n0, 0);
        }
        if (++s == C::STAGES) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
    if (!ok && lane == 0) {
      timed_out = !*abort_flag;
      *abort_flag = 1;
    }
    __syncwarp();
  } else if (warp == C::MMA_WARP) {
    if (leader) {
      // ---------------------------------------------------------------- MMA issuer (leader only)
      const uint32_t idesc = make_idesc(1u, 1u, 256, BN) | (p.a_mn ? 1u << 15 : 0u) | (p.b_mn ? 1u << 16 : 0u);
      const uint32_t a0 = smem_u32(smem), b0 = a0 + 3 * C::PLANE_BYTES;
      const uint64_t adesc0 = p.a_mn ? make_smem_desc_mn(a0) : make_smem_desc_sw128(a0);
      const uint64_t bdesc0 = p.b_mn ? make_smem_desc_mn(b0) : make_smem_desc_sw128(b0);
      const uint64_t astep = p.a_mn ? 128 : 2, bstep = p.b_mn ? 128 : 2;
      uint32_t s = 0, ph = 0, buf = 0, bph = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        int left = 0;  // stages until the accumulator is handed over
        uint32_t cur = 0;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = warp_mbar_wait(&aux->full[s], ph, abort_flag);
          if (!ok) break;
          const bool fresh = left == 0;
          if (fresh) {
            ok = warp_mbar_wait(&aux->tempty[buf], bph ^ 1u, abort_flag);
            if (!ok) break;
            cur = buf;
            buf ^= 1u;
            if (buf == 0) bph ^= 1u;
            left = min(p.promote, num_kb - kb);
          }
          tc_fence_after();
          const uint64_t off = static_cast<uint64_t>(s * (C::STAGE_BYTES >> 4));
          uint32_t accumulate = fresh ? 0u : 1u;
          for (int q = p.planes - 1; q >= 0; --q) {  // the smallest parts first
            qat_mma4(tmem_base + cur * 256, adesc0 + off + static_cast<uint64_t>(q * (C::PLANE_BYTES >> 4)), bdesc0 + off, astep, bstep, idesc, accumulate);
            accumulate = 1;
          }
          tc_commit_pair_elect(&aux->empty[s]);
          if (--left == 0) tc_commit_pair_elect(&aux->tfull[cur]);
          if (++s == C::STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      if (!ok && lane == 0) {
        timed_out = !*abort_flag;
        *abort_flag = 1;
      }
      // Nothing of the pair may still be reading shared memory or writing TMEM when the CTAs retire.
      tc_commit_pair_elect(&aux->drain);
      mbar_wait_drain(&aux->drain, 0);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue warps (both CTAs)
    const int q = warp & 3;
    const int half = warp >> 2;
    const float scalar = p.scalar != nullptr ? *p.scalar : 1.0f;
    uint8_t* stage = smem + C::OUT_OFFSET + warp * 4096;
    uint32_t buf = 0, bph = 0, piece = 0;
    bool ok = true;
    int t = pair;
    for (; t < num_tiles && ok; t += num_pairs) {
      const int row0 = (t % p.num_m) * 256 + static_cast<int>(rank) * 128 + q * 32;
      const int col0 = (t / p.num_m) * BN + half * C::COLS;
      // scales and bias of this half's columns, read by all lanes as broadcasts
      asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
      const int i = threadIdx.x & 127;
      if (i < C::COLS) {
        aux->cs[half * C::COLS + i] = (p.col != nullptr && col0 + i < p.N) ? p.col[col0 + i] : 1.0f;
        aux->bias[half * C::COLS + i] = (p.bias != nullptr && col0 + i < p.N) ? p.bias[col0 + i] : 0.0f;
      }
      asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
      float rs = __fmul_rn(scalar, (p.row != nullptr && row0 + lane < p.M) ? p.row[row0 + lane] : 1.0f);
      // the power of two goes with the factor, or before one that it would take out of fp32's range
      const bool apart = fabsf(rs) < kApart;
      if (!apart) rs = __fmul_rn(rs, p.down);
      float run[C::COLS];
      for (int kb = 0; kb < num_kb; kb += p.promote) {
        if (!warp_mbar_wait(&aux->tfull[buf], bph, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * 256 + half * C::COLS;
        const uint32_t done = buf;
#pragma unroll
        for (int c = 0; c < C::COLS; c += 32) {
          uint32_t v[32];
          tmem_ld32(addr + c, v);
          if (kb == 0) {
#pragma unroll
            for (int j = 0; j < 32; ++j) run[c + j] = __uint_as_float(v[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) run[c + j] = __fadd_rn(run[c + j], __uint_as_float(v[j]));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(&aux->tempty[done], 0));
        buf ^= 1u;
        if (buf == 0) bph ^= 1u;
      }
      if (!ok) break;
      if (__any_sync(0xffffffffu, apart)) {
#pragma unroll
        for (int e = 0; e < C::COLS; ++e) run[e] = apart ? __fmul_rn(run[e], p.down) : run[e];
      }
#pragma unroll
      for (int c = 0; c < C::COLS; c += 16) {
        uint8_t* dst = stage + (piece & 1) * 2048;
        if (lane == 0) tma_store_wait_read<1>();  // the store of two pieces ago has been read
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int e = c + 4 * k + j;
            const float y = __fmul_rn(run[e], __fmul_rn(rs, aux->cs[half * C::COLS + e]));
            w[j] = __float_as_uint(p.bias != nullptr ? __fadd_rn(y, aux->bias[half * C::COLS + e]) : y);
          }
          const uint32_t addr = smem_u32(dst) + lane * 64 + ((k ^ ((lane >> 1) & 3)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          if (row0 < p.M && col0 + c < p.N) tma_store_3d(&tmap_d, dst, col0 + c, row0, 0);
          tma_store_commit();
        }
        ++piece;
      }
    }
    if (lane == 0) tma_store_wait_read<0>();
    if (!ok && lane == 0) {
      timed_out = !*abort_flag;
      *abort_flag = 1;
    }
    // a warp that gave up still takes part in the barriers of the tiles that are left
    if (!ok)
      for (t += num_pairs; t < num_tiles; t += num_pairs) {
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
      }
  }

  if (timed_out && p.status != nullptr) atomicExch(p.status, static_cast<int32_t>(QLIN_ERR_TIMEOUT));
  if (*abort_flag) {
    // a wait gave up: copies of this CTA may still be in flight; give them time to land before the
    // shared memory is handed back
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 2000000ull) __nanosleep(256);
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive_wait();
  if (warp == C::MMA_WARP) {
    __syncwarp();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------------ host side
static int qat_map(CUtensorMap* tm, const void* base, int64_t cols, int64_t rows, int64_t planes, int box_x, int box_y, bool f32) {
  typedef CUresult (*Fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                         CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  Fn enc = reinterpret_cast<Fn>(tensor_map_encoder());
  if (enc == nullptr) return fail(QLIN_ERR_DEVICE, "cuTensorMapEncodeTiled is not available from this driver");
  const int64_t elt = f32 ? 4 : 2;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(planes)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(cols * elt), static_cast<cuuint64_t>(cols * rows * elt)};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(box_x), static_cast<cuuint32_t>(box_y), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(tm, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, f32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                         f32 ? CU_TENSOR_MAP_L2_PROMOTION_NONE : CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(QLIN_ERR_BAD_ALIGN, "cuTensorMapEncodeTiled failed with CUresult %d", static_cast<int>(r));
  return QLIN_OK;
}

template <int BN>
static int launch_qat_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const QatGemmParams& p, cudaStream_t stream) {
  using C = QatCfg<BN>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return fail(QLIN_ERR_DEVICE, "device ordinal %d out of range", dev);
  if (!configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(qat_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess) return fail(QLIN_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    configured[dev] = true;
  }
  // as many pairs as have a tile of this product or of the fp32 one
  const int64_t tiles = static_cast<int64_t>(p.num_m) * p.num_n, fp_tiles = static_cast<int64_t>((p.M + kFpM - 1) / kFpM) * ((p.N + 63) / 64);
  const int64_t busy = tiles > (fp_tiles + 1) / 2 ? tiles : (fp_tiles + 1) / 2;
  int pairs = sm_count() / 2;
  if (pairs > busy) pairs = static_cast<int>(busy);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs), 1, 1);
  cfg.blockDim = dim3(C::THREADS, 1, 1);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, qat_gemm_kernel<BN>, ta, tb, td, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QLIN_ERR_LAUNCH, "qlin_qat_gemm: %s", cudaGetErrorString(e));
  }
  return QLIN_OK;
}

static int prep_grid(int64_t work) {
  const int64_t most = static_cast<int64_t>(sm_count()) * 8, blocks = (work + kPrepThreads - 1) / kPrepThreads;
  const int64_t cap = most < kQatFlagSlots ? most : kQatFlagSlots;
  return static_cast<int>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

// The grids of the kernels that make the operands: one flag a block.
static int act_grid(const qlin_qat_args* a) { return prep_grid(static_cast<int64_t>(a->tokens) * a->in / 8); }
static int weight_grid(const qlin_qat_args* a) { return prep_grid(static_cast<int64_t>((a->out + 63) / 64) * ((a->in + 63) / 64) * kPrepThreads); }
static int split_strips(const qlin_qat_args* a) { return (a->out + 8 * kSplitThreads - 1) / (8 * kSplitThreads); }
// Rows of a block of the split kernel: sixteen, or as many as leave one flag a block.
static int split_block_rows(const qlin_qat_args* a) {
  const int most = kQatFlagSlots / split_strips(a) > 0 ? kQatFlagSlots / split_strips(a) : 1, need = (a->tokens + most - 1) / most;
  return need > 16 ? need : 16;
}
static int split_row_blocks(const qlin_qat_args* a) { return (a->tokens + split_block_rows(a) - 1) / split_block_rows(a); }
static int longer_exp(const qlin_qat_args* a) {
  int e = 0;
  while ((int64_t{1} << e) < (a->tokens > a->out ? a->tokens : a->out)) ++e;
  return e;
}
static float split_huge(const qlin_qat_args* a) { return std::ldexp(1.0f, kSumExp - longer_exp(a)); }
static float split_far(const qlin_qat_args* a) { return std::ldexp(1.0f, kShift - 36 - longer_exp(a)); }
static int split_grid(const qlin_qat_args* a) { return split_row_blocks(a) * split_strips(a); }

}  // namespace qlin

using namespace qlin;

extern "C" int32_t qlin_qat_flag_count(void) { return 3 * kQatFlagSlots; }
extern "C" int32_t qlin_qat_max_out(void) { return 8 * kSplitThreads * kQatFlagSlots; }

static bool qat_shape_ok(const qlin_qat_args* a) {
  return a->tokens > 0 && a->out <= qlin_qat_max_out() && a->in > 0 && a->out > 0 && a->in % 8 == 0 && a->out % 8 == 0 && static_cast<int64_t>(a->tokens) * a->in < (int64_t{1} << 40) &&
         static_cast<int64_t>(a->tokens) * a->out < (int64_t{1} << 40);
}

extern "C" int qlin_qat_codes(const qlin_qat_args* a, int32_t backward, void* stream) {
  if (a == nullptr) return fail(QLIN_ERR_NULL, "qlin_qat_codes: args is NULL");
  if (!qat_shape_ok(a)) return fail(QLIN_ERR_BAD_SHAPE, "qlin_qat: in and out must be positive multiples of 8");
  if (a->num_bits_x < 2 || a->num_bits_x > 8 || a->num_bits_w < 2 || a->num_bits_w > 8) return fail(QLIN_ERR_UNSUPPORTED, "qlin_qat: 2 to 8 bits");
  if (a->flags == nullptr || a->step == nullptr || a->scale == nullptr ||
      (!backward && (a->clip_x == nullptr || a->clip_w == nullptr || (a->variant == QLIN_PACT_TWO_SIDED && a->clipn_x == nullptr))))
    return fail(QLIN_ERR_NULL, "qlin_qat_codes: a pointer is NULL");
  if (a->variant == QLIN_PACT_SYMMETRIC && a->clip_kept == nullptr) return fail(QLIN_ERR_NULL, "qlin_qat_codes: the symmetric quantizer needs clip_kept");
  if (!aligned16(a->x) || !aligned16(a->w) || !aligned16(a->x_codes) || !aligned16(a->w_codes)) return fail(QLIN_ERR_BAD_ALIGN, "qlin_qat_codes: 16-byte alignment");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  QatCodesParams p = {};
  p.num_bits = a->num_bits_x;
  p.given = backward;
  p.variant = a->variant;
  if (a->x_codes != nullptr) {
    p.x = a->x;
    p.codes = static_cast<__nv_bfloat16*>(a->x_codes);
    p.clip = a->clip_x;
    p.clipn = a->clipn_x;
    p.scale = a->step;
    p.clip_kept = a->clip_kept;
    p.flags = a->flags;
    p.rows = a->tokens;
    p.cols = a->in;
    p.ldo = a->in;
    qat_act_codes_kernel<<<act_grid(a), kPrepThreads, 0, s>>>(p);
    QLIN_CHECK_LAUNCH("qlin_qat_codes");
  }
  if (a->w_codes != nullptr) {
    p.x = a->w;
    p.codes = static_cast<__nv_bfloat16*>(a->w_codes);
    p.num_bits = a->num_bits_w;
    p.clip = a->clip_w;
    p.scale = a->scale;
    p.flags = a->flags + kQatFlagSlots;
    p.rows = a->out;
    p.cols = a->in;
    p.ldo = backward ? a->out : a->in;
    p.transposed = backward;  // gx = g w contracts over w's rows
    qat_weight_codes_kernel<<<weight_grid(a), kPrepThreads, 0, s>>>(p);
    QLIN_CHECK_LAUNCH("qlin_qat_codes");
  }
  return QLIN_OK;
}

extern "C" int qlin_qat_split(const qlin_qat_args* a, void* stream) {
  if (a == nullptr) return fail(QLIN_ERR_NULL, "qlin_qat_split: args is NULL");
  if (!qat_shape_ok(a)) return fail(QLIN_ERR_BAD_SHAPE, "qlin_qat: in and out must be positive multiples of 8");
  if (a->g == nullptr || a->g_planes == nullptr || a->scale == nullptr || a->rcp == nullptr || a->flags == nullptr) return fail(QLIN_ERR_NULL, "qlin_qat_split: a pointer is NULL");
  if (!aligned16(a->g_planes) || !aligned16(a->scale)) return fail(QLIN_ERR_BAD_ALIGN, "qlin_qat_split: 16-byte alignment");
  if (a->colsum != nullptr && (a->workspace == nullptr || !aligned16(a->workspace))) return fail(QLIN_ERR_NULL, "qlin_qat_split: column sums need a workspace");
  QatSplitParams p = {a->g, a->scale, static_cast<__nv_bfloat16*>(a->g_planes), a->flags + 2 * kQatFlagSlots, a->colsum != nullptr ? a->workspace : nullptr, a->rcp, a->tokens, a->out,
                      split_block_rows(a), a->step, split_huge(a), split_far(a)};
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  qat_split_kernel<<<split_grid(a), kSplitThreads, 0, s>>>(p);
  QLIN_CHECK_LAUNCH("qlin_qat_split");
  if (a->colsum != nullptr) {
    qat_colsum_kernel<<<(a->out + 31) / 32, 256, 0, s>>>(a->workspace, split_row_blocks(a), a->out, a->colsum);
    QLIN_CHECK_LAUNCH("qlin_qat_split");
  }
  return QLIN_OK;
}

extern "C" int64_t qlin_qat_colsum_workspace_bytes(int32_t tokens, int32_t out) {
  qlin_qat_args a = {};
  a.tokens = tokens;
  a.out = out;
  return tokens > 0 && out > 0 ? static_cast<int64_t>(split_row_blocks(&a)) * out * 4 : 0;
}

extern "C" int qlin_qat_product(const qlin_qat_args* a, int32_t which, void* stream) {
  if (a == nullptr) return fail(QLIN_ERR_NULL, "qlin_qat_product: args is NULL");
  if (!qat_shape_ok(a)) return fail(QLIN_ERR_BAD_SHAPE, "qlin_qat: in and out must be positive multiples of 8");
  if (which < 0 || which > 2) return fail(QLIN_ERR_UNSUPPORTED, "qlin_qat_product: which must be 0, 1 or 2");
  if (a->d == nullptr || !aligned16(a->d) || !aligned16(a->x) || !aligned16(a->w)) return fail(QLIN_ERR_BAD_ALIGN, "qlin_qat_product: x, w and d must be 16-byte aligned");
  const int64_t T = a->tokens, I = a->in, O = a->out;
  QatGemmParams p = {};
  QatFp32Params& f = p.f;
  p.status = a->status;
  p.d = a->d;
  p.flags = a->flags;
  const void *pa, *pb;
  int64_t a_cols, a_rows, b_cols, b_rows;
  if (which == 0) {
    p.M = a->tokens, p.N = a->out, p.K = a->in, p.planes = 1;
    p.col = a->scale, p.scalar = a->step, p.bias = a->bias;
    pa = a->x_codes, pb = a->w_codes;
    a_cols = I, a_rows = T, b_cols = I, b_rows = O;
    f.a = a->x, f.a_m = I, f.a_k = 1, f.b = a->w, f.b_n = I, f.b_k = 1;
  } else if (which == 1) {
    p.M = a->tokens, p.N = a->in, p.K = a->out, p.planes = 3;
    pa = a->g_planes, pb = a->w_codes;
    a_cols = O, a_rows = T, b_cols = O, b_rows = I;
    f.a = a->g, f.a_m = O, f.a_k = 1, f.b = a->w, f.b_n = 1, f.b_k = I;
  } else {
    p.M = a->out, p.N = a->in, p.K = a->tokens, p.planes = 3, p.a_mn = p.b_mn = 1;
    p.row = a->rcp, p.scalar = a->step;
    pa = a->g_planes, pb = a->x_codes;
    a_cols = O, a_rows = T, b_cols = I, b_rows = T;
    f.a = a->g, f.a_m = 1, f.a_k = O, f.b = a->x, f.b_n = 1, f.b_k = I;
  }
  p.down = which == 0 ? 1.0f : kShiftDown;
  f.a_vec = aligned16(f.a);
  const int64_t rows = (p.M + kFpM - 1) / kFpM, ctas = sm_count() / 2 * 2;
  const auto rounds = [&](int width) { return (rows * ((p.N + width - 1) / width) + ctas - 1) / ctas; };
  f.wide = 8 * rounds(128) <= 5 * rounds(64);  // a round of 64 columns took 0.63 of one of 128 (264 and 420 us at 4096 terms)
  // a product looks at the flags of its own two operands: the others may have been left out
  p.flag_n[0] = which == 1 ? 0 : act_grid(a);
  p.flag_n[1] = which == 2 ? 0 : weight_grid(a);
  p.flag_n[2] = which == 0 ? 0 : split_grid(a);
  if (pa == nullptr || pb == nullptr || f.a == nullptr || f.b == nullptr || a->flags == nullptr) return fail(QLIN_ERR_NULL, "qlin_qat_product: a pointer is NULL");
  const int num_kb = (p.K + 63) / 64;
  // The sums of the forward product are whole numbers, exact in fp32 up to 2^24 and truncated beyond: one accumulator for as
  // many terms as stay below that whatever the codes are.
  p.promote = which == 0 ? (1 << 24) / (256 * 127) / 64 : 1;
  if (p.promote > num_kb) p.promote = num_kb;
  p.num_m = (p.M + 255) / 256;
  // The widest tile with the least work in the busiest pair: rounds of tiles times tile width.
  int bn = 256;
  int64_t best = INT64_MAX;
  const int widths[3] = {256, 192, 128};
  for (int w : widths) {
    if (w == 192 && p.b_mn) continue;  // boxes of 64 columns: a half tile of 96 is not a whole number of them
    const int64_t tiles = static_cast<int64_t>(p.num_m) * ((p.N + w - 1) / w), pairs = sm_count() / 2;
    const int64_t cost = (tiles + pairs - 1) / pairs * (w + 32);
    if (cost < best) best = cost, bn = w;
  }
  p.num_n = (p.N + bn - 1) / bn;
  CUtensorMap ta, tb, td;
  int rc = p.a_mn ? qat_map(&ta, pa, a_cols, a_rows, p.planes, 64, 64, false) : qat_map(&ta, pa, a_cols, a_rows, p.planes, 64, 128, false);
  if (rc != QLIN_OK) return rc;
  rc = p.b_mn ? qat_map(&tb, pb, b_cols, b_rows, 1, 64, 64, false) : qat_map(&tb, pb, b_cols, b_rows, 1, 64, bn / 2, false);
  if (rc != QLIN_OK) return rc;
  rc = qat_map(&td, a->d, p.N, p.M, 1, 16, 32, true);
  if (rc != QLIN_OK) return rc;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return bn == 256 ? launch_qat_gemm<256>(ta, tb, td, p, s) : bn == 192 ? launch_qat_gemm<192>(ta, tb, td, p, s) : launch_qat_gemm<128>(ta, tb, td, p, s);
}
