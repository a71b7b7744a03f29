// qlin_gemm: persistent, warp-specialised tcgen05 GEMM for 8-bit operands on sm_100a.
//
//   D[M,N] = epilogue( C + sum over K-chunks of f( A[M,Kc] . B[N,Kc]^T ) )
//
// Both operands are K-major ("NT"), which is the layout the reference hands to its Triton / CUTLASS
// kernels (activations [m,k]; weight [n,k] passed as its .t() view).
//
// Per CTA (one per SM, 320 or 640 threads):
//   warp E      TMA producer (E = number of epilogue warps: 8 unchunked, 16 chunked): 128-byte-swizzled [128 x 128B] A tile and [BN x 128B] B tile per stage
//   warp E+1    MMA issuer: tcgen05.mma.cta_group::1 (M=128, N=BN, K=32 bytes per instruction),
//               accumulators in tensor memory; owns the TMEM allocation (chunked: three issuers, see MMA_WARPS)
//   warps 0..E-1 epilogue: tcgen05.ld of the accumulator, chunk rounding / running sum, dequantise,
//               global stores.  Warp w reads TMEM lanes 32*(w%4).. and column half w/4.
// Unchunked: BN=256, two 256-column accumulators so the epilogue of tile i overlaps the mainloop of
// tile i+1.  Chunked: BN=128, four 128-column accumulators; every K-chunk is a fresh accumulation
// that the epilogue warps drain, round and add to a running sum held in registers.
//
// Three kernels share this file: the CTA-pair kernel (cta_group::2, unchunked problems of at least 256 rows), the
// single-CTA kernel described above (chunked problems and the shapes in between), and the few-row kernel (at most
// 128 rows: weight rows as the MMA's M dimension, K split over a thread-block cluster).  Environment switches for
// A/B measurements: QLIN_GEMM_PAIR=0, QLIN_GEMM_SKINNY=0, QLIN_GEMM_LOWBYTE=0 select the kernel or mode each replaces.
//
// All mbarrier waits are bounded; a wait that runs out raises an abort flag, the CTA drains its
// copies and MMAs, frees TMEM, writes QLIN_ERR_TIMEOUT to the status word and returns.
#include <cstdlib>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "qlin_internal.h"
#include "qlin_ptx.cuh"

namespace qlin {

constexpr int kBM = 128;          // rows of A per tile = MMA M
constexpr int kBK = 128;          // bytes of K per pipeline stage = one swizzle row
constexpr int kGroupM = 16;       // m-blocks per raster group
constexpr int kTmemCols = 512;
constexpr int kStageOutBytes = 4096;  // per epilogue warp: 32 rows x 128 bytes of output

struct Aux {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t tfull[4];
  uint64_t tempty[4];
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
  float cs[256];
  float bias[256];
};

// SHORT_K: batched products whose tiles are a few K blocks deep (attention scores; short_batched has the rule).  They are written
// as fast as the epilogue goes: sixteen warps and three stages.
// The CTA-pair kernel, whose main loop counts, lost 3 to 7 % with sixteen warps and the five stages that they leave room for.
template <bool CHUNKED, bool SHORT_K = false>
struct Cfg {
  static constexpr int BN = CHUNKED ? 128 : 256;
  static constexpr int NBUF = CHUNKED ? 4 : 2;
  static constexpr int STAGES = CHUNKED ? 5 : (SHORT_K ? 3 : 4);
  // Epilogue warps: w % 4 selects the 32 TMEM lanes a warp may read, w / 4 its column slice.  The
  // chunked kernel drains an accumulator per K-chunk, a chain of short dependent steps, and hides
  // that latency with twice as many, narrower warps.
  static constexpr int EPI_WARPS = CHUNKED || SHORT_K ? 16 : 8;
  static constexpr int PRODUCER_WARP = EPI_WARPS;
  static constexpr int MMA_WARP = EPI_WARPS + 1;
  // Issuing the MMAs and the barrier traffic of one chunk takes a warp about 700 cycles, several times what the tensor pipe
  // needs for it: the chunked kernel shares the issue out, two warps taking every other chunk and, in low-byte mode, a third
  // keeping the untruncated total.  4096 x 8192 x 4096, 8 bits: chunks of 32 / 64 / 128 730 / 431 / 371 -> 643 / 372 / 256 us.
  // Without any hand-over of accumulators the issue side would take 246 us at 64 and the epilogue side 302.
  static constexpr int MMA_WARPS = CHUNKED ? 3 : 1;
  static constexpr int THREADS = (EPI_WARPS + 1 + MMA_WARPS) * 32;
  static constexpr int A_BYTES = kBM * kBK;
  static constexpr int B_BYTES = BN * kBK;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int COLS_PER_WARP = BN / (EPI_WARPS / 4);  // 128 columns, 64 (SHORT_K) or 32 (chunked)
  static constexpr int OUT_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int AUX_OFFSET = OUT_OFFSET + EPI_WARPS * kStageOutBytes;
  static constexpr int SMEM_BYTES = AUX_OFFSET + static_cast<int>(sizeof(Aux));
};
static_assert(Cfg<false>::SMEM_BYTES <= 232448 && Cfg<true>::SMEM_BYTES <= 232448 && Cfg<false, true>::SMEM_BYTES <= 232448, "shared memory budget");

struct GemmParams {
  const void* c;
  void* d;
  const float* rs;
  const float* cs;
  const float* bias;
  int32_t* status;
  int64_t ldc, ldd;
  int32_t M, N;
  int32_t kbytes;      // K in bytes
  int32_t chunk_k32;   // 32-byte MMA steps per accumulation chunk
  int32_t trun_bits, max_acc_bits, trunc_then_acc, clamp_dl16;
  int32_t epilogue, rs_stride, cs_stride, prod_round, scale_round, mid_round, acc_round, out_dtype;
  int32_t num_m, num_n, max_ctas;
  int32_t scatter_rows, scatter_row0;
  uint8_t* scatter_d[8];
  int32_t f8_ab_format;  // float kinds: operand format of the instruction descriptor, 0 = e4m3, 1 = e5m2
  int32_t batch;             // batched launch: problems stacked along the rows of A, B and along D (see qlin_gemm_batched)
  int64_t batch_stride_d;    // elements of the output type between the problems' outputs
  int32_t low_byte_mode;  // chunked int8, 8 truncated bits: the total on the tensor core, the chunks' low bytes on the ALU
  int32_t sk_mt, sk_split, sk_stages;  // few-row kernel: padded row count, K splits (= cluster size), pipeline stages
  int32_t dependent;                   // launched as the dependent of the quantiser that writes A and the row scales
  int32_t chain;                       // Chain of the epilogue (tiled stores)
};

// The epilogues that calls of this package ask for, compiled without a decision inside; any other combination of roundings
// takes kChainAny, which decides per step of 16 columns.
enum Chain : int32_t {
  kChainAny = 0,
  kChainRaw,         // accumulators as they are
  kChainProdBf16,    // SCALE_PROD, product rounded to bf16 then fp16, result to fp16: the deployed Linear of a bf16 model
  kChainProdF16,     // the same with the product rounded to fp16 once: fp16 and fp32 models
  kChainSeqBf16,     // SCALE_SEQ with both steps rounded to bf16: the FP8 Linear of a bf16 model
  kChainSeq,         // SCALE_SEQ without rounding steps
  kChainAcc16Tensor  // SCALE_ACC16 with one scale per operand: the batched product of attention
};

__device__ __forceinline__ float round_to(float y, int dt) {
  if (dt == QLIN_DT_F16) return __half2float(__float2half_rn(y));
  if (dt == QLIN_DT_BF16) return __bfloat162float(__float2bfloat16_rn(y));
  return y;
}

// The per-chunk rounding of the reference kernels.
template <bool F8>
__device__ __forceinline__ uint32_t chunk_round(uint32_t p, bool clamp, int32_t lo, int32_t hi, uint32_t rb,
                                                uint32_t mask, bool dl16) {
  if (!F8) {
    if (clamp) {
      int32_t v = static_cast<int32_t>(p);
      v = v > hi ? hi : v;
      v = v < lo ? lo : v;
      p = static_cast<uint32_t>(v);
    }
    return (p + rb) & mask;
  } else {
    p = (p + rb) & mask;
    if (dl16) {
      float x = __uint_as_float(p);
      const float dl16_max = 8581545984.0f;
      const float dl16_min = 4.665707820095122e-10f;
      if (x >= dl16_max) x = __int_as_float(0x7f800000);
      if (x <= -dl16_max) x = __int_as_float(0xff800000);
      if (fabsf(x) < dl16_min) x = 0.0f;
      p = __float_as_uint(x);
    }
    return p;
  }
}

template <bool F8>
__device__ __forceinline__ uint32_t acc_add(uint32_t a, uint32_t b) {
  if (F8) return __float_as_uint(__fadd_rn(__uint_as_float(a), __uint_as_float(b)));
  return a + b;
}

__device__ __forceinline__ void tile_coords(int t, int num_m, int num_n, int& mb, int& nb) {
  const int per_group = kGroupM * num_n;
  const int g = t / per_group;
  const int first_m = g * kGroupM;
  const int gsz = min(num_m - first_m, kGroupM);
  const int r = t - g * per_group;
  mb = first_m + r % gsz;
  nb = r / gsz;
}

// Accumulator -> output value (fp32, already rounded the way the epilogue mode asks).
template <bool F8>
__device__ __forceinline__ float dequant_one(const GemmParams& p, uint32_t v, float rs, float cs, float bias,
                                             bool prod, bool has_bias) {
  float a = F8 ? __uint_as_float(v) : __int2float_rn(static_cast<int32_t>(v));
  if (p.epilogue == QLIN_EPI_SCALE_ACC16) a = round_to(a, QLIN_DT_F16);
  float t;
  if (prod) {
    const float s = round_to(round_to(__fmul_rn(rs, cs), p.prod_round), p.scale_round);
    t = __fmul_rn(a, s);
  } else {
    t = round_to(__fmul_rn(__fmul_rn(a, rs), cs), p.mid_round);
  }
  if (has_bias) t = __fadd_rn(t, bias);
  return round_to(t, p.acc_round);
}

__device__ __forceinline__ uint32_t pack16(const GemmParams& p, float lo, float hi) {
  if (p.out_dtype == QLIN_DT_BF16) {
    return static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(lo))) |
           (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(hi))) << 16);
  }
  return static_cast<uint32_t>(__half_as_ushort(__float2half_rn(lo))) |
         (static_cast<uint32_t>(__half_as_ushort(__float2half_rn(hi))) << 16);
}

// Byte address of output row `row`, column 0 (`elt` bytes per element) of the output that starts at `dbase`.  With
// row-block scatter the block of scatter_rows rows that contains `row` lives in its own buffer (possibly another GPU's).
__device__ __forceinline__ uint8_t* out_row(const GemmParams& p, uint8_t* dbase, int row, int elt) {
  if (p.scatter_rows > 0) {
    const int owner = row / p.scatter_rows;
    return p.scatter_d[owner] + static_cast<int64_t>(row - owner * p.scatter_rows + p.scatter_row0) * p.ldd * elt;
  }
  return dbase + static_cast<int64_t>(row) * p.ldd * elt;
}

// ---- dequantisation of 32 accumulator columns held by one thread -------------------------------------------------
// Every step of the chain is a loop over 16 column pairs on packed fp32x2 arithmetic and packed conversions, and which
// rounding a step applies is decided once per step, not once per element.  An epilogue that asked per element (and
// rounded with the scalar conversions, which issue at a quarter of the rate) took about 17 us for a 128 x 256 tile of a
// CTA: 53 us of GEMM at 4096 x 768 x 3072 with fp32 output, 32 us at 517 x 4096 x 4096 with fp16 output.
template <int DT>
__device__ __forceinline__ float2 round2(float2 t) {
  if (DT == QLIN_DT_F16) return __half22float2(__float22half2_rn(t));
  if (DT == QLIN_DT_BF16) {
    const __nv_bfloat162 b2 = __float22bfloat162_rn(t);
    const uint32_t bw = *reinterpret_cast<const uint32_t*>(&b2);
    return make_float2(__uint_as_float(bw << 16), __uint_as_float(bw & 0xFFFF0000u));
  }
  return t;
}
__device__ __forceinline__ float2 pair_of(const uint32_t (&v)[32], int j) { return make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])); }
__device__ __forceinline__ void set_pair(uint32_t (&v)[32], int j, float2 t) {
  v[2 * j] = __float_as_uint(t.x);
  v[2 * j + 1] = __float_as_uint(t.y);
}
template <int DT>
__device__ __forceinline__ void round32(uint32_t (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) set_pair(v, j, round2<DT>(pair_of(v, j)));
}
__device__ __forceinline__ void round32_if(uint32_t (&v)[32], int dt) {
  if (dt == QLIN_DT_F16) {
    round32<QLIN_DT_F16>(v);
  } else if (dt == QLIN_DT_BF16) {
    round32<QLIN_DT_BF16>(v);
  }
}
template <int PROD, int SCALE>
__device__ __forceinline__ void mul_prod32(uint32_t (&v)[32], float rs, const float* cs) {
  const float2 rs2 = make_float2(rs, rs);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float2 sc = round2<SCALE>(round2<PROD>(__fmul2_rn(rs2, *reinterpret_cast<const float2*>(cs + 2 * j))));
    set_pair(v, j, __fmul2_rn(pair_of(v, j), sc));
  }
}
template <int PROD>
__device__ __forceinline__ void mul_prod32_if(uint32_t (&v)[32], float rs, const float* cs, int scale_round) {
  if (scale_round == QLIN_DT_F16) {
    mul_prod32<PROD, QLIN_DT_F16>(v, rs, cs);
  } else if (scale_round == QLIN_DT_BF16) {
    mul_prod32<PROD, QLIN_DT_BF16>(v, rs, cs);
  } else {
    mul_prod32<PROD, QLIN_DT_F32>(v, rs, cs);
  }
}
// Accumulators in, output values (fp32 bits, already rounded the way the epilogue mode asks) out.
template <bool F8>
__device__ __forceinline__ void dequant32(const GemmParams& p, uint32_t (&v)[32], float rs, const float* cs, const float* bias) {
  if (!F8) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__int2float_rn(static_cast<int32_t>(v[j])));
  }
  if (p.epilogue == QLIN_EPI_SCALE_PROD) {
    if (p.prod_round == QLIN_DT_BF16) {
      mul_prod32_if<QLIN_DT_BF16>(v, rs, cs, p.scale_round);
    } else if (p.prod_round == QLIN_DT_F16) {
      mul_prod32_if<QLIN_DT_F16>(v, rs, cs, p.scale_round);
    } else {
      mul_prod32_if<QLIN_DT_F32>(v, rs, cs, p.scale_round);
    }
  } else {
    if (p.epilogue == QLIN_EPI_SCALE_ACC16) round32<QLIN_DT_F16>(v);
    const float2 rs2 = make_float2(rs, rs);
#pragma unroll
    for (int j = 0; j < 16; ++j) set_pair(v, j, __fmul2_rn(__fmul2_rn(pair_of(v, j), rs2), *reinterpret_cast<const float2*>(cs + 2 * j)));
    round32_if(v, p.mid_round);
  }
  if (p.bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 16; ++j) set_pair(v, j, __fadd2_rn(pair_of(v, j), *reinterpret_cast<const float2*>(bias + 2 * j)));
  }
  round32_if(v, p.acc_round);
}
// 32 values -> 16 words of two 16-bit numbers.
__device__ __forceinline__ void pack32(const uint32_t (&v)[32], uint32_t* w, bool bf16) {
  if (bf16) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const __nv_bfloat162 o = __float22bfloat162_rn(pair_of(v, j));
      w[j] = *reinterpret_cast<const uint32_t*>(&o);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const __half2 o = __float22half2_rn(pair_of(v, j));
      w[j] = *reinterpret_cast<const uint32_t*>(&o);
    }
  }
}

// Coalesced store through this warp's 32 x 128-byte staging tile.  `w` holds this thread's row as
// 32 packed 32-bit words (128 bytes).  The tile is written with a 16-byte-chunk XOR swizzle so both
// the row-per-lane writes and the row-contiguous reads are bank-conflict free; every global store
// instruction then covers four full 128-byte lines.  `chunks` of the row's eight 16-byte pieces lie inside the output.
__device__ __forceinline__ void store_tile_coalesced(uint8_t* stage, const uint32_t (&w)[32], uint8_t* gbase,
                                                     int64_t row_pitch_bytes, int rows_valid, int lane, int chunks) {
  const uint32_t sbase = smem_u32(stage);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t addr = sbase + lane * 128 + ((c ^ (lane & 7)) << 4);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[4 * c]), "r"(w[4 * c + 1]),
                 "r"(w[4 * c + 2]), "r"(w[4 * c + 3])
                 : "memory");
  }
  __syncwarp();
  const int c = lane & 7;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3);
    uint32_t x0, x1, x2, x3;
    const uint32_t addr = sbase + r * 128 + ((c ^ (r & 7)) << 4);
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x0), "=r"(x1), "=r"(x2), "=r"(x3) : "r"(addr) : "memory");
    if (r < rows_valid && c < chunks) *reinterpret_cast<uint4*>(gbase + r * row_pitch_bytes + c * 16) = make_uint4(x0, x1, x2, x3);
  }
  __syncwarp();
}

// The same through the same staging tile for rows that do not start, or an edge that does not end, on a 16-byte boundary:
// a warp writes a row at a time, 4 bytes a lane (2 bytes where the rows of a 2-byte output are not 4-byte aligned), so
// each store instruction still covers consecutive bytes of one row; a thread storing its own row element by element
// touches 32 rows with every instruction.  `bytes` of the 128-byte row lie inside the output.
__device__ __forceinline__ void store_tile_narrow(uint8_t* stage, const uint32_t (&w)[32], uint8_t* gbase, int64_t row_pitch_bytes,
                                                  int rows_valid, int lane, int bytes) {
  const uint32_t sbase = smem_u32(stage);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t addr = sbase + lane * 128 + ((c ^ (lane & 7)) << 4);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[4 * c]), "r"(w[4 * c + 1]),
                 "r"(w[4 * c + 2]), "r"(w[4 * c + 3])
                 : "memory");
  }
  __syncwarp();
  const bool words = ((reinterpret_cast<uintptr_t>(gbase) | static_cast<uintptr_t>(row_pitch_bytes)) & 3u) == 0;
  const int rows = rows_valid < 32 ? rows_valid : 32;
#pragma unroll 4
  for (int r = 0; r < rows; ++r) {
    uint8_t* g = gbase + r * row_pitch_bytes;
    if (words) {
      uint32_t x;
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(x) : "r"(sbase + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4) : "memory");
      if (4 * lane + 4 <= bytes) {
        reinterpret_cast<uint32_t*>(g)[lane] = x;
      } else if (4 * lane < bytes) {
        reinterpret_cast<uint16_t*>(g)[2 * lane] = static_cast<uint16_t>(x);
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = h * 32 + lane;
        uint16_t x;
        asm volatile("ld.shared.b16 %0, [%1];" : "=h"(x) : "r"(sbase + r * 128 + (((e >> 3) ^ (r & 7)) << 4) + (e & 7) * 2) : "memory");
        if (2 * e < bytes) reinterpret_cast<uint16_t*>(g)[e] = x;
      }
    }
  }
  __syncwarp();
}

// Loads 32 columns of the optional initial accumulator C for one row (zeros when absent / outside).
template <int NC>
__device__ __forceinline__ void load_c_row(const GemmParams& p, uint32_t (&v)[NC], int row, int col0) {
#pragma unroll
  for (int j = 0; j < NC; ++j) v[j] = 0u;
  if (p.c == nullptr || row >= p.M) return;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(p.c) + static_cast<int64_t>(row) * p.ldc + col0;
#pragma unroll
  for (int j = 0; j < NC; ++j)
    if (col0 + j < p.N) v[j] = src[j];
}

// What the epilogue of a launch does, worked out once per thread.
struct EpiCtx {
  uint8_t* dbase;  // output of this tile's problem
  uint8_t* stage;  // this warp's staging tile
  bool two_byte, vec_ok, scaled;
};
__device__ __forceinline__ EpiCtx make_epi_ctx(const GemmParams& p, uint8_t* stage) {
  EpiCtx e;
  e.dbase = reinterpret_cast<uint8_t*>(p.d);
  e.stage = stage;
  e.scaled = p.epilogue != QLIN_EPI_RAW;
  e.two_byte = e.scaled && p.out_dtype != QLIN_DT_F32;
  const int elt = e.two_byte ? 2 : 4;
  e.vec_ok = (p.scatter_rows > 0 || (reinterpret_cast<uintptr_t>(p.d) & 15u) == 0) && ((p.ldd * elt) % 16 == 0) &&
             (p.batch <= 1 || (p.batch_stride_d * elt) % 16 == 0);
  return e;
}

// Stores one staging tile: this thread's row of `cols` columns (32 words).
__device__ __forceinline__ void emit_words(const GemmParams& p, const EpiCtx& e, const uint32_t (&w)[32], int row0, int lane, int col0, int cols) {
  const int elt = e.two_byte ? 2 : 4;
  const int left = min(p.N - col0, cols);
  if (left <= 0) return;
  uint8_t* g = out_row(p, e.dbase, row0, elt) + static_cast<int64_t>(col0) * elt;
  if (e.vec_ok && (left * elt) % 16 == 0) {
    store_tile_coalesced(e.stage, w, g, p.ldd * elt, p.M - row0, lane, left * elt / 16);
  } else {
    store_tile_narrow(e.stage, w, g, p.ldd * elt, p.M - row0, lane, left * elt);
  }
}

// Emits 64 accumulator columns [col0, col0 + 64) of this thread's row, given as two halves.
template <bool F8>
__device__ __forceinline__ void emit64(const GemmParams& p, const EpiCtx& e, uint32_t (&lo)[32], uint32_t (&hi)[32], int row0, int lane, int col0,
                                       const float* s_cs, const float* s_bias, float rs) {
  if (e.scaled) {
    dequant32<F8>(p, lo, rs, s_cs, s_bias);
    dequant32<F8>(p, hi, rs, s_cs + 32, s_bias + 32);
  }
  if (e.two_byte) {
    uint32_t w[32];  // 64 columns = one 128-byte staging row
    pack32(lo, w, p.out_dtype == QLIN_DT_BF16);
    pack32(hi, w + 16, p.out_dtype == QLIN_DT_BF16);
    emit_words(p, e, w, row0, lane, col0, 64);
  } else {
    emit_words(p, e, lo, row0, lane, col0, 32);
    emit_words(p, e, hi, row0, lane, col0 + 32, 32);
  }
}

// Emits 32 accumulator columns of this thread's row (the chunked kernel's final store).
template <bool F8>
__device__ __forceinline__ void emit32(const GemmParams& p, const EpiCtx& e, uint32_t (&v)[32], int row0, int lane, int col0, const float* s_cs,
                                       const float* s_bias, float rs) {
  if (e.scaled) dequant32<F8>(p, v, rs, s_cs, s_bias);
  if (e.two_byte) {
    uint32_t w[32];
    pack32(v, w, p.out_dtype == QLIN_DT_BF16);
#pragma unroll
    for (int j = 16; j < 32; ++j) w[j] = 0u;
    emit_words(p, e, w, row0, lane, col0, 32);
  } else {
    emit_words(p, e, v, row0, lane, col0, 32);
  }
}

// ---- the epilogue with tiled stores -------------------------------------------------------------------------------
// A loop over steps of 16 accumulator columns: the next step's tcgen05.ld is in flight while this step's values are scaled,
// rounded and packed; 64 bytes of every row (32 columns of a 2-byte type, 16 of a 4-byte type) make a piece of 32 rows,
// written to one of this warp's two 2 KB buffers with the 64-byte swizzle and stored by one TMA instruction, which also cuts
// off rows and columns beyond the output.  Bound by instruction issue and its latencies, not by stores: straight-line code over
// 64 columns with staged 16-byte stores (emit64, still used for outputs TMA cannot address) took up to 1300 instructions a
// warp and tile, fetched anew for every tile.  Kernel times before and after: attention scores 64 x 2048 x 128 x 2048 210 -> 108
// us (537 MB written at 5.0 TB/s), 4096 x 768 x 3072 with fp32 output 25.5 -> 21.5, 517 x 4096 x 4096 fp16 20.5 -> 18.8.
template <int N>
__device__ __forceinline__ float2 pair_n(const uint32_t (&v)[N], int j) { return make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])); }
template <int N>
__device__ __forceinline__ void set_pair_n(uint32_t (&v)[N], int j, float2 t) {
  v[2 * j] = __float_as_uint(t.x);
  v[2 * j + 1] = __float_as_uint(t.y);
}
template <int DT>
__device__ __forceinline__ void round16(uint32_t (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) set_pair_n(v, j, round2<DT>(pair_n(v, j)));
}
__device__ __forceinline__ void round16_if(uint32_t (&v)[16], int dt) {
  if (dt == QLIN_DT_F16) {
    round16<QLIN_DT_F16>(v);
  } else if (dt == QLIN_DT_BF16) {
    round16<QLIN_DT_BF16>(v);
  }
}
template <int PROD, int SCALE>
__device__ __forceinline__ void mul_prod16(uint32_t (&v)[16], float rs, const float* cs) {
  const float2 rs2 = make_float2(rs, rs);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 sc = round2<SCALE>(round2<PROD>(__fmul2_rn(rs2, *reinterpret_cast<const float2*>(cs + 2 * j))));
    set_pair_n(v, j, __fmul2_rn(pair_n(v, j), sc));
  }
}
template <int PROD>
__device__ __forceinline__ void mul_prod16_if(uint32_t (&v)[16], float rs, const float* cs, int scale_round) {
  if (scale_round == QLIN_DT_F16) {
    mul_prod16<PROD, QLIN_DT_F16>(v, rs, cs);
  } else if (scale_round == QLIN_DT_BF16) {
    mul_prod16<PROD, QLIN_DT_BF16>(v, rs, cs);
  } else {
    mul_prod16<PROD, QLIN_DT_F32>(v, rs, cs);
  }
}
// Accumulators of 16 columns in, output values (fp32 bits, rounded the way the epilogue asks) out: dequant32, step by step.
// `cst` is the one column scale of kChainAcc16Tensor.  A last rounding that packing to OUT repeats is left to it.
template <bool F8, int CH, int OUT>
__device__ __forceinline__ void dequant16(const GemmParams& p, uint32_t (&v)[16], float rs, float cst, const float* cs, const float* bias) {
  if (CH == kChainRaw) return;
  if (!F8) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__int2float_rn(static_cast<int32_t>(v[j])));
  }
  const float2 rs2 = make_float2(rs, rs);
  if (CH == kChainProdBf16) {
    mul_prod16<QLIN_DT_BF16, QLIN_DT_F16>(v, rs, cs);
  } else if (CH == kChainProdF16) {
    mul_prod16<QLIN_DT_F16, QLIN_DT_F32>(v, rs, cs);
  } else if (CH == kChainAcc16Tensor) {
    round16<QLIN_DT_F16>(v);
    const float2 cs2 = make_float2(cst, cst);
#pragma unroll
    for (int j = 0; j < 8; ++j) set_pair_n(v, j, __fmul2_rn(__fmul2_rn(pair_n(v, j), rs2), cs2));
    return;
  } else if (CH == kChainAny && p.epilogue == QLIN_EPI_SCALE_PROD) {
    if (p.prod_round == QLIN_DT_BF16) {
      mul_prod16_if<QLIN_DT_BF16>(v, rs, cs, p.scale_round);
    } else if (p.prod_round == QLIN_DT_F16) {
      mul_prod16_if<QLIN_DT_F16>(v, rs, cs, p.scale_round);
    } else {
      mul_prod16_if<QLIN_DT_F32>(v, rs, cs, p.scale_round);
    }
  } else {
    if (CH == kChainAny && p.epilogue == QLIN_EPI_SCALE_ACC16) round16<QLIN_DT_F16>(v);
#pragma unroll
    for (int j = 0; j < 8; ++j) set_pair_n(v, j, __fmul2_rn(__fmul2_rn(pair_n(v, j), rs2), *reinterpret_cast<const float2*>(cs + 2 * j)));
    if (CH == kChainSeqBf16) round16<QLIN_DT_BF16>(v);
    if (CH == kChainAny) round16_if(v, p.mid_round);
  }
  if (p.bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) set_pair_n(v, j, __fadd2_rn(pair_n(v, j), *reinterpret_cast<const float2*>(bias + 2 * j)));
  }
  if ((CH == kChainProdBf16 || CH == kChainProdF16) && OUT != QLIN_DT_F16) round16<QLIN_DT_F16>(v);
  if (CH == kChainSeqBf16 && OUT != QLIN_DT_BF16) round16<QLIN_DT_BF16>(v);
  if (CH == kChainAny) round16_if(v, p.acc_round);
}

constexpr int kPieceBytes = 2048;  // 32 rows x 64 bytes
__device__ __forceinline__ void piece_write(uint32_t sbase, int lane, int chunk, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
  const uint32_t addr = sbase + lane * 64 + ((chunk ^ ((lane >> 1) & 3)) << 4);
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w0), "r"(w1), "r"(w2), "r"(w3) : "memory");
}

// What the epilogue of one warp needs for a tile: its 32 rows from `row0` and `cols` (a multiple of 32) columns from `col0` of
// problem `bi`, held in TMEM from `taddr`; scales and bias of those columns in shared memory.
struct TilePart {
  const CUtensorMap* tmap_d;
  uint8_t* stage;  // this warp's two pieces
  uint32_t taddr;
  int cols, row0, col0, bi, lane;
  float rs, cst;
  const float* cs;
  const float* bias;
};

// `piece` counts the pieces this warp has written; `release` is called once the accumulator has been read.
template <bool F8, int CH, int OUT, typename Release>
__device__ __forceinline__ void drain_tile(const GemmParams& p, const TilePart& t, uint32_t& piece, Release release) {
  uint32_t va[16], vb[16];
  tmem_issue16(t.taddr, va);
  auto put = [&](uint32_t (&v)[16], int half, int col) {
    const uint32_t sbase = smem_u32(t.stage) + (piece & 1) * kPieceBytes;
    constexpr bool two_byte = OUT != QLIN_DT_F32;
    uint32_t w[two_byte ? 8 : 16];
    if (two_byte) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (OUT == QLIN_DT_BF16) {
          const __nv_bfloat162 o = __float22bfloat162_rn(pair_n(v, j));
          w[j] = *reinterpret_cast<const uint32_t*>(&o);
        } else {
          const __half2 o = __float22half2_rn(pair_n(v, j));
          w[j] = *reinterpret_cast<const uint32_t*>(&o);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) w[j] = v[j];
    }
    if (!two_byte || half == 0) {  // the buffer's previous store, two pieces ago, has been read
      if (t.lane == 0) tma_store_wait_read<1>();
      __syncwarp();
    }
#pragma unroll
    for (int c = 0; c < (two_byte ? 2 : 4); ++c) piece_write(sbase, t.lane, (two_byte ? 2 * half : 0) + c, w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
    if (!two_byte || half == 1) {
      fence_proxy_async();
      __syncwarp();
      const int x = two_byte ? col - 16 : col;
      if (t.lane == 0) {
        if (t.row0 < p.M && x < p.N) tma_store_3d(t.tmap_d, t.stage + (piece & 1) * kPieceBytes, x, t.row0, t.bi);
        tma_store_commit();  // a piece outside the output is an empty group: the wait above counts pieces
      }
      ++piece;
    }
  };
#pragma unroll 1
  for (int j = 0; j < t.cols; j += 32) {
    tmem_wait16(va);
    tmem_issue16(t.taddr + j + 16, vb);
    dequant16<F8, CH, OUT>(p, va, t.rs, t.cst, t.cs + j, t.bias + j);
    put(va, 0, t.col0 + j);
    tmem_wait16(vb);
    if (j + 32 < t.cols) {
      tmem_issue16(t.taddr + j + 32, va);
    } else {
      release();
    }
    dequant16<F8, CH, OUT>(p, vb, t.rs, t.cst, t.cs + j + 16, t.bias + j + 16);
    put(vb, 1, t.col0 + j + 16);
  }
}

// Which chain and output type a launch has are kernel arguments, so every warp of the grid takes the same branch.
template <bool F8, int CH, typename Release>
__device__ __forceinline__ void drain_tile_to(const GemmParams& p, const TilePart& t, uint32_t& piece, Release release) {
  if (p.out_dtype == QLIN_DT_BF16) {
    drain_tile<F8, CH, QLIN_DT_BF16>(p, t, piece, release);
  } else if (p.out_dtype == QLIN_DT_F16) {
    drain_tile<F8, CH, QLIN_DT_F16>(p, t, piece, release);
  } else {
    drain_tile<F8, CH, QLIN_DT_F32>(p, t, piece, release);
  }
}
template <bool F8, typename Release>
__device__ __forceinline__ void drain_tile_any(const GemmParams& p, const TilePart& t, uint32_t& piece, Release release) {
  if (p.chain == kChainRaw) {
    drain_tile<F8, kChainRaw, QLIN_DT_F32>(p, t, piece, release);
  } else if (p.chain == kChainSeq) {
    drain_tile_to<F8, kChainSeq>(p, t, piece, release);
  } else if (F8 && p.chain == kChainSeqBf16) {
    drain_tile<F8, kChainSeqBf16, QLIN_DT_BF16>(p, t, piece, release);
  } else if (!F8 && p.chain == kChainProdBf16) {
    drain_tile<F8, kChainProdBf16, QLIN_DT_BF16>(p, t, piece, release);
  } else if (!F8 && p.chain == kChainProdF16) {
    drain_tile_to<F8, kChainProdF16>(p, t, piece, release);
  } else if (!F8 && p.chain == kChainAcc16Tensor) {
    drain_tile_to<F8, kChainAcc16Tensor>(p, t, piece, release);
  } else {
    drain_tile_to<F8, kChainAny>(p, t, piece, release);
  }
}

// The column scales and bias of one column (thread i: column i of the tile) and the row scale of this thread's row, fetched a
// tile ahead so that their latency is not in the way of the accumulator they belong to.
struct TileScales {
  float cs, bias, rs;
};
__device__ __forceinline__ TileScales fetch_scales(const GemmParams& p, int col, bool has_col, int row) {
  TileScales t;
  t.cs = (p.cs != nullptr && has_col && col < p.N) ? p.cs[static_cast<int64_t>(col) * p.cs_stride] : 1.0f;
  t.bias = (p.bias != nullptr && has_col && col < p.N) ? p.bias[col] : 0.0f;
  t.rs = (p.rs != nullptr && row < p.M) ? p.rs[static_cast<int64_t>(row) * p.rs_stride] : 1.0f;
  return t;
}

// BATCHED: p.batch problems of the same shape whose operands are stacked along the rows (A is [batch * M, K], B is
// [batch * N, K]); a tile of problem b starts at row b * M of A and row b * N of B, its rows and columns beyond the
// problem's M and N belong to the next problem (or lie outside and read as zeros) and are dropped by the epilogue's
// bounds checks, and its output goes to D + b * batch_stride_d.
// TILED: outputs that TMA can address are stored by drain_tile_any (tmap_d); the others, and chunked problems, by emit64 / emit32.
template <bool F8, bool CHUNKED, bool BATCHED = false, bool TILED = false, bool SHORT_K = false>
__global__ void __launch_bounds__(Cfg<CHUNKED, SHORT_K>::THREADS, 1)
qlin_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 const __grid_constant__ CUtensorMap tmap_d, const GemmParams p) {
  using C = Cfg<CHUNKED, SHORT_K>;
  extern __shared__ __align__(1024) uint8_t smem[];
  Aux* aux = reinterpret_cast<Aux*>(smem + C::AUX_OFFSET);
  volatile int* abort_flag = &aux->abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // The 128-byte swizzle atoms need a 1024-byte aligned base; dynamic shared memory starts at the
  // base of the CTA's window, so this only guards against a toolchain that would place it elsewhere.
  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, static_cast<int32_t>(QLIN_ERR_BAD_ALIGN));
    return;
  }

  const int total_k32 = (p.kbytes + 31) / 32;
  // chunks that tile a 128-byte K block exactly (32, 64 or 128 elements, K a multiple of 128)
  const bool chunk_fast = CHUNKED && (p.chunk_k32 == 1 || p.chunk_k32 == 2 || p.chunk_k32 == 4) && (total_k32 % 4 == 0);
  // low-byte mode: the last accumulator holds the tile's untruncated total, the others rotate over the chunks
  const bool low_mode = CHUNKED && !F8 && p.low_byte_mode != 0;
  const int mma_warps = low_mode ? 3 : (chunk_fast ? 2 : 1);  // issuing warps: each releases every stage

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&aux->full[s], 1);
      mbar_init(&aux->empty[s], mma_warps);
    }
    for (int b = 0; b < C::NBUF; ++b) {
      mbar_init(&aux->tfull[b], 1);
      mbar_init(&aux->tempty[b], C::EPI_WARPS);
    }
    mbar_init(&aux->drain, mma_warps);
    aux->abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == C::MMA_WARP) {
    tmem_alloc(&aux->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  if (warp == C::PRODUCER_WARP && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    if (TILED) tma_prefetch_desc(&tmap_d);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = aux->tmem_base;

  const int per_batch = p.num_m * p.num_n;
  const int num_tiles = BATCHED ? per_batch * p.batch : per_batch;
  const int num_kb = (p.kbytes + kBK - 1) / kBK;
  bool timed_out = false;

  if (warp == C::PRODUCER_WARP) {
    // ------------------------------------------------------------------ TMA producer
    // The whole warp walks the loop converged; one elected lane issues.  The next stage's
    // barrier is polled (non-blocking) before the current stage is issued, which takes the
    // barrier round trip off the loop's critical path.
    griddep_wait();
    uint32_t s = 0, ph = 0, issued = 0;
    bool ok = true;
    bool ready = false;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      int mb, nb;
      const int bi = BATCHED ? t / per_batch : 0;
      tile_coords(t - bi * per_batch, p.num_m, p.num_n, mb, nb);
      const int ya = mb * kBM + bi * p.M, yb = nb * C::BN + bi * p.N;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!ready) {
          ok = warp_mbar_wait(&aux->empty[s], ph ^ 1u, abort_flag);
          if (!ok) break;
        }
        const uint32_t ns = (s + 1 == C::STAGES) ? 0u : s + 1;
        const uint32_t nph = (ns == 0u) ? (ph ^ 1u) : ph;
        const uint32_t peek = warp_mbar_test_begin(&aux->empty[ns], nph ^ 1u);
        uint8_t* sa = smem + s * C::STAGE_BYTES;
        tma_issue_stage(&aux->full[s], C::STAGE_BYTES, sa, &tmap_a, ya, sa + C::A_BYTES, &tmap_b, yb, kb * kBK);
        ++issued;
        ready = warp_mbar_test_end(peek);
        s = ns;
        ph = nph;
      }
    }
    if (!ok) {
      if (lane == 0) {
        timed_out = !*abort_flag;
        *abort_flag = 1;
      }
      // Let the copies already issued land before the CTA gives its shared memory back.
      for (uint32_t st = 0; st < static_cast<uint32_t>(C::STAGES); ++st) {
        if (issued <= st) continue;
        const uint32_t last = ((issued - 1 - st) / C::STAGES);  // index of the last fill of stage st
        mbar_wait_drain(&aux->full[st], last & 1u);
      }
    }
    __syncwarp();
  } else if (CHUNKED && chunk_fast && warp >= C::MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuers of whole chunks
    // Every issuing warp walks over all stages (so that the stage barriers of all stay in step), issues its share and
    // commits the stage.  Warp 0 and 1 take the even and the odd chunks, counted over all tiles; warp 2 the total.
    const int mw = warp - C::MMA_WARP;
    if (mw < mma_warps) {
      const uint32_t idesc = F8 ? make_idesc(1u, static_cast<uint32_t>(p.f8_ab_format), kBM, C::BN) : make_idesc(2u, 1u, kBM, C::BN);
      const uint64_t adesc0 = make_smem_desc_sw128(smem_u32(smem));
      const uint64_t bdesc0 = make_smem_desc_sw128(smem_u32(smem) + C::A_BYTES);
      const uint32_t nbuf = low_mode ? C::NBUF - 1 : C::NBUF;
      const uint32_t d_total = tmem_base + (C::NBUF - 1) * C::BN;
      const int cpk = 4 / p.chunk_k32;
      uint32_t s = 0, ph = 0;              // smem stage and its phase
      uint32_t buf = 0, bph = 0, turn = 0;  // accumulator of the next chunk, its phase, whose chunk it is
      uint32_t tot_ph = 0;
      bool ok = true, ready = false, tready = false;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        if (mw == 2) {  // the epilogue warps must have read the previous tile's total before it is overwritten
          ok = warp_mbar_wait(&aux->tempty[C::NBUF - 1], tot_ph ^ 1u, abort_flag);
          if (!ok) break;
          tot_ph ^= 1u;
        }
        for (int kb = 0; kb < num_kb && ok; ++kb) {
          if (!ready) {
            ok = warp_mbar_wait(&aux->full[s], ph, abort_flag);
            if (!ok) break;
          }
          tc_fence_after();
          const uint32_t ns = (s + 1 == C::STAGES) ? 0u : s + 1;
          const uint32_t nph = (ns == 0u) ? (ph ^ 1u) : ph;
          const uint32_t peek = warp_mbar_test_begin(&aux->full[ns], nph);
          const uint64_t adesc = adesc0 + static_cast<uint64_t>(s * (C::STAGE_BYTES >> 4));
          const uint64_t bdesc = bdesc0 + static_cast<uint64_t>(s * (C::STAGE_BYTES >> 4));
          if (mw == 2) {
            tc_mma4_release<F8 ? 1 : 0>(d_total, adesc, bdesc, idesc, kb > 0 ? 1u : 0u, &aux->empty[s]);
            if (kb == num_kb - 1) tc_commit_elect(&aux->tfull[C::NBUF - 1]);
          } else {
            for (int c = 0; c < cpk && ok; ++c) {
              const uint32_t nb = (buf + 1 == nbuf) ? 0u : buf + 1;
              const uint32_t nbph = (nb == 0u) ? (bph ^ 1u) : bph;
              if (turn == static_cast<uint32_t>(mw)) {
                if (!tready) {
                  ok = warp_mbar_wait(&aux->tempty[buf], bph ^ 1u, abort_flag);
                  if (!ok) break;
                }
                tc_fence_after();
                // this warp's next chunk is the next but one: its accumulator is polled before this chunk is issued
                const uint32_t nb2 = (nb + 1 == nbuf) ? 0u : nb + 1;
                const uint32_t nbph2 = (nb2 == 0u) ? (nbph ^ 1u) : nbph;
                const uint32_t tpeek = warp_mbar_test_begin(&aux->tempty[nb2], nbph2 ^ 1u);
                const uint64_t off = static_cast<uint64_t>(c * p.chunk_k32 * 2);
                const uint32_t d = tmem_base + buf * C::BN;
                if (p.chunk_k32 == 1) {
                  tc_mma_chunk<F8 ? 1 : 0, 1>(d, adesc + off, bdesc + off, idesc, &aux->tfull[buf]);
                } else if (p.chunk_k32 == 2) {
                  tc_mma_chunk<F8 ? 1 : 0, 2>(d, adesc + off, bdesc + off, idesc, &aux->tfull[buf]);
                } else {
                  tc_mma_chunk<F8 ? 1 : 0, 4>(d, adesc + off, bdesc + off, idesc, &aux->tfull[buf]);
                }
                tready = warp_mbar_test_end(tpeek);
              }
              turn ^= 1u;
              buf = nb;
              bph = nbph;
            }
            if (ok) tc_commit_elect(&aux->empty[s]);
          }
          ready = warp_mbar_test_end(peek);
          s = ns;
          ph = nph;
        }
      }
      if (!ok && lane == 0) {
        timed_out = !*abort_flag;
        *abort_flag = 1;
      }
      // Nothing may still be reading shared memory or writing TMEM when the CTA retires.
      tc_commit_elect(&aux->drain);
      mbar_wait_drain(&aux->drain, 0);
    }
    __syncwarp();
  } else if (warp > C::MMA_WARP) {
    // the further issuing warps have nothing to do in this mode
  } else if (warp == C::MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuer
    // One instruction stream feeds the tensor pipe, so this loop is latency-critical: no
    // divisions, positions carried as counters, a whole 128-byte K block issued by one fused
    // statement, and the next stage's barrier polled before the current block is issued.
    const uint32_t idesc = F8 ? make_idesc(1u, static_cast<uint32_t>(p.f8_ab_format), kBM, C::BN) : make_idesc(2u, 1u, kBM, C::BN);
    const uint64_t adesc0 = make_smem_desc_sw128(smem_u32(smem));
    const uint64_t bdesc0 = make_smem_desc_sw128(smem_u32(smem) + C::A_BYTES);
    uint32_t s = 0, ph = 0;          // smem stage and its phase
    uint32_t buf = 0, bph = 0;       // TMEM accumulator buffer to use next and its phase
    bool ok = true;
    bool ready = false;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      uint32_t accumulate = 0, cur = 0;
      int chunk_pos = 0;
      int k32_left = total_k32;
      for (int kb = 0; kb < num_kb && ok; ++kb) {
        if (!ready) {
          ok = warp_mbar_wait(&aux->full[s], ph, abort_flag);
          if (!ok) break;
        }
        tc_fence_after();
        const uint32_t ns = (s + 1 == C::STAGES) ? 0u : s + 1;
        const uint32_t nph = (ns == 0u) ? (ph ^ 1u) : ph;
        const uint32_t peek = warp_mbar_test_begin(&aux->full[ns], nph);
        const uint64_t adesc = adesc0 + static_cast<uint64_t>(s * (C::STAGE_BYTES >> 4));
        const uint64_t bdesc = bdesc0 + static_cast<uint64_t>(s * (C::STAGE_BYTES >> 4));
        if (!CHUNKED && k32_left >= 4) {
          if (kb == 0) {
            ok = warp_mbar_wait(&aux->tempty[buf], bph ^ 1u, abort_flag);
            if (!ok) break;
            tc_fence_after();
            cur = buf;
            if (++buf == C::NBUF) {
              buf = 0;
              bph ^= 1u;
            }
          }
          tc_mma4_release<F8 ? 1 : 0>(tmem_base + cur * C::BN, adesc, bdesc, idesc, accumulate, &aux->empty[s]);
          accumulate = 1;
          k32_left -= 4;
          if (k32_left == 0) tc_commit_elect(&aux->tfull[cur]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (k32_left > 0 && ok) {
              if (chunk_pos == 0 && (CHUNKED || accumulate == 0)) {
                ok = warp_mbar_wait(&aux->tempty[buf], bph ^ 1u, abort_flag);
                if (ok) {
                  tc_fence_after();
                  cur = buf;
                  accumulate = 0;
                  if (++buf == C::NBUF) {
                    buf = 0;
                    bph ^= 1u;
                  }
                }
              }
              if (ok) {
                ++chunk_pos;
                --k32_left;
                const bool last_of_chunk = chunk_pos == p.chunk_k32 || k32_left == 0;
                tc_mma1<F8 ? 1 : 0>(tmem_base + cur * C::BN, adesc + static_cast<uint64_t>(j * 2),
                                    bdesc + static_cast<uint64_t>(j * 2), idesc, accumulate);
                if (last_of_chunk) tc_commit_elect(&aux->tfull[cur]);
                accumulate = 1;
                if (last_of_chunk) chunk_pos = 0;
              }
            }
          }
          if (ok) tc_commit_elect(&aux->empty[s]);
        }
        ready = warp_mbar_test_end(peek);
        s = ns;
        ph = nph;
      }
    }
    if (!ok && lane == 0) {
      timed_out = !*abort_flag;
      *abort_flag = 1;
    }
    // Nothing may still be reading shared memory or writing TMEM when the CTA retires.
    tc_commit_elect(&aux->drain);
    mbar_wait_drain(&aux->drain, 0);
    __syncwarp();
  } else if constexpr (TILED) {
    // ------------------------------------------------------------------ epilogue warps, tiled stores
    const int q = warp & 3;
    const int half = warp >> 2;  // column half of this warp
    TilePart part;
    part.tmap_d = &tmap_d;
    part.stage = smem + C::OUT_OFFSET + warp * kStageOutBytes;
    part.cols = C::COLS_PER_WARP;
    part.lane = lane;
    part.rs = part.cst = 1.0f;
    part.cs = aux->cs + half * C::COLS_PER_WARP;
    part.bias = aux->bias + half * C::COLS_PER_WARP;
    const bool staged = p.chain != kChainRaw && p.chain != kChainAcc16Tensor;  // the chain takes a scale or bias per column
    uint32_t ebuf = 0, ebph = 0, piece = 0;
    bool ok = true;
    TileScales next;
    auto prefetch = [&](int t) {
      if (!staged || t >= num_tiles) return;
      int mb, nb;
      tile_coords(BATCHED ? t % per_batch : t, p.num_m, p.num_n, mb, nb);
      next = fetch_scales(p, nb * C::BN + half * C::COLS_PER_WARP + static_cast<int>(threadIdx.x & 127), (threadIdx.x & 127) < C::COLS_PER_WARP, mb * kBM + q * 32 + lane);
    };
    griddep_wait();  // the row scales may come from the launch before
    if (p.chain == kChainAcc16Tensor) {
      part.rs = p.rs != nullptr ? *p.rs : 1.0f;
      part.cst = p.cs != nullptr ? *p.cs : 1.0f;
    }
    prefetch(blockIdx.x);
    int t = blockIdx.x;
    for (; t < num_tiles && ok; t += gridDim.x) {
      int mb, nb;
      const int bi = BATCHED ? t / per_batch : 0;
      tile_coords(t - bi * per_batch, p.num_m, p.num_n, mb, nb);
      if (staged) {
        // Stage the column scales and bias of this half once; all lanes then read them as broadcasts.
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        if ((threadIdx.x & 127) < C::COLS_PER_WARP) {
          aux->cs[half * C::COLS_PER_WARP + (threadIdx.x & 127)] = next.cs;
          aux->bias[half * C::COLS_PER_WARP + (threadIdx.x & 127)] = next.bias;
        }
        part.rs = next.rs;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        prefetch(t + gridDim.x);
      }
      const uint32_t buf = ebuf, bph = ebph;
      if (++ebuf == C::NBUF) {
        ebuf = 0;
        ebph ^= 1u;
      }
      if (!warp_mbar_wait(&aux->tfull[buf], bph, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after();
      part.taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * C::BN + half * C::COLS_PER_WARP;
      part.row0 = mb * kBM + q * 32;
      part.col0 = nb * C::BN + half * C::COLS_PER_WARP;
      part.bi = bi;
      drain_tile_any<F8>(p, part, piece, [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&aux->tempty[buf]);
      });
    }
    if (lane == 0) tma_store_wait_read<0>();  // the stores read this CTA's shared memory
    if (!ok && lane == 0) {
      timed_out = !*abort_flag;
      *abort_flag = 1;
    }
    // a warp that gave up still takes part in the barriers of the tiles that are left: another may have seen its accumulator
    // complete a moment before the abort and be on its way to them
    if (!ok && staged)
      for (t += gridDim.x; t < num_tiles; t += gridDim.x) {
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
      }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    const int q = warp & 3;
    const int half = warp >> 2;  // column slice of this warp
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    EpiCtx epi = make_epi_ctx(p, smem + C::OUT_OFFSET + warp * kStageOutBytes);
    const bool clamp = !F8 && p.max_acc_bits < 32;
    const int32_t lo = clamp ? -(1 << (p.max_acc_bits - 1)) : 0;
    const int32_t hi = clamp ? (1 << (p.max_acc_bits - 1)) - 1 : 0;
    const uint32_t rb = p.trun_bits > 0 ? (1u << (p.trun_bits - 1)) : 0u;
    const uint32_t mask = p.trun_bits > 0 ? ~((1u << p.trun_bits) - 1u) : 0xFFFFFFFFu;
    const bool dl16 = F8 && p.clamp_dl16;
    const bool scaled = epi.scaled;
    uint32_t ebuf = 0, ebph = 0;
    bool eready = false;
    bool ok = true;
    const bool elow = low_mode;
    const uint32_t enbuf = elow ? C::NBUF - 1 : C::NBUF;
    uint32_t tot_ph = 0;
    TileScales next;
    auto prefetch = [&](int t) {
      if (!scaled || t >= num_tiles) return;
      int mb, nb;
      tile_coords(BATCHED ? t % per_batch : t, p.num_m, p.num_n, mb, nb);
      next = fetch_scales(p, nb * C::BN + static_cast<int>(threadIdx.x), static_cast<int>(threadIdx.x) < C::BN, mb * kBM + q * 32 + lane);
    };
    griddep_wait();  // the row scales may come from the launch before
    prefetch(blockIdx.x);
    int t = blockIdx.x;
    for (; t < num_tiles && ok; t += gridDim.x) {
      int mb, nb;
      const int bi = BATCHED ? t / per_batch : 0;
      tile_coords(t - bi * per_batch, p.num_m, p.num_n, mb, nb);
      if (BATCHED) epi.dbase = static_cast<uint8_t*>(p.d) + static_cast<int64_t>(bi) * p.batch_stride_d * (epi.two_byte ? 2 : 4);
      const int row0 = mb * kBM + q * 32;
      const int row = row0 + lane;
      const int col_w = nb * C::BN + half * C::COLS_PER_WARP;
      float rs = 1.0f;
      if (scaled) {
        // Stage this tile's column scales and bias once; all lanes then read them as broadcasts.
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_WARPS * 32) : "memory");
        if (static_cast<int>(threadIdx.x) < C::BN) {
          aux->cs[threadIdx.x] = next.cs;
          aux->bias[threadIdx.x] = next.bias;
        }
        rs = next.rs;
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_WARPS * 32) : "memory");
        prefetch(t + gridDim.x);
      }
      if constexpr (!CHUNKED) {
        const uint32_t buf = ebuf, bph = ebph;
        if (++ebuf == C::NBUF) {
          ebuf = 0;
          ebph ^= 1u;
        }
        if (!warp_mbar_wait(&aux->tfull[buf], bph, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll 1
        for (int j = 0; j < C::COLS_PER_WARP; j += 64) {
          const int off = half * C::COLS_PER_WARP + j;
          uint32_t lo[32], hi[32];
          tmem_ld64(tmem_base + lane_base + buf * C::BN + off, lo, hi);
          if (p.c != nullptr) {
            uint32_t cv[32];
            load_c_row<32>(p, cv, row, col_w + j);
#pragma unroll
            for (int i = 0; i < 32; ++i) lo[i] = acc_add<F8>(cv[i], lo[i]);
            load_c_row<32>(p, cv, row, col_w + j + 32);
#pragma unroll
            for (int i = 0; i < 32; ++i) hi[i] = acc_add<F8>(cv[i], hi[i]);
          }
          emit64<F8>(p, epi, lo, hi, row0, lane, col_w + j, aux->cs + off, aux->bias + off, rs);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&aux->tempty[buf]);
      } else {
        uint32_t run[C::COLS_PER_WARP];
        load_c_row<C::COLS_PER_WARP>(p, run, row, col_w);
        int k32_left = total_k32;
#pragma unroll 1
        while (k32_left > 0) {
          k32_left -= p.chunk_k32;
          const uint32_t buf = ebuf, bph = ebph;
          if (++ebuf == enbuf) {
            ebuf = 0;
            ebph ^= 1u;
          }
          if (!eready && !warp_mbar_wait(&aux->tfull[buf], bph, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (elow) {
            // ((p + 128) >> 8) << 8 = p - sext8(low byte of p): the sum of the chunks is the untruncated total (kept by
            // the tensor core in its own accumulator) minus the sum of the sign-extended low bytes.  Only the low bits
            // of the chunk's accumulator are read (two columns per register), one dp4a per element picks its byte.
            uint32_t v16[C::COLS_PER_WARP / 2];
            tmem_ld32_low16(tmem_base + lane_base + buf * C::BN + half * C::COLS_PER_WARP, v16);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&aux->tempty[buf]);
            const uint32_t epeek = warp_mbar_test_begin(&aux->tfull[ebuf], ebph);
#pragma unroll
            for (int i = 0; i < C::COLS_PER_WARP / 2; ++i) {
              run[2 * i] = static_cast<uint32_t>(__dp4a(static_cast<int>(v16[i]), 0x000000FF, static_cast<int>(run[2 * i])));
              run[2 * i + 1] = static_cast<uint32_t>(__dp4a(static_cast<int>(v16[i]), 0x00FF0000, static_cast<int>(run[2 * i + 1])));
            }
            eready = warp_mbar_test_end(epeek);
            continue;
          }
          uint32_t v[C::COLS_PER_WARP];
          tmem_ld32(tmem_base + lane_base + buf * C::BN + half * C::COLS_PER_WARP, v);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&aux->tempty[buf]);
          // poll the next chunk's barrier now; the answer is consumed after this chunk's arithmetic
          const uint32_t epeek = warp_mbar_test_begin(&aux->tfull[ebuf], ebph);
          if (p.trunc_then_acc && !clamp && !dl16) {
            // the common case, kept free of per-element predicates: run += (p + rb) & mask
#pragma unroll
            for (int i = 0; i < C::COLS_PER_WARP; ++i) run[i] = acc_add<F8>(run[i], (v[i] + rb) & mask);
          } else if (p.trunc_then_acc) {
#pragma unroll
            for (int i = 0; i < C::COLS_PER_WARP; ++i)
              run[i] = acc_add<F8>(run[i], chunk_round<F8>(v[i], clamp, lo, hi, rb, mask, dl16));
          } else {
#pragma unroll
            for (int i = 0; i < C::COLS_PER_WARP; ++i)
              run[i] = chunk_round<F8>(acc_add<F8>(run[i], v[i]), clamp, lo, hi, rb, mask, dl16);
          }
          eready = warp_mbar_test_end(epeek);
        }
        if (!ok) break;
        if (elow) {
          if (!warp_mbar_wait(&aux->tfull[C::NBUF - 1], tot_ph, abort_flag)) {
            ok = false;
            break;
          }
          tot_ph ^= 1u;
          tc_fence_after();
          uint32_t tot[C::COLS_PER_WARP];
          tmem_ld32(tmem_base + lane_base + (C::NBUF - 1) * C::BN + half * C::COLS_PER_WARP, tot);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&aux->tempty[C::NBUF - 1]);
#pragma unroll
          for (int i = 0; i < C::COLS_PER_WARP; ++i) run[i] += tot[i];
        }
        if (!ok) break;
        emit32<F8>(p, epi, run, row0, lane, col_w, aux->cs + half * C::COLS_PER_WARP, aux->bias + half * C::COLS_PER_WARP, rs);
      }
    }
    if (!ok && lane == 0) {
      timed_out = !*abort_flag;
      *abort_flag = 1;
    }
    // a warp that gave up still takes part in the barriers of the tiles that are left: another may have seen its accumulator
    // complete a moment before the abort and be on its way to them
    if (!ok && scaled)
      for (t += gridDim.x; t < num_tiles; t += gridDim.x) {
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_WARPS * 32) : "memory");
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_WARPS * 32) : "memory");
      }
  }

  if (timed_out && p.status != nullptr) atomicExch(p.status, static_cast<int32_t>(QLIN_ERR_TIMEOUT));
  tc_fence_before();
  __syncthreads();
  if (warp == C::MMA_WARP) {
    __syncwarp();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------------------------------------
// CTA-pair variant of the unchunked kernel (cta_group::2).  A cluster of two CTAs computes a
// 256 x 256 tile: CTA r of the pair loads rows [128 r, 128 r + 128) of the A tile and of the B tile
// into its own shared memory (32 KB per stage instead of 48 KB for the same MMA work per SM, so six
// stages fit and the L2 -> SM traffic per operation drops by a third), the even CTA issues the MMAs
// for both, and each CTA drains its own 128 accumulator rows.  Barriers:
//   full[s]   leader's copy: 1 arrival (the leader's expect_tx) + the bytes of both CTAs' loads
//   empty[s]  every CTA's own copy, arrived on by the leader's commit (two-CTA mask)
//   tfull[b]  every CTA's own copy, arrived on by the leader's commit (two-CTA mask)
//   tempty[b] leader's copy: one arrival per epilogue warp of both CTAs
// ------------------------------------------------------------------------------------------------
struct PairCfg {
  static constexpr int BN = 256;
  static constexpr int NBUF = 2;
  static constexpr int STAGES = 6;
  static constexpr int EPI_WARPS = 8;
  static constexpr int PRODUCER_WARP = EPI_WARPS;
  static constexpr int MMA_WARP = EPI_WARPS + 1;
  static constexpr int THREADS = (EPI_WARPS + 2) * 32;
  static constexpr int A_BYTES = kBM * kBK;        // this CTA's 128 rows of A
  static constexpr int B_BYTES = (BN / 2) * kBK;   // this CTA's 128 rows of B
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int COLS_PER_WARP = BN / (EPI_WARPS / 4);
  static constexpr int OUT_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int AUX_OFFSET = OUT_OFFSET + EPI_WARPS * kStageOutBytes;
  static constexpr int SMEM_BYTES = AUX_OFFSET + static_cast<int>(sizeof(Aux));
};
static_assert(PairCfg::SMEM_BYTES <= 232448, "shared memory budget");
constexpr int kGroupM2 = 8;  // 256-row blocks per raster group

__device__ __forceinline__ void tile_coords2(int t, int num_m, int num_n, int& mb, int& nb) {
  const int per_group = kGroupM2 * num_n;
  const int g = t / per_group;
  const int first_m = g * kGroupM2;
  const int gsz = min(num_m - first_m, kGroupM2);
  const int r = t - g * per_group;
  mb = first_m + r % gsz;
  nb = r / gsz;
}

template <bool F8, bool TILED>
__global__ void __launch_bounds__(PairCfg::THREADS, 1)
qlin_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ CUtensorMap tmap_d,
                      const GemmParams p) {
  using C = PairCfg;
  extern __shared__ __align__(1024) uint8_t smem[];
  Aux* aux = reinterpret_cast<Aux*>(smem + C::AUX_OFFSET);
  volatile int* abort_flag = &aux->abort_flag;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const bool aligned = (smem_u32(smem) & 1023u) == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&aux->full[s], 1);
      mbar_init(&aux->empty[s], 1);
    }
    for (int b = 0; b < C::NBUF; ++b) {
      mbar_init(&aux->tfull[b], 1);
      mbar_init(&aux->tempty[b], 2 * C::EPI_WARPS);
    }
    mbar_init(&aux->drain, 1);
    aux->abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == C::MMA_WARP) {
    tmem_alloc_pair(&aux->tmem_base, kTmemCols);
    tmem_relinquish_pair();
  }
  if (warp == C::PRODUCER_WARP && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    if (TILED) tma_prefetch_desc(&tmap_d);
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive_wait();  // both CTAs' barriers exist before either touches the other's
  tc_fence_after();
  const uint32_t tmem_base = aux->tmem_base;

  const int num_m2 = (p.M + 2 * kBM - 1) / (2 * kBM);
  const int num_tiles = num_m2 * p.num_n;
  const int num_kb = (p.kbytes + kBK - 1) / kBK;
  const int total_k32 = (p.kbytes + 31) / 32;
  bool timed_out = false;

  if (!aligned) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, static_cast<int32_t>(QLIN_ERR_BAD_ALIGN));
  } else if (warp == C::PRODUCER_WARP) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    griddep_wait();
    uint32_t s = 0, ph = 0;
    bool ok = true, ready = false;
    for (int t = pair; t < num_tiles && ok; t += num_pairs) {
      int mb, nb;
      tile_coords2(t, num_m2, p.num_n, mb, nb);
      const int ya = mb * 2 * kBM + static_cast<int>(rank) * kBM;
      const int yb = nb * C::BN + static_cast<int>(rank) * (C::BN / 2);
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!ready) {
          ok = warp_mbar_wait(&aux->empty[s], ph ^ 1u, abort_flag);
          if (!ok) break;
        }
        const uint32_t ns = (s + 1 == C::STAGES) ? 0u : s + 1;
        const uint32_t nph = (ns == 0u) ? (ph ^ 1u) : ph;
        const uint32_t peek = warp_mbar_test_begin(&aux->empty[ns], nph ^ 1u);
        uint8_t* sa = smem + s * C::STAGE_BYTES;
        tma_issue_stage_pair(map_to_cta(&aux->full[s], 0), leader, 2 * C::STAGE_BYTES, sa, &tmap_a, ya, sa + C::A_BYTES, &tmap_b, yb,
                             kb * kBK);
        ready = warp_mbar_test_end(peek);
        s = ns;
        ph = nph;
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
      const uint32_t idesc = F8 ? make_idesc(1u, static_cast<uint32_t>(p.f8_ab_format), 2 * kBM, C::BN) : make_idesc(2u, 1u, 2 * kBM, C::BN);
      const uint64_t adesc0 = make_smem_desc_sw128(smem_u32(smem));
      const uint64_t bdesc0 = make_smem_desc_sw128(smem_u32(smem) + C::A_BYTES);
      uint32_t s = 0, ph = 0, buf = 0, bph = 0;
      bool ok = true, ready = false;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        uint32_t accumulate = 0, cur = 0;
        int k32_left = total_k32;
        for (int kb = 0; kb < num_kb && ok; ++kb) {
          if (!ready) {
            ok = warp_mbar_wait(&aux->full[s], ph, abort_flag);
            if (!ok) break;
          }
          tc_fence_after();
          const uint32_t ns = (s + 1 == C::STAGES) ? 0u : s + 1;
          const uint32_t nph = (ns == 0u) ? (ph ^ 1u) : ph;
          const uint32_t peek = warp_mbar_test_begin(&aux->full[ns], nph);
          const uint64_t adesc = adesc0 + static_cast<uint64_t>(s * (C::STAGE_BYTES >> 4));
          const uint64_t bdesc = bdesc0 + static_cast<uint64_t>(s * (C::STAGE_BYTES >> 4));
          if (kb == 0) {
            ok = warp_mbar_wait(&aux->tempty[buf], bph ^ 1u, abort_flag);
            if (!ok) break;
            tc_fence_after();
            cur = buf;
            if (++buf == C::NBUF) {
              buf = 0;
              bph ^= 1u;
            }
          }
          if (k32_left >= 4) {
            tc_mma4_release_pair<F8 ? 1 : 0>(tmem_base + cur * C::BN, adesc, bdesc, idesc, accumulate, &aux->empty[s]);
            accumulate = 1;
            k32_left -= 4;
          } else {
            for (int j = 0; j < k32_left; ++j) {
              tc_mma1_pair<F8 ? 1 : 0>(tmem_base + cur * C::BN, adesc + static_cast<uint64_t>(j * 2), bdesc + static_cast<uint64_t>(j * 2),
                                       idesc, accumulate);
              accumulate = 1;
            }
            k32_left = 0;
            tc_commit_pair_elect(&aux->empty[s]);
          }
          if (k32_left == 0) tc_commit_pair_elect(&aux->tfull[cur]);
          ready = warp_mbar_test_end(peek);
          s = ns;
          ph = nph;
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
  } else if constexpr (TILED) {
    // ------------------------------------------------------------------ epilogue warps (both CTAs), tiled stores
    const int q = warp & 3;
    const int half = warp >> 2;  // column half of this warp
    TilePart part;
    part.tmap_d = &tmap_d;
    part.stage = smem + C::OUT_OFFSET + warp * kStageOutBytes;
    part.cols = C::COLS_PER_WARP;
    part.lane = lane;
    part.rs = part.cst = 1.0f;
    part.cs = aux->cs + half * C::COLS_PER_WARP;
    part.bias = aux->bias + half * C::COLS_PER_WARP;
    const bool staged = p.chain != kChainRaw && p.chain != kChainAcc16Tensor;  // the chain takes a scale or bias per column
    uint32_t ebuf = 0, ebph = 0, piece = 0;
    bool ok = true;
    TileScales next;
    auto prefetch = [&](int t) {
      if (!staged || t >= num_tiles) return;
      int mb, nb;
      tile_coords2(t, num_m2, p.num_n, mb, nb);
      next = fetch_scales(p, nb * C::BN + static_cast<int>(threadIdx.x), true, mb * 2 * kBM + static_cast<int>(rank) * kBM + q * 32 + lane);
    };
    griddep_wait();  // the row scales may come from the launch before
    if (p.chain == kChainAcc16Tensor) {
      part.rs = p.rs != nullptr ? *p.rs : 1.0f;
      part.cst = p.cs != nullptr ? *p.cs : 1.0f;
    }
    prefetch(pair);
    int t = pair;
    for (; t < num_tiles && ok; t += num_pairs) {
      int mb, nb;
      tile_coords2(t, num_m2, p.num_n, mb, nb);
      if (staged) {
        // Stage the column scales and bias of this half once; all lanes then read them as broadcasts.
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        aux->cs[threadIdx.x] = next.cs;
        aux->bias[threadIdx.x] = next.bias;
        part.rs = next.rs;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        prefetch(t + num_pairs);
      }
      const uint32_t buf = ebuf, bph = ebph;
      if (++ebuf == C::NBUF) {
        ebuf = 0;
        ebph ^= 1u;
      }
      if (!warp_mbar_wait(&aux->tfull[buf], bph, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after();
      part.taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * C::BN + half * C::COLS_PER_WARP;
      part.row0 = mb * 2 * kBM + static_cast<int>(rank) * kBM + q * 32;
      part.col0 = nb * C::BN + half * C::COLS_PER_WARP;
      part.bi = 0;
      drain_tile_any<F8>(p, part, piece, [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(&aux->tempty[buf], 0));
      });
    }
    if (lane == 0) tma_store_wait_read<0>();  // the stores read this CTA's shared memory
    if (!ok && lane == 0) {
      timed_out = !*abort_flag;
      *abort_flag = 1;
    }
    // a warp that gave up still takes part in the barriers of the tiles that are left: another may have seen its accumulator
    // complete a moment before the abort and be on its way to them
    if (!ok && staged)
      for (t += num_pairs; t < num_tiles; t += num_pairs) {
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
      }
  } else {
    // ------------------------------------------------------------------ epilogue warps (both CTAs)
    const int q = warp & 3;
    const int half = warp >> 2;
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    const EpiCtx epi = make_epi_ctx(p, smem + C::OUT_OFFSET + warp * kStageOutBytes);
    const bool scaled = epi.scaled;
    uint32_t ebuf = 0, ebph = 0;
    bool ok = true;
    TileScales next;
    auto prefetch = [&](int t) {
      if (!scaled || t >= num_tiles) return;
      int mb, nb;
      tile_coords2(t, num_m2, p.num_n, mb, nb);
      next = fetch_scales(p, nb * C::BN + static_cast<int>(threadIdx.x), static_cast<int>(threadIdx.x) < C::BN,
                          mb * 2 * kBM + static_cast<int>(rank) * kBM + q * 32 + lane);
    };
    griddep_wait();  // the row scales may come from the launch before
    prefetch(pair);
    int t = pair;
    for (; t < num_tiles && ok; t += num_pairs) {
      int mb, nb;
      tile_coords2(t, num_m2, p.num_n, mb, nb);
      const int row0 = mb * 2 * kBM + static_cast<int>(rank) * kBM + q * 32;
      const int row = row0 + lane;
      const int col_w = nb * C::BN + half * C::COLS_PER_WARP;
      float rs = 1.0f;
      if (scaled) {
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_WARPS * 32) : "memory");
        if (static_cast<int>(threadIdx.x) < C::BN) {
          aux->cs[threadIdx.x] = next.cs;
          aux->bias[threadIdx.x] = next.bias;
        }
        rs = next.rs;
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_WARPS * 32) : "memory");
        prefetch(t + num_pairs);
      }
      const uint32_t buf = ebuf, bph = ebph;
      if (++ebuf == C::NBUF) {
        ebuf = 0;
        ebph ^= 1u;
      }
      if (!warp_mbar_wait(&aux->tfull[buf], bph, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll 1
      for (int j = 0; j < C::COLS_PER_WARP; j += 64) {
        const int off = half * C::COLS_PER_WARP + j;
        uint32_t lo[32], hi[32];
        tmem_ld64(tmem_base + lane_base + buf * C::BN + off, lo, hi);
        if (p.c != nullptr) {
          uint32_t cv[32];
          load_c_row<32>(p, cv, row, col_w + j);
#pragma unroll
          for (int i = 0; i < 32; ++i) lo[i] = acc_add<F8>(cv[i], lo[i]);
          load_c_row<32>(p, cv, row, col_w + j + 32);
#pragma unroll
          for (int i = 0; i < 32; ++i) hi[i] = acc_add<F8>(cv[i], hi[i]);
        }
        emit64<F8>(p, epi, lo, hi, row0, lane, col_w + j, aux->cs + off, aux->bias + off, rs);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(&aux->tempty[buf], 0));
    }
    if (!ok && lane == 0) {
      timed_out = !*abort_flag;
      *abort_flag = 1;
    }
    // a warp that gave up still takes part in the barriers of the tiles that are left: another may have seen its accumulator
    // complete a moment before the abort and be on its way to them
    if (!ok && scaled)
      for (t += num_pairs; t < num_tiles; t += num_pairs) {
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_WARPS * 32) : "memory");
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_WARPS * 32) : "memory");
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
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------------------------------------
// Few-row kernel (M <= 128, unchunked): the decode-time shapes, where the weight matrix is read once
// and everything else is small.  The operands swap roles: 128 rows of the WEIGHT are the MMA's M
// dimension and the M activation rows, padded to a multiple of 32, are its N dimension, so a K block
// costs 128 x MT x 128 multiply-adds of tensor time instead of the 128 x 256 x 128 a weight-as-B tile
// costs whatever M is, and the kernel runs at the rate the weights stream in.  One CTA per
// (128 output channels, K split); the CTAs of one channel block form a cluster, park their partial
// accumulators in their own shared memory, and after a cluster barrier CTA r sums rows r, r+S, ...
// over the splits in split order through distributed shared memory (a fixed order: the result does not
// depend on scheduling), dequantises and stores them.  Accumulator lane = output channel, so the
// stores of one row are contiguous across the warp.
// Launched as the dependent of the row quantiser, the producer fills the stages with weights before it waits for the
// codes.  Quantiser and GEMM, bf16 in and out, one after the other -> as a pair: 1 x 4096 x 14336 23.1 -> 18.7 us, 37 x 14336 x
// 4096 24.7 -> 20.6, 517 x 4096 x 4096 (CTA-pair kernel) 25.8 -> 23.2.  The weights of one launch stream at 4.3 TB/s; tiles of
// 104 rows on 138 SMs instead of 128 on 112, other K orders per CTA, other L2 promotions and two smaller CTAs per SM
// were measured within 0.4 us of this at 58.7 MB.
//   warps 0-3  epilogue (TMEM lanes 32 w ..), warp 4 TMA producer, warp 5 MMA issuer / TMEM owner
// ------------------------------------------------------------------------------------------------
constexpr int kSkEpiWarps = 8;  // warp w reads TMEM lanes 32 (w % 4) .., half w / 4 of the 32-row groups
constexpr int kSkProducerWarp = kSkEpiWarps;
constexpr int kSkMmaWarp = kSkEpiWarps + 1;
constexpr int kSkThreads = (kSkEpiWarps + 2) * 32;
constexpr int kSkWBytes = kBM * kBK;  // 128 weight rows x 128 bytes of K per stage
constexpr int kSkTmemCols = 128;

template <bool F8>
__device__ __forceinline__ void skinny_emit(const GemmParams& p, uint32_t v, int m, int n, float rs, float cs, float bias,
                                            bool prod, bool has_bias) {
  if (p.c != nullptr) v = acc_add<F8>(reinterpret_cast<const uint32_t*>(p.c)[static_cast<int64_t>(m) * p.ldc + n], v);
  if (p.epilogue == QLIN_EPI_RAW) {
    reinterpret_cast<uint32_t*>(p.d)[static_cast<int64_t>(m) * p.ldd + n] = v;
    return;
  }
  const float y = dequant_one<F8>(p, v, rs, cs, bias, prod, has_bias);
  if (p.out_dtype == QLIN_DT_F32) {
    reinterpret_cast<float*>(p.d)[static_cast<int64_t>(m) * p.ldd + n] = y;
  } else {
    reinterpret_cast<uint16_t*>(p.d)[static_cast<int64_t>(m) * p.ldd + n] = static_cast<uint16_t>(pack16(p, y, 0.0f) & 0xFFFFu);
  }
}

// Sum of one accumulator element over the NS splits, in split order; the loads are issued together.
template <bool F8, int NS>
__device__ __forceinline__ uint32_t skinny_sum_splits(const uint32_t* src) {
  uint32_t t[NS];
#pragma unroll
  for (int q = 0; q < NS; ++q) t[q] = ld_cluster_u32(map_to_cta(src, static_cast<uint32_t>(q)));
  uint32_t acc = t[0];
#pragma unroll
  for (int q = 1; q < NS; ++q) acc = acc_add<F8>(acc, t[q]);
  return acc;
}

template <bool F8>
__global__ void __launch_bounds__(kSkThreads, 1)
qlin_gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                        const GemmParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int MT = p.sk_mt, S = p.sk_split, STG = p.sk_stages;
  const int stage_bytes = kSkWBytes + MT * kBK;
  Aux* aux = reinterpret_cast<Aux*>(smem + STG * stage_bytes);
  volatile int* abort_flag = &aux->abort_flag;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tile = blockIdx.x / S;
  const int sp = S > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  const int num_kb = (p.kbytes + kBK - 1) / kBK;
  const int kb0 = static_cast<int>(static_cast<int64_t>(sp) * num_kb / S);
  const int kb1 = static_cast<int>(static_cast<int64_t>(sp + 1) * num_kb / S);
  const bool scaled = p.epilogue != QLIN_EPI_RAW;
  const bool prod = p.epilogue == QLIN_EPI_SCALE_PROD;
  const bool has_bias = p.bias != nullptr;

  // Every thread of every CTA of the cluster reaches the two cluster barriers below, whatever happens before them.
  const bool bad = (smem_u32(smem) & 1023u) != 0;
  if (bad && threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, static_cast<int32_t>(QLIN_ERR_BAD_ALIGN));

  if (threadIdx.x == 0) {
    for (int s = 0; s < STG; ++s) {
      mbar_init(&aux->full[s], 1);
      mbar_init(&aux->empty[s], 1);
    }
    mbar_init(&aux->tfull[0], 1);
    mbar_init(&aux->drain, 1);
    aux->abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == kSkMmaWarp) {
    tmem_alloc(&aux->tmem_base, kSkTmemCols);
    tmem_relinquish();
  }
  if (warp == kSkProducerWarp && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = aux->tmem_base;
  bool timed_out = false;
  float* s_rs = aux->cs;  // the row scales of the (at most 128) activation rows, read by every epilogue thread
  uint32_t* part = reinterpret_cast<uint32_t*>(smem);  // [MT][128] partial accumulators, over the drained pipeline stages

  if (bad) {
    // nothing: fall through to the barriers
  } else if (warp == kSkProducerWarp) {
    // ------------------------------------------------------------------ TMA producer
    uint32_t s = 0, ph = 0, issued = 0;
    bool ok = true;
    const uint32_t tx = static_cast<uint32_t>(stage_bytes);
    const int pre = min(STG, kb1 - kb0);  // the first fill of the stages: weights now, activations once they are there
    for (int i = 0; i < pre; ++i) tma_issue_first(&aux->full[i], tx, smem + i * stage_bytes, &tmap_w, tile * kBM, (kb0 + i) * kBK);
    griddep_wait();
    for (int i = 0; i < pre; ++i) tma_issue_second(&aux->full[i], smem + i * stage_bytes + kSkWBytes, &tmap_x, 0, (kb0 + i) * kBK);
    issued = static_cast<uint32_t>(pre);
    if (pre == STG) ph = 1;
    for (int kb = kb0 + pre; kb < kb1; ++kb) {
      ok = warp_mbar_wait(&aux->empty[s], ph ^ 1u, abort_flag);
      if (!ok) break;
      uint8_t* sa = smem + s * stage_bytes;
      tma_issue_stage(&aux->full[s], tx, sa, &tmap_w, tile * kBM, sa + kSkWBytes, &tmap_x, 0, kb * kBK);
      ++issued;
      if (++s == static_cast<uint32_t>(STG)) {
        s = 0;
        ph ^= 1u;
      }
    }
    if (!ok) {
      if (lane == 0) {
        timed_out = !*abort_flag;
        *abort_flag = 1;
      }
      for (uint32_t st = 0; st < static_cast<uint32_t>(STG); ++st) {
        if (issued <= st) continue;
        const uint32_t last = (issued - 1 - st) / static_cast<uint32_t>(STG);
        mbar_wait_drain(&aux->full[st], last & 1u);
      }
    }
    __syncwarp();
  } else if (warp == kSkMmaWarp) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t idesc = F8 ? make_idesc(1u, static_cast<uint32_t>(p.f8_ab_format), kBM, static_cast<uint32_t>(MT))
                              : make_idesc(2u, 1u, kBM, static_cast<uint32_t>(MT));
    const uint64_t wdesc0 = make_smem_desc_sw128(smem_u32(smem));
    const uint64_t xdesc0 = make_smem_desc_sw128(smem_u32(smem) + kSkWBytes);
    uint32_t s = 0, ph = 0, accumulate = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      ok = warp_mbar_wait(&aux->full[s], ph, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const uint64_t off = static_cast<uint64_t>(s * (stage_bytes >> 4));
      tc_mma4_release<F8 ? 1 : 0>(tmem_base, wdesc0 + off, xdesc0 + off, idesc, accumulate, &aux->empty[s]);
      accumulate = 1;
      if (++s == static_cast<uint32_t>(STG)) {
        s = 0;
        ph ^= 1u;
      }
    }
    if (ok) tc_commit_elect(&aux->tfull[0]);
    if (!ok && lane == 0) {
      timed_out = !*abort_flag;
      *abort_flag = 1;
    }
    tc_commit_elect(&aux->drain);
    mbar_wait_drain(&aux->drain, 0);
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue warps, first half
    const int q = warp & 3;
    const int n_local = q * 32 + lane;
    const int n = tile * kBM + n_local;
    griddep_wait();
    if (static_cast<int>(threadIdx.x) < MT)
      s_rs[threadIdx.x] = (scaled && p.rs != nullptr && static_cast<int>(threadIdx.x) < p.M) ? p.rs[static_cast<int64_t>(threadIdx.x) * p.rs_stride] : 1.0f;
    asm volatile("bar.sync 1, %0;" ::"n"(kSkEpiWarps * 32) : "memory");
    if (warp_mbar_wait(&aux->tfull[0], 0, abort_flag)) {
      tc_fence_after();
      const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
      float cs = 1.0f, bias = 0.0f;
      if (S == 1 && n < p.N && scaled) {
        if (p.cs != nullptr) cs = p.cs[static_cast<int64_t>(n) * p.cs_stride];
        if (has_bias) bias = p.bias[n];
      }
#pragma unroll 1
      for (int c = (warp >> 2) * 32; c < MT; c += 64) {
        if (c >= p.M) break;
        uint32_t v[32];
        tmem_ld32(tmem_base + lane_base + c, v);
        if (S == 1) {
          if (n < p.N) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (c + j < p.M) skinny_emit<F8>(p, v[j], c + j, n, s_rs[c + j], cs, bias, prod, has_bias);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c + j < p.M) part[(c + j) * kBM + n_local] = v[j];
        }
      }
      tc_fence_before();
    } else if (lane == 0) {
      timed_out = !*abort_flag;
      *abort_flag = 1;
    }
    __syncwarp();
  }

  if (S > 1) {
    __syncwarp();
    cluster_arrive_wait();  // every split's partial tile is in its CTA's shared memory
    if (!bad && warp < kSkEpiWarps) {
      const int n_local = threadIdx.x & (kBM - 1);
      const int n = tile * kBM + n_local;
      if (n < p.N) {
        float cs = 1.0f, bias = 0.0f;
        if (scaled) {
          if (p.cs != nullptr) cs = p.cs[static_cast<int64_t>(n) * p.cs_stride];
          if (has_bias) bias = p.bias[n];
        }
        // this CTA's rows are sp, sp + S, ...; the two halves of the epilogue warps take every other one of them
        // two rows per iteration: both rows' loads are in flight before the first sum is needed
        auto sum_row = [&](int m) -> uint32_t {
          const uint32_t* src = part + m * kBM + n_local;
          if (S == 2) return skinny_sum_splits<F8, 2>(src);
          if (S == 4) return skinny_sum_splits<F8, 4>(src);
          return skinny_sum_splits<F8, 8>(src);
        };
        for (int m = sp + S * static_cast<int>(threadIdx.x >> 7); m < p.M; m += 4 * S) {
          const int m2 = m + 2 * S;
          const uint32_t acc = sum_row(m);
          const uint32_t acc2 = m2 < p.M ? sum_row(m2) : 0u;
          skinny_emit<F8>(p, acc, m, n, s_rs[m], cs, bias, prod, has_bias);
          if (m2 < p.M) skinny_emit<F8>(p, acc2, m2, n, s_rs[m2], cs, bias, prod, has_bias);
        }
      }
    }
    __syncwarp();
    cluster_arrive_wait();  // nobody leaves while a neighbour still reads its shared memory
  }

  if (timed_out && p.status != nullptr) atomicExch(p.status, static_cast<int32_t>(QLIN_ERR_TIMEOUT));
  tc_fence_before();
  __syncthreads();
  if (warp == kSkMmaWarp) {
    __syncwarp();
    tmem_dealloc(tmem_base, kSkTmemCols);
  }
}

// ---------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
  }
  return fn;
}

void* tensor_map_encoder() { return reinterpret_cast<void*>(get_encode_fn()); }

// [rows, kbytes] byte matrix with `ld_bytes` between rows, read in boxes of [box_rows x 128 bytes].
static int make_operand_map(CUtensorMap* tm, const void* base, int64_t rows, int64_t kbytes, int64_t ld_bytes,
                            int box_rows) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return fail(QLIN_ERR_DEVICE, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(kbytes), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld_bytes)};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(kBK), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(QLIN_ERR_BAD_ALIGN, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return QLIN_OK;
}

// The output of `batch` problems as a [batch, M, N] tensor read in pieces of 32 rows x 64 bytes.  Returns false where TMA cannot
// address it (base, row pitch or problem stride off a 16-byte boundary) or rows end inside 16 bytes that are not all theirs.
static bool make_output_map(CUtensorMap* tm, const GemmParams& p) {
  const bool two_byte = p.epilogue != QLIN_EPI_RAW && p.out_dtype != QLIN_DT_F32;
  const int64_t elt = two_byte ? 2 : 4;
  const int64_t pitch = p.ldd * elt, stride = p.batch > 1 ? p.batch_stride_d * elt : pitch * p.M;
  if (!aligned16(p.d) || pitch % 16 != 0 || stride % 16 != 0 || (p.N * elt) % 16 != 0 || stride >= (int64_t{1} << 40) || pitch >= (int64_t{1} << 40)) return false;
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return false;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(p.N), static_cast<cuuint64_t>(p.M), static_cast<cuuint64_t>(p.batch > 1 ? p.batch : 1)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(pitch), static_cast<cuuint64_t>(stride)};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(64 / elt), 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(tm, two_byte ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, p.d, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static bool no_round(int dt) { return dt == QLIN_DT_NONE || dt == QLIN_DT_F32; }

// The compiled epilogue that rounds where this launch's does.
static int32_t pick_chain(const GemmParams& p, bool f8) {
  if (p.epilogue == QLIN_EPI_RAW) return kChainRaw;
  if (p.epilogue == QLIN_EPI_SCALE_PROD && !f8 && p.acc_round == QLIN_DT_F16) {
    if (p.prod_round == QLIN_DT_BF16 && p.scale_round == QLIN_DT_F16 && p.out_dtype == QLIN_DT_BF16) return kChainProdBf16;
    // rounding to fp16 twice is rounding once
    if ((no_round(p.prod_round) || p.prod_round == QLIN_DT_F16) && p.scale_round == QLIN_DT_F16) return kChainProdF16;
  }
  if (p.epilogue == QLIN_EPI_SCALE_SEQ) {
    if (no_round(p.mid_round) && no_round(p.acc_round)) return kChainSeq;
    if (f8 && p.mid_round == QLIN_DT_BF16 && p.acc_round == QLIN_DT_BF16 && p.out_dtype == QLIN_DT_BF16) return kChainSeqBf16;
  }
  if (p.epilogue == QLIN_EPI_SCALE_ACC16 && !f8 && p.rs_stride == 0 && p.cs_stride == 0 && p.bias == nullptr && no_round(p.mid_round) && no_round(p.acc_round))
    return kChainAcc16Tensor;
  return kChainAny;
}

// A launch with a cluster size and, for a GEMM behind its quantiser, the programmatic dependency.
struct LaunchCfg {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  LaunchCfg(int grid, int threads, size_t smem, cudaStream_t stream, int cluster, bool dependent) {
    cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
    cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    if (cluster > 1) {
      attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
      attr[cfg.numAttrs].val.clusterDim.x = static_cast<unsigned>(cluster);
      attr[cfg.numAttrs].val.clusterDim.y = 1;
      attr[cfg.numAttrs].val.clusterDim.z = 1;
      ++cfg.numAttrs;
    }
    if (dependent) {
      attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
      ++cfg.numAttrs;
    }
  }
};

template <bool F8, bool CHUNKED, bool BATCHED, bool TILED, bool SHORT_K>
static int launch_as(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const GemmParams& p, cudaStream_t stream) {
  using C = Cfg<CHUNKED, SHORT_K>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return fail(QLIN_ERR_DEVICE, "device ordinal %d out of range", dev);
  const auto kernel = qlin_gemm_kernel<F8, CHUNKED, BATCHED, TILED, SHORT_K>;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess) return fail(QLIN_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    configured[dev] = true;
  }
  const int64_t tiles = static_cast<int64_t>(p.num_m) * p.num_n * (BATCHED ? p.batch : 1);
  int grid = tiles < sm_count() ? static_cast<int>(tiles) : sm_count();
  if (p.max_ctas > 0 && grid > p.max_ctas) grid = p.max_ctas;
  LaunchCfg lc(grid, C::THREADS, C::SMEM_BYTES, stream, 1, p.dependent != 0);
  const cudaError_t le = cudaLaunchKernelEx(&lc.cfg, kernel, ta, tb, td, p);
  if (le != cudaSuccess) {
    cudaGetLastError();
    return fail(QLIN_ERR_LAUNCH, "qlin_gemm: %s", cudaGetErrorString(le));
  }
  return QLIN_OK;
}
// Batched products that the epilogue bounds: K of three blocks, and of four where there are few tiles of few columns, whose chain of
// columns a warp is then half as long.  Heads x m x k x n, four stages and eight warps -> three and sixteen (us).  bf16 out: 64 x 2048 x
// 128 x 2048 124 -> 102, 64 x 1024 x 256 x 1024 36.5 -> 33.2, 64 x 512 x 512 x 64 10.2 -> 9.9, 64 x 384 x 384 x 128 9.6 -> 8.9, at 64 x 2048 x 384 x
// 2048 139 -> 145 (fp32 out 230 -> 193); but 64 x 1024 x 1024 x 128 20.8 -> 23.2, 64 x 1536 x 1536 x 64 39.4 -> 44.3, 64 x 2048 x 2048 x 64
// 60.9 -> 66.6.
static bool short_batched(const GemmParams& p) {
  const int64_t tiles = static_cast<int64_t>(p.num_m) * p.num_n * p.batch;
  return p.kbytes <= 3 * kBK || (p.kbytes <= 4 * kBK && p.N <= 128 && tiles <= 2 * sm_count());
}

// `td`: the output's map, or null for outputs that TMA does not store.
template <bool F8, bool CHUNKED, bool BATCHED = false>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap* td, const GemmParams& p, cudaStream_t stream) {
  if constexpr (!CHUNKED) {
    if (td != nullptr) {
      if constexpr (BATCHED) {
        if (short_batched(p)) return launch_as<F8, false, true, true, true>(ta, tb, *td, p, stream);
      }
      return launch_as<F8, false, BATCHED, true, false>(ta, tb, *td, p, stream);
    }
  }
  return launch_as<F8, CHUNKED, BATCHED, false, false>(ta, tb, ta, p, stream);
}

// Largest number of two-CTA clusters of the pair kernel that can be resident at once (cached per device).
template <bool F8, bool TILED>
static int pair_max_clusters() {
  static int cached[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 0;
  if (cached[dev] != 0) return cached[dev] > 0 ? cached[dev] : 0;
  cached[dev] = -1;
  const auto kernel = qlin_gemm_pair_kernel<F8, TILED>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg::SMEM_BYTES) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sm_count() & ~1), 1, 1);
  cfg.blockDim = dim3(PairCfg::THREADS, 1, 1);
  cfg.dynamicSmemBytes = PairCfg::SMEM_BYTES;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cached[dev] = n > 0 ? n : -1;
  return n > 0 ? n : 0;
}

template <bool F8, bool TILED>
static int launch_pair_as(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const GemmParams& p, cudaStream_t stream) {
  int clusters = pair_max_clusters<F8, TILED>();
  if (clusters <= 0) return 1;  // not available: the caller takes the single-CTA kernel
  const int tiles = ((p.M + 2 * kBM - 1) / (2 * kBM)) * p.num_n;
  if (clusters > tiles) clusters = tiles;
  if (p.max_ctas > 0 && clusters > p.max_ctas / 2) clusters = p.max_ctas / 2 > 0 ? p.max_ctas / 2 : 1;
  LaunchCfg lc(2 * clusters, PairCfg::THREADS, PairCfg::SMEM_BYTES, stream, 2, p.dependent != 0);
  const cudaError_t e = cudaLaunchKernelEx(&lc.cfg, qlin_gemm_pair_kernel<F8, TILED>, ta, tb, td, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QLIN_ERR_LAUNCH, "qlin_gemm (CTA-pair kernel): %s", cudaGetErrorString(e));
  }
  return QLIN_OK;
}
template <bool F8>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap* td, const GemmParams& p, cudaStream_t stream) {
  return td != nullptr ? launch_pair_as<F8, true>(ta, tb, *td, p, stream) : launch_pair_as<F8, false>(ta, tb, ta, p, stream);
}

// The CTA-pair kernel is used for unchunked problems of at least 256 rows unless QLIN_GEMM_PAIR=0.
static bool pair_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("QLIN_GEMM_PAIR");
    v = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

static bool low_byte_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("QLIN_GEMM_LOWBYTE");
    v = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

// The few-row kernel is used for unchunked problems of at most 128 rows unless QLIN_GEMM_SKINNY=0.
static bool skinny_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("QLIN_GEMM_SKINNY");
    v = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

template <bool F8>
static int launch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, GemmParams p, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return fail(QLIN_ERR_DEVICE, "device ordinal %d out of range", dev);
  const int smem_max = 232448;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(qlin_gemm_skinny_kernel<F8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
    if (e != cudaSuccess) return fail(QLIN_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    configured[dev] = true;
  }
  const int stage_bytes = kSkWBytes + p.sk_mt * kBK;
  int stages = (smem_max - static_cast<int>(sizeof(Aux))) / stage_bytes;
  p.sk_stages = stages > 8 ? 8 : stages;
  const int tiles = (p.N + kBM - 1) / kBM;
  // K splits: the largest power of two that keeps one CTA per SM and at least four K blocks per split
  const int num_kb = (p.kbytes + kBK - 1) / kBK;
  int split = 1;
  while (split < 8 && tiles * split * 2 <= sm_count() && num_kb / (split * 2) >= 4) split *= 2;
  p.sk_split = split;
  LaunchCfg lc(tiles * split, kSkThreads, static_cast<size_t>(p.sk_stages) * stage_bytes + sizeof(Aux), stream, split, p.dependent != 0);
  cudaError_t e = cudaLaunchKernelEx(&lc.cfg, qlin_gemm_skinny_kernel<F8>, tw, tx, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QLIN_ERR_LAUNCH, "qlin_gemm (few-row kernel): %s", cudaGetErrorString(e));
  }
  return QLIN_OK;
}

static bool is_round_dtype(int dt) {
  return dt == QLIN_DT_NONE || dt == QLIN_DT_F32 || dt == QLIN_DT_F16 || dt == QLIN_DT_BF16;
}

}  // namespace qlin

using namespace qlin;

// batch > 1: the problems' operands are stacked along the rows (dense), one launch of the batched single-CTA kernel.
// dependent: the launch before on the stream is the row quantiser that writes a->a and a->row_scale (and none of the other operands).
static int gemm_impl(const qlin_gemm_args* a, void* stream, int32_t batch, int64_t stride_d, bool dependent = false) {
  if (a == nullptr) return fail(QLIN_ERR_NULL, "qlin_gemm: args is NULL");
  if (a->a == nullptr || a->b == nullptr || (a->d == nullptr && a->scatter_rows <= 0))
    return fail(QLIN_ERR_NULL, "qlin_gemm: a, b or d is NULL");
  if (a->scatter_rows < 0 || (a->scatter_rows > 0 && a->scatter_rows % 128 != 0))
    return fail(QLIN_ERR_BAD_SHAPE, "qlin_gemm: scatter_rows must be a multiple of 128");
  if (a->scatter_rows > 0) {
    const int64_t owners = (static_cast<int64_t>(a->M) + a->scatter_rows - 1) / a->scatter_rows;
    if (owners > 8) return fail(QLIN_ERR_BAD_SHAPE, "qlin_gemm: more than 8 scatter destinations");
    for (int i = 0; i < owners; ++i) {
      if (a->scatter_d[i] == nullptr) return fail(QLIN_ERR_NULL, "qlin_gemm: scatter_d[%d] is NULL", i);
      if (!aligned16(a->scatter_d[i])) return fail(QLIN_ERR_BAD_ALIGN, "qlin_gemm: scatter_d[%d] is not 16-byte aligned", i);
    }
    if (a->c != nullptr) return fail(QLIN_ERR_UNSUPPORTED, "qlin_gemm: scatter with an accumulator input is not provided");
  }
  if (a->M < 0 || a->N < 0 || a->K < 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_gemm: negative dimension");
  if (a->kind != QLIN_DT_I8 && a->kind != QLIN_DT_F8E4M3 && a->kind != QLIN_DT_F8E5M2)
    return fail(QLIN_ERR_BAD_DTYPE, "qlin_gemm: kind must be QLIN_DT_I8, QLIN_DT_F8E4M3 or QLIN_DT_F8E5M2");
  const bool f8 = a->kind != QLIN_DT_I8;
  if (a->M == 0 || a->N == 0) return QLIN_OK;
  if (a->K == 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_gemm: K must be positive");
  if (a->lda < a->K || a->ldb < a->K || a->ldd < a->N || (a->c != nullptr && a->ldc < a->N))
    return fail(QLIN_ERR_BAD_SHAPE, "qlin_gemm: leading dimension smaller than the row length");
  if (!aligned16(a->a) || !aligned16(a->b) || a->lda % 16 != 0 || a->ldb % 16 != 0)
    return fail(QLIN_ERR_BAD_ALIGN, "qlin_gemm: a and b must be 16-byte aligned with lda, ldb multiples of 16");
  if (a->epilogue == QLIN_EPI_RAW) {
    if (a->out_dtype != (f8 ? QLIN_DT_F32 : QLIN_DT_I32))
      return fail(QLIN_ERR_BAD_DTYPE, "qlin_gemm: raw output is int32 for int8 operands and fp32 for fp8 operands");
  } else if (a->epilogue >= QLIN_EPI_SCALE_PROD && a->epilogue <= QLIN_EPI_SCALE_ACC16) {
    if (a->out_dtype != QLIN_DT_F32 && a->out_dtype != QLIN_DT_F16 && a->out_dtype != QLIN_DT_BF16)
      return fail(QLIN_ERR_BAD_DTYPE, "qlin_gemm: scaled output must be fp32, fp16 or bf16");
    if (!is_round_dtype(a->prod_round) || !is_round_dtype(a->scale_round) || !is_round_dtype(a->mid_round) || !is_round_dtype(a->acc_round))
      return fail(QLIN_ERR_BAD_DTYPE, "qlin_gemm: rounding dtypes must be NONE, F32, F16 or BF16");
    if ((a->row_scale_stride != 0 && a->row_scale_stride != 1) || (a->col_scale_stride != 0 && a->col_scale_stride != 1))
      return fail(QLIN_ERR_BAD_SHAPE, "qlin_gemm: scale strides must be 0 or 1");
  } else {
    return fail(QLIN_ERR_UNSUPPORTED, "qlin_gemm: unknown epilogue %d", a->epilogue);
  }
  if (a->trun_bits < 0 || a->trun_bits > (f8 ? 22 : 31))
    return fail(QLIN_ERR_UNSUPPORTED, "qlin_gemm: trun_bits out of range");
  if (!f8 && (a->max_acc_bits < 2 || a->max_acc_bits > 32))
    return fail(QLIN_ERR_UNSUPPORTED, "qlin_gemm: max_acc_bits must be in [2, 32]");
  if (a->chunk_k > 0 && a->chunk_k % 32 != 0)
    return fail(QLIN_ERR_UNSUPPORTED, "qlin_gemm: chunk_k must be a multiple of 32");

  const bool needs_chunks = (a->trun_bits > 0) || (!f8 && a->max_acc_bits < 32) || (f8 && a->clamp_dl16);
  const bool chunked = needs_chunks;  // without a per-chunk function the chunking is not observable for ints
  const int total_k32 = (a->K + 31) / 32;
  int chunk_k32 = total_k32;
  if (chunked && a->chunk_k > 0 && a->chunk_k < a->K) chunk_k32 = a->chunk_k / 32;

  GemmParams p;
  p.c = a->c;
  p.d = a->d;
  p.rs = a->row_scale;
  p.cs = a->col_scale;
  p.bias = a->bias;
  p.status = a->status;
  p.ldc = a->ldc;
  p.ldd = a->ldd;
  p.M = a->M;
  p.N = a->N;
  p.kbytes = a->K;
  p.chunk_k32 = chunk_k32;
  p.trun_bits = a->trun_bits;
  p.max_acc_bits = f8 ? 32 : a->max_acc_bits;
  p.trunc_then_acc = a->trunc_then_acc;
  p.clamp_dl16 = a->clamp_dl16;
  p.epilogue = a->epilogue;
  p.rs_stride = a->row_scale_stride;
  p.cs_stride = a->col_scale_stride;
  p.prod_round = a->prod_round;
  p.scale_round = a->scale_round;
  p.mid_round = a->mid_round;
  p.acc_round = a->acc_round;
  p.out_dtype = a->out_dtype;
  p.max_ctas = a->max_ctas;
  p.scatter_rows = a->scatter_rows;
  p.scatter_row0 = a->scatter_row0;
  p.f8_ab_format = a->kind == QLIN_DT_F8E5M2 ? 1 : 0;
  for (int i = 0; i < 8; ++i) p.scatter_d[i] = static_cast<uint8_t*>(a->scatter_d[i]);
  const int bn = chunked ? Cfg<true>::BN : Cfg<false>::BN;
  p.num_m = (a->M + kBM - 1) / kBM;
  p.num_n = (a->N + bn - 1) / bn;

  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  p.sk_mt = p.sk_split = p.sk_stages = 0;
  p.dependent = dependent ? 1 : 0;
  p.batch = batch;
  p.batch_stride_d = stride_d;
  // int8 chunks with the low byte rounded away, summed after rounding, no clamp, chunks of 32 / 64 / 128 that tile K:
  // sum of ((p + 128) >> 8 << 8) = sum of p - sum of sext8(p), the first sum kept by the tensor core (QLIN_GEMM_LOWBYTE=0: off)
  p.low_byte_mode = (chunked && !f8 && a->trun_bits == 8 && a->trunc_then_acc && a->max_acc_bits >= 32 &&
                     (chunk_k32 == 1 || chunk_k32 == 2 || chunk_k32 == 4) && total_k32 % 4 == 0 && low_byte_enabled())
                        ? 1
                        : 0;
  // unchunked products whose output TMA can address are stored by it; an accumulator input or row-block scatter keeps emit64, and the
  // few-row kernel stores by itself
  p.chain = pick_chain(p, f8);
  CUtensorMap tmap_d;
  const auto output_map = [&]() -> const CUtensorMap* { return !chunked && p.c == nullptr && p.scatter_rows <= 0 && make_output_map(&tmap_d, p) ? &tmap_d : nullptr; };
  if (batch > 1) {
    if (chunked || a->c != nullptr || a->scatter_rows != 0) return fail(QLIN_ERR_UNSUPPORTED, "qlin_gemm_batched: one launch takes unchunked problems without accumulator input or scatter");
    if (static_cast<int64_t>(batch) * a->M > 0x7fffffff || static_cast<int64_t>(batch) * a->N > 0x7fffffff)
      return fail(QLIN_ERR_BAD_SHAPE, "qlin_gemm_batched: batch * rows exceeds the coordinate range");
    CUtensorMap ta, tb;
    int rc = make_operand_map(&ta, a->a, static_cast<int64_t>(batch) * a->M, a->K, a->lda, kBM);
    if (rc != QLIN_OK) return rc;
    rc = make_operand_map(&tb, a->b, static_cast<int64_t>(batch) * a->N, a->K, a->ldb, bn);
    if (rc != QLIN_OK) return rc;
    return f8 ? launch<true, false, true>(ta, tb, output_map(), p, s) : launch<false, false, true>(ta, tb, output_map(), p, s);
  }
  if (!chunked && a->M <= kBM && a->scatter_rows == 0 && a->max_ctas <= 0 && skinny_enabled()) {
    // weight rows as the MMA's M dimension, the few activation rows (padded to 32) as its N dimension
    p.sk_mt = (a->M + 31) / 32 * 32;
    CUtensorMap tw, tx;
    int rc = make_operand_map(&tw, a->b, a->N, a->K, a->ldb, kBM);
    if (rc != QLIN_OK) return rc;
    rc = make_operand_map(&tx, a->a, a->M, a->K, a->lda, p.sk_mt);
    if (rc != QLIN_OK) return rc;
    rc = f8 ? launch_skinny<true>(tw, tx, p, s) : launch_skinny<false>(tw, tx, p, s);
    // a device that cannot place the cluster (fewer SMs per GPC than the split needs): the wide tile below does the job
    if (rc != QLIN_ERR_LAUNCH) return rc;
    p.sk_mt = p.sk_split = p.sk_stages = 0;
  }

  const CUtensorMap* td = output_map();
  CUtensorMap ta, tb;
  int rc = make_operand_map(&ta, a->a, a->M, a->K, a->lda, kBM);
  if (rc != QLIN_OK) return rc;
  rc = make_operand_map(&tb, a->b, a->N, a->K, a->ldb, bn);
  if (rc != QLIN_OK) return rc;

  if (!chunked && a->M >= 2 * kBM && pair_enabled()) {
    CUtensorMap tb_half;  // each CTA of a pair loads 128 of the tile's 256 B rows
    rc = make_operand_map(&tb_half, a->b, a->N, a->K, a->ldb, PairCfg::BN / 2);
    if (rc != QLIN_OK) return rc;
    rc = f8 ? launch_pair<true>(ta, tb_half, td, p, s) : launch_pair<false>(ta, tb_half, td, p, s);
    if (rc <= 0) return rc;
  }
  if (f8) return chunked ? launch<true, true>(ta, tb, td, p, s) : launch<true, false>(ta, tb, td, p, s);
  return chunked ? launch<false, true>(ta, tb, td, p, s) : launch<false, false>(ta, tb, td, p, s);
}

extern "C" int qlin_gemm(const qlin_gemm_args* a, void* stream) { return gemm_impl(a, stream, 1, 0); }

extern "C" int qlin_quant_gemm(const qlin_quant_args* q, const qlin_scalar_src src[4], const qlin_gemm_args* g, void* stream) {
  if (q == nullptr || g == nullptr) return fail(QLIN_ERR_NULL, "qlin_quant_gemm: args is NULL");
  if (q->codes == nullptr || q->codes != g->a || q->rows != g->M || q->cols != g->K || q->ldq != g->lda)
    return fail(QLIN_ERR_BAD_SHAPE, "qlin_quant_gemm: the quantiser's codes must be the GEMM's a operand");
  if (g->b == q->codes || g->c != nullptr || g->scatter_rows != 0)
    return fail(QLIN_ERR_UNSUPPORTED, "qlin_quant_gemm: no accumulator input and no row-block scatter");
  const int rc = act_quant_impl(q, src, stream);
  if (rc != QLIN_OK) return rc;
  return gemm_impl(g, stream, 1, 0, true);
}

extern "C" int qlin_gemm_batched(const qlin_gemm_args* a, int32_t batch, int64_t stride_a, int64_t stride_b, int64_t stride_d, void* stream) {
  if (a == nullptr) return fail(QLIN_ERR_NULL, "qlin_gemm_batched: args is NULL");
  if (batch < 0 || stride_a < 0 || stride_b < 0 || stride_d < 0) return fail(QLIN_ERR_BAD_SHAPE, "qlin_gemm_batched: negative batch or stride");
  if (a->c != nullptr || a->scatter_rows != 0) return fail(QLIN_ERR_UNSUPPORTED, "qlin_gemm_batched: no accumulator input and no row-block scatter");
  if (batch > 1 && (stride_a % 16 != 0 || stride_b % 16 != 0)) return fail(QLIN_ERR_BAD_ALIGN, "qlin_gemm_batched: operand strides must be multiples of 16 bytes");
  if (batch == 0) return QLIN_OK;
  const int64_t out_elt = (a->epilogue == QLIN_EPI_RAW || a->out_dtype == QLIN_DT_F32) ? 4 : 2;
  const bool needs_chunks = (a->trun_bits > 0) || (a->kind == QLIN_DT_I8 && a->max_acc_bits < 32) || (a->kind != QLIN_DT_I8 && a->clamp_dl16);
  // dense stacks of unchunked problems: one launch whose tiles walk over all problems
  if (batch > 1 && !needs_chunks && stride_a == static_cast<int64_t>(a->M) * a->lda && stride_b == static_cast<int64_t>(a->N) * a->ldb &&
      a->M > 0 && a->N > 0 && static_cast<int64_t>(batch) * a->M <= 0x7fffffff && static_cast<int64_t>(batch) * a->N <= 0x7fffffff)
    return gemm_impl(a, stream, batch, stride_d);
  qlin_gemm_args one = *a;
  for (int32_t i = 0; i < batch; ++i) {
    one.a = static_cast<const uint8_t*>(a->a) + i * stride_a;
    one.b = static_cast<const uint8_t*>(a->b) + i * stride_b;
    one.d = static_cast<uint8_t*>(a->d) + i * stride_d * out_elt;
    const int rc = gemm_impl(&one, stream, 1, 0);
    if (rc != QLIN_OK) return rc;
  }
  return QLIN_OK;
}
