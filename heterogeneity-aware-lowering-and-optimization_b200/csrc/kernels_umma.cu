// NHWC implicit-GEMM convolution and GEMM on the Blackwell tensor cores (sm_100a).
//
//   D[M, K_out] = A[M, R*S*C] * B[K_out, R*S*C]^T       M = N*P*Q output pixels
//
// A is never materialised: a TMA load in im2col mode (cp.async.bulk.tensor.4d...im2col) gathers,
// for one filter tap (r,s) and one chunk of input channels, the 128 input pixels that feed 128
// consecutive output pixels, applying stride and zero padding in hardware.  A 1x1 / stride-1 /
// unpadded convolution and a plain GEMM use an ordinary tiled 2-d load instead.  B (filters
// repacked to [K_out][R*S][C]) comes through a tiled 3-d load, so the channel tail of a tap is
// zero-filled rather than running into the next tap.  Both land in shared memory in the
// 128/64/32-byte swizzled K-major layout that tcgen05.mma reads through shared-memory descriptors.
//
// One persistent CTA per SM walks its tiles (128 pixels x BN channels):
//   warp 0      producer of A: waits for a free stage, arms its mbarrier with the byte count, issues TMA
//   warp 1      allocates tensor memory, issues tcgen05.mma (one lane), commits to mbarriers
//   16 warps    staged epilogue: tcgen05.ld the fp32 / int32 accumulators (one TMEM lane = one output pixel per
//               thread), apply the fused epilogue, write 16-byte pieces into a ring of 128-row x 128-byte boxes
//   1 warp      producer of B, on the same stages and barriers
//   1 warp      drains the ring (TMA stores, plain or through a 4-d map of a head-permuted tensor) and arms freed
//               boxes again (TMA loads of residual boxes)
//   (the direct variant, for fp32 / int32 outputs, runs 8 epilogue warps that store rows straight to global memory)
// Two accumulator buffers in tensor memory let the epilogue of tile i overlap the MMAs of tile i+1.
//
// The CTA-pair variant (clusters of two, tcgen05 cta_group::2) computes 256-row tiles across two SMs: each CTA
// loads its own rows of A and half of the filter tile, the first CTA issues the MMAs for both.
//
// Every mbarrier wait is bounded: when the limit expires the waiter records a code in the
// plan's status word, raises a CTA-wide abort flag, and every role falls through to the common
// exit where tensor memory is released.  The host reports ODLA_TIMEOUT.
#include <cuda.h>

#include <algorithm>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "epilogue.cuh"
#include "tensor_maps.h"
#include "umma_ptx.cuh"

namespace b200 {

namespace {

constexpr int BM = 128;
// Epilogue organisation.  Staged kernels (results leave through the shared-memory ring) run 16 epilogue
// warps on 16-column chunks: four warps per scheduler hide the latency of each other's tensor-memory
// and shared-memory reads, and 16 columns keep a thread under 96 registers.  The direct kernel (fp32 /
// int32 outputs, rows stored straight to global memory) keeps 8 warps on 32-column chunks.
template <bool STAGED> struct EpiCfg {
  static constexpr int kWarps = STAGED ? 16 : 8;     // epilogue warps (a multiple of 4: one per TMEM lane quarter)
  static constexpr int kChunk = STAGED ? 16 : 32;    // accumulator columns per tcgen05.ld
  static constexpr int kFilterWarp = 2 + kWarps;      // producer of B
  static constexpr int kStorerWarp = 3 + kWarps;      // drains finished boxes with TMA stores, arms them again (residual loads)
  static constexpr int kThreads = 32 * (4 + kWarps);
};
constexpr int kMaxRing = 8;

struct UmmaParams {
  int M_total, K_out, C, R, S, P, Q;
  int stride_h, stride_w, pad_t, pad_l;
  int im2col;          // 1: im2col TMA for A, 0: tiled 2-d TMA
  int kbe;             // elements of K per stage
  int kb_bytes;        // bytes of K per stage: 128, 64 or 32 (= swizzle span)
  int chunks_per_tap;  // ceil(C / kbe)
  int num_kb;          // R*S*chunks_per_tap
  int bps;             // operand boxes (k-blocks) per pipeline stage
  int num_it;          // ceil(num_kb / bps): stage fills per tile
  int BN, stages, m_tiles, n_tiles, total_tiles;
  uint32_t idesc;      // tcgen05 instruction descriptor
  uint32_t desc_hi;    // upper 32 bits of the shared-memory matrix descriptors
  int acc_int;         // accumulators are int32
  int rows_per_batch;  // batched GEMM: output rows per B matrix (0 = one shared B)
  int b_n_major;       // batched GEMM: B boxes hold [k rows][64 columns] (MN-major operand) instead of [n rows][64 k]
  int b_kstep;         // descriptor advance of B per 32 bytes of K, in 16-byte units: 2 (K-major) or 128 (16 rows of 128 bytes)
  int staged;          // epilogue goes through a shared-memory tile and TMA stores
  int res_tma;         // the residual tile is brought into that tile by TMA
  int out_esz;         // bytes per output element
  int stage_boxes;     // 128-row x 128-byte boxes per output tile
  int ring_boxes;      // boxes in the staging ring (>= stage_boxes)
  int box_arrivals;    // epilogue warps that write into one box
  int epi_interleave;  // groups take every fourth chunk instead of a contiguous run
  int pair;            // 1: two CTAs of a cluster share each 256-row tile (tcgen05 cta_group::2), each loading half of B
  int bn_load;         // rows of B this CTA brings into shared memory per k-block (BN, or BN/2 in pair mode)
  int store_mode, store_S, store_NH;  // permuted store through a 4-d map (see UmmaConv)
  int epi_mode;        // kernel variant: 0 direct, 1 staged straight-line forms, 2 staged general form, 3 staged straight-line LeakyReLU form
  int fast_variant;    // mode 1: accumulator conversion (0 fp32, 1 int32 by conversion, 2 int32 by integer add) * 2 + residual
  int tmem_cols;
  uint32_t spin_limit;  // attempts before a bounded wait gives up
  int splits;          // > 1: the split kernel, this many CTAs share a tile's reduction
  int bm;              // rows of its tiles: 128 or 64
  int split_data_bytes;  // ... shared memory before its barriers: the operand stages, reused by the partial tile
  int y_ld;            // row pitch of y in elements (split kernel)
  int split_plain;     // ... whose results take finish_plain
  int b_constant;      // B is written by no kernel: its loads need not wait for the kernel in front
  int test_skip_stage;  // test hook: the producer of CTA 0 leaves the last stage of its first tile unarmed, so the MMA lane's wait runs out
  void* y;
  int* status;
  Epilogue ep;
};

__device__ __forceinline__ unsigned long long gtime() { unsigned long long t; asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)); return t; }
#ifdef UMMA_DEBUG_TS
#define TS(i) do { if (blockIdx.x == 0 && p.status) { ((unsigned long long*)p.status)[4 + (i)] = gtime(); ((unsigned long long*)p.status)[20 + (i)] = (unsigned long long)clock64(); } } while (0)
#else
#define TS(i) do {} while (0)
#endif
// ------------------------------------------------------------------- epilogue ----
// One thread owns one output pixel (row) and CW consecutive channels held in v[] (registers: every
// index below is a compile-time constant after unrolling).
template <int CW>
__device__ __forceinline__ void load_vec(const float* __restrict__ src, int col0, int kmax, bool full, float (&out)[CW]) {
  if (full) {
#pragma unroll
    for (int q = 0; q < CW / 4; ++q) {
      float4 f = __ldg((const float4*)(src + col0) + q);
      out[4 * q] = f.x; out[4 * q + 1] = f.y; out[4 * q + 2] = f.z; out[4 * q + 3] = f.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < CW; ++j) out[j] = __ldg(src + min(col0 + j, kmax));
  }
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// Where a thread's channel segment lives in the shared-memory staging box (128-byte swizzle:
// 16-byte piece j of row r sits at piece j ^ (r & 7)).
struct StagePos {
  uint32_t row_addr;  // shared address of the 128-byte box row
  int j0;             // first 16-byte piece of the segment inside the row
  int rxor;           // r & 7
};
__device__ __forceinline__ uint32_t stage_piece(const StagePos& sp, int q) { return sp.row_addr + (uint32_t)(((sp.j0 + q) ^ sp.rxor) << 4); }

// OUT: the output storage type when known at compile time (DT_F16 / DT_BF16 / DT_S8), or -1 to
// branch on it at run time.  STAGED: results go to the shared-memory staging box and the residual
// (res_smem) is read from it.  `pre`/`use_pre`: residual pieces already fetched into registers (direct
// epilogue).  One instantiation per combination keeps the instruction footprint of the epilogue small:
// with few resident warps an epilogue that overflows the instruction cache stalls on every fetch.
template <int OUT, bool STAGED, int CW>
__device__ __forceinline__ void epilogue_chunk(const UmmaParams& p, float (&v)[CW], int64_t row, int col0, int ncols, const uint4 (&pre)[4], bool use_pre,
                                               const StagePos& sp, bool res_smem_in) {
  const Epilogue& ep = p.ep;
  constexpr bool staged = STAGED;
  const bool res_smem = STAGED && res_smem_in;
  const int out_dt = OUT >= 0 ? OUT : ep.out_dt;
  const bool colsall = ncols == CW;
  const bool full = colsall;                                         // per-channel vectors can be read 16 bytes at a time: col0 is a multiple of CW
  const bool gvec = colsall && (p.K_out & 15) == 0;                  // the row segment in global memory is 16-byte aligned for every element size
  const bool gvec32 = (p.K_out & 3) == 0;                            // ... for 4-byte outputs rows of a multiple of 4 elements are enough
  const int kmax = p.K_out - 1;
  const int64_t base = row * p.K_out + col0;
  float rv[CW];
  const bool has_res = ep.res != nullptr;
  if (has_res) {
    const bool vec = res_smem || use_pre || gvec;
    if (vec && (ep.res_dt == DT_F16 || ep.res_dt == DT_BF16)) {
      constexpr int NQ = CW / 8;
      const uint4* rp = (const uint4*)((const uint16_t*)ep.res + base);
      uint4 u[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) u[q] = res_smem ? lds128(stage_piece(sp, q)) : (use_pre ? pre[q] : __ldg(rp + q));
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          float2 f = ep.res_dt == DT_F16 ? __half22float2(((const __half2*)&u[q])[t]) : __bfloat1622float2(((const __nv_bfloat162*)&u[q])[t]);
          rv[q * 8 + 2 * t] = f.x;
          rv[q * 8 + 2 * t + 1] = f.y;
        }
      }
    } else if (vec && ep.res_dt == DT_S8) {
      constexpr int NQ = CW / 16;
      const uint4* rp = (const uint4*)((const int8_t*)ep.res + base);
      uint4 u[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) u[q] = res_smem ? lds128(stage_piece(sp, q)) : (use_pre ? pre[q] : __ldg(rp + q));
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const uint32_t* w = (const uint32_t*)&u[q];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
#pragma unroll
          for (int b = 0; b < 4; ++b) rv[q * 16 + t * 4 + b] = __fmul_rn((float)(signed char)(w[t] >> (8 * b)), ep.res_scale);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        float r = 0.f;
        if (j < ncols && row < p.M_total) {
          r = load_as_float(ep.res, ep.res_dt, base + j);
          if (ep.res_dt == DT_S8) r = __fmul_rn(r, ep.res_scale);
        }
        rv[j] = r;
      }
    }
  }
  float cv[CW];
  if (ep.mul) {
    load_vec<CW>(ep.mul, col0, kmax, full, cv);
#pragma unroll
    for (int j = 0; j < CW; ++j) v[j] = __fmul_rn(v[j], cv[j]);
  }
  if (ep.alpha != 1.f) {
#pragma unroll
    for (int j = 0; j < CW; ++j) v[j] = __fmul_rn(v[j], ep.alpha);
  }
  if (ep.add1) {
    load_vec<CW>(ep.add1, col0, kmax, full, cv);
#pragma unroll
    for (int j = 0; j < CW; ++j) v[j] = __fadd_rn(v[j], cv[j]);
  }
  if (ep.add2) {
    load_vec<CW>(ep.add2, col0, kmax, full, cv);
#pragma unroll
    for (int j = 0; j < CW; ++j) v[j] = __fadd_rn(v[j], cv[j]);
  }
  if (ep.add_full) {
#pragma unroll
    for (int j = 0; j < CW; ++j)
      if (j < ncols && row < p.M_total) v[j] = __fadd_rn(v[j], __fmul_rn(ep.beta_full, load_as_float(ep.add_full, ep.add_full_dt, base + j)));
  }
  if (ep.act != ACT_NONE && ep.act_first) {
#pragma unroll
    for (int j = 0; j < CW; ++j) v[j] = apply_act(ep.act, v[j], ep.act_a, ep.act_b);
  }
  if (has_res) {
#pragma unroll
    for (int j = 0; j < CW; ++j) v[j] = __fadd_rn(v[j], rv[j]);
  }
  if (ep.act != ACT_NONE && !ep.act_first) {
    if (ep.act == ACT_RELU) {
#pragma unroll
      for (int j = 0; j < CW; ++j) v[j] = fmaxf(v[j], 0.f);
    } else {
#pragma unroll
      for (int j = 0; j < CW; ++j) v[j] = apply_act(ep.act, v[j], ep.act_a, ep.act_b);
    }
  }
  // ---- store ----
  if (out_dt == DT_F16 || out_dt == DT_BF16) {
    constexpr int NQ = CW / 8;
    uint4 u[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (out_dt == DT_F16) {
        __half2* h = (__half2*)&u[q];
#pragma unroll
        for (int t = 0; t < 4; ++t) h[t] = __floats2half2_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1]);
      } else {
        __nv_bfloat162* h = (__nv_bfloat162*)&u[q];
#pragma unroll
        for (int t = 0; t < 4; ++t) h[t] = __floats2bfloat162_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1]);
      }
    }
    if (staged) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) sts128(stage_piece(sp, q), u[q]);
    } else if (row < p.M_total) {
      uint16_t* out = (uint16_t*)p.y + base;
      if (gvec) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) ((uint4*)out)[q] = u[q];
      } else {
        const uint16_t* e = (const uint16_t*)u;
#pragma unroll
        for (int j = 0; j < CW; ++j) if (j < ncols) out[j] = e[j];
      }
    }
  } else if (out_dt == DT_S8) {
    constexpr int NQ = CW / 16;
    uint4 u[NQ];
    uint32_t* w = (uint32_t*)u;
#pragma unroll
    for (int t = 0; t < CW / 4; ++t) {
      uint32_t qb[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const float t4 = ep.out_multiply ? __fmul_rn(v[t * 4 + b], ep.out_inv) : __fdiv_rn(v[t * 4 + b], ep.out_scale);
        qb[b] = (uint32_t)rne_sat_s8(t4);
      }
      // low bytes of the four results -> one word (three byte permutes)
      w[t] = __byte_perm(__byte_perm(qb[0], qb[1], 0x0040), __byte_perm(qb[2], qb[3], 0x0040), 0x5410);
    }
    if (staged) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) sts128(stage_piece(sp, q), u[q]);
    } else if (row < p.M_total) {
      int8_t* out = (int8_t*)p.y + base;
      if (gvec) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) ((uint4*)out)[q] = u[q];
      } else {
        const int8_t* e = (const int8_t*)u;
#pragma unroll
        for (int j = 0; j < CW; ++j) if (j < ncols) out[j] = e[j];
      }
    }
  } else if (row < p.M_total) {  // DT_F32
    float* out = (float*)p.y + base;
    if (gvec32) {   // whole 16-byte pieces, then at most three single elements (ncols is a multiple of 4 here)
#pragma unroll
      for (int q = 0; q < CW / 4; ++q) if (4 * q + 3 < ncols) ((float4*)out)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < CW; ++j) if (j < ncols) out[j] = v[j];
    }
  }
}

// Two fp32 additions in one instruction (add.rn.f32x2, sm_100): same rounding as two __fadd_rn.
// CAUTION: an add.rn.f32x2 that consumes the result of a mul.rn.f32x2 is contracted into one fused multiply-add by
// the assembler in spite of the .rn qualifiers (measured: 27 % of random inputs differ in the last bit from
// mul-then-add; each instruction on its own, and a packed multiply followed by scalar __fadd_rn, are exact).  A sum
// whose operand comes from fmul2_rn therefore uses __fadd_rn.
__device__ __forceinline__ void fadd2_rn(float& a0, float& a1, float b0, float b1) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "f"(b0), "f"(b1));
}
__device__ __forceinline__ void fmul2_rn(float& a0, float& a1, float b0, float b1) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "f"(b0), "f"(b1));
}
// Exact conversions without the conversion pipe (its rate, a quarter of the ALU's, bounded the int8 epilogue):
//   int32 -> fp32 for |a| < 2^22: 0x4B400000 is 2^23 + 2^22 = 12582912.f, whose ulp is 1, so adding a to the bit pattern
//     gives 12582912 + a exactly and the subtraction is exact as well;
//   int8 -> fp32: the byte with its sign bit flipped (b + 128, 0..255) placed in the mantissa of 2^23 is 8388608 + 128 + b;
//   fp32 -> int8 with round-to-nearest-even and saturation: clamp to [-128, 127] (or [0, 127] under a ReLU), add
//     12582912.f -- the addition rounds to an integer, ties to even -- and take the low byte (two's complement).
constexpr uint32_t kMagicBits = 0x4B400000u;
constexpr float kMagic = 12582912.f;
__device__ __forceinline__ float s8_byte_to_float(uint32_t word_flipped, int b) {
  return __fadd_rn(__uint_as_float(__byte_perm(word_flipped, 0x4B000000u, 0x7540u + (uint32_t)b)), -8388736.f);
}
// The staged epilogue's chunk: 16 consecutive channels of one output row, residual read from and result
// written to the row's place in the staging box.  Only what a staged launch can need is here (the launcher
// sends everything else to the direct epilogue), so the loop around it stays small.
template <int OUT, bool ANYACT>
__device__ __forceinline__ void epilogue_chunk_staged(const UmmaParams& p, float (&v)[16], int col0, const StagePos& sp) {
  const Epilogue& ep = p.ep;
  const bool full = col0 + 16 <= p.K_out;  // the last chunk of a row may be cut short: its vectors are read with clamped indices
  const int kmax = p.K_out - 1;
  float cv[16];
  if (ep.mul) {
    load_vec<16>(ep.mul, col0, kmax, full, cv);
#pragma unroll
    for (int j = 0; j < 16; j += 2) fmul2_rn(v[j], v[j + 1], cv[j], cv[j + 1]);
  }
  if (ep.alpha != 1.f) {
#pragma unroll
    for (int j = 0; j < 16; j += 2) fmul2_rn(v[j], v[j + 1], ep.alpha, ep.alpha);
  }
  const bool after_mul = ep.mul != nullptr || ep.alpha != 1.f;  // v[] comes out of a packed multiplication
  if (ep.add1) {
    load_vec<16>(ep.add1, col0, kmax, full, cv);
    if (after_mul) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __fadd_rn(v[j], cv[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 16; j += 2) fadd2_rn(v[j], v[j + 1], cv[j], cv[j + 1]);
    }
  }
  if (ep.add2) {
    load_vec<16>(ep.add2, col0, kmax, full, cv);
    if (after_mul && !ep.add1) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __fadd_rn(v[j], cv[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 16; j += 2) fadd2_rn(v[j], v[j + 1], cv[j], cv[j + 1]);
    }
  }
  if (ANYACT && ep.act_first) apply_act_all<16>(ep.act, v, ep.act_a, ep.act_b);
  if (p.res_tma) {
    if (OUT == DT_S8) {
      const uint4 u = lds128(stage_piece(sp, 0));
      const uint32_t* w = (const uint32_t*)&u;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t wf = w[t] ^ 0x80808080u;
#pragma unroll
        for (int b = 0; b < 4; b += 2) {
          float r0 = s8_byte_to_float(wf, b), r1 = s8_byte_to_float(wf, b + 1);
          fmul2_rn(r0, r1, ep.res_scale, ep.res_scale);
          v[t * 4 + b] = __fadd_rn(v[t * 4 + b], r0);
          v[t * 4 + b + 1] = __fadd_rn(v[t * 4 + b + 1], r1);
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint4 u = lds128(stage_piece(sp, q));
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float2 f = OUT == DT_F16 ? __half22float2(((const __half2*)&u)[t]) : __bfloat1622float2(((const __nv_bfloat162*)&u)[t]);
          if (after_mul && !ep.add1 && !ep.add2) { v[q * 8 + 2 * t] = __fadd_rn(v[q * 8 + 2 * t], f.x); v[q * 8 + 2 * t + 1] = __fadd_rn(v[q * 8 + 2 * t + 1], f.y); }
          else fadd2_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1], f.x, f.y);
        }
      }
    }
  }
  if (ANYACT) {
    if (!ep.act_first) apply_act_all<16>(ep.act, v, ep.act_a, ep.act_b);
  }
  // (plain int8 outputs take their ReLU as the lower bound of the saturating clamp below)
  // (two-byte outputs take their ReLU after packing, two values per instruction: rounding is monotonic and keeps the sign)
  const bool relu_packed = !ANYACT && ep.act == ACT_RELU && OUT != DT_S8;
  if (OUT == DT_S8 && !ANYACT) {
    // requantisation by multiplication; the ReLU (if any) is the lower clamp: max(v, 0) * m == max(v * m, 0) for m > 0
    const float lo = ep.act == ACT_RELU && ep.out_inv > 0.f ? 0.f : -128.f;
    uint4 u;
    uint32_t* w = (uint32_t*)&u;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      float q[4];
#pragma unroll
      for (int b = 0; b < 4; b += 2) {
        q[b] = v[t * 4 + b]; q[b + 1] = v[t * 4 + b + 1];
        fmul2_rn(q[b], q[b + 1], ep.out_inv, ep.out_inv);
        q[b] = fminf(fmaxf(q[b], lo), 127.f); q[b + 1] = fminf(fmaxf(q[b + 1], lo), 127.f);
        fadd2_rn(q[b], q[b + 1], kMagic, kMagic);  // (the clamp sits between the multiplication and this addition)
      }
      w[t] = __byte_perm(__byte_perm(__float_as_uint(q[0]), __float_as_uint(q[1]), 0x0040), __byte_perm(__float_as_uint(q[2]), __float_as_uint(q[3]), 0x0040), 0x5410);
    }
    sts128(stage_piece(sp, 0), u);
  } else if (OUT == DT_S8) {
    uint4 u;
    uint32_t* w = (uint32_t*)&u;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint32_t qb[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const float t4 = ep.out_multiply ? __fmul_rn(v[t * 4 + b], ep.out_inv) : __fdiv_rn(v[t * 4 + b], ep.out_scale);
        qb[b] = (uint32_t)rne_sat_s8(t4);
      }
      w[t] = __byte_perm(__byte_perm(qb[0], qb[1], 0x0040), __byte_perm(qb[2], qb[3], 0x0040), 0x5410);
    }
    sts128(stage_piece(sp, 0), u);
  } else {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint4 u;
      if (OUT == DT_F16) {
        __half2* h = (__half2*)&u;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          h[t] = __floats2half2_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1]);
          if (relu_packed) h[t] = __hmax2(h[t], __float2half2_rn(0.f));
        }
      } else {
        __nv_bfloat162* h = (__nv_bfloat162*)&u;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          h[t] = __floats2bfloat162_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1]);
          if (relu_packed) h[t] = __hmax2(h[t], __float2bfloat162_rn(0.f));
        }
      }
      sts128(stage_piece(sp, q), u);
    }
  }
}


// The staged epilogue of the common layer forms as straight-line code (MODE 1): every decision that does not depend on
// the data is a template parameter or was made on the host, because the general chunk above spends a fifth of its
// instructions on branches over the launch's configuration.  The launcher guarantees: full 16-column chunks, alpha = 1,
// exactly one per-channel addend (`addv`), a per-channel multiplier exactly when the accumulators are integers,
// activation none or ReLU after the residual, int8 outputs requantised by multiplication.
//   ACC 0: fp32 accumulators; 1: int32 -> fp32 by conversion; 2: int32 -> fp32 by the exact integer-add form (|acc| < 2^22)
//   RES: a residual tile of the output's type waits in the staging box
template <int OUT, int ACC, bool RES>
__device__ __forceinline__ void chunk_fast(const uint32_t (&r)[16], const float* __restrict__ mulv, const float* __restrict__ addv, float res_scale,
                                           float out_inv, float lo, uint32_t relu_floor, const StagePos& sp) {
  float v[16];
  if (ACC == 2) {
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      v[j] = __uint_as_float(r[j] + kMagicBits); v[j + 1] = __uint_as_float(r[j + 1] + kMagicBits);
      fadd2_rn(v[j], v[j + 1], -kMagic, -kMagic);
    }
  } else if (ACC == 1) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = (float)(int32_t)r[j];
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
  }
  float cv[16];
  if (ACC != 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) { const float4 f = __ldg((const float4*)mulv + q); cv[4 * q] = f.x; cv[4 * q + 1] = f.y; cv[4 * q + 2] = f.z; cv[4 * q + 3] = f.w; }
#pragma unroll
    for (int j = 0; j < 16; j += 2) fmul2_rn(v[j], v[j + 1], cv[j], cv[j + 1]);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) { const float4 f = __ldg((const float4*)addv + q); cv[4 * q] = f.x; cv[4 * q + 1] = f.y; cv[4 * q + 2] = f.z; cv[4 * q + 3] = f.w; }
  if (ACC != 0) {  // the sum consumes a packed product: scalar additions (see fadd2_rn)
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __fadd_rn(v[j], cv[j]);
  } else {
#pragma unroll
    for (int j = 0; j < 16; j += 2) fadd2_rn(v[j], v[j + 1], cv[j], cv[j + 1]);
  }
  if (OUT == DT_S8) {
    if (RES) {
      const uint4 u = lds128(stage_piece(sp, 0));
      const uint32_t* w = (const uint32_t*)&u;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t wf = w[t] ^ 0x80808080u;
#pragma unroll
        for (int b = 0; b < 4; b += 2) {
          float r0 = s8_byte_to_float(wf, b), r1 = s8_byte_to_float(wf, b + 1);
          fmul2_rn(r0, r1, res_scale, res_scale);
          v[t * 4 + b] = __fadd_rn(v[t * 4 + b], r0);
          v[t * 4 + b + 1] = __fadd_rn(v[t * 4 + b + 1], r1);
        }
      }
    }
    uint4 u;
    uint32_t* w = (uint32_t*)&u;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      float q[4];
#pragma unroll
      for (int b = 0; b < 4; b += 2) {
        q[b] = v[t * 4 + b]; q[b + 1] = v[t * 4 + b + 1];
        fmul2_rn(q[b], q[b + 1], out_inv, out_inv);
        q[b] = fminf(fmaxf(q[b], lo), 127.f); q[b + 1] = fminf(fmaxf(q[b + 1], lo), 127.f);
        fadd2_rn(q[b], q[b + 1], kMagic, kMagic);  // (the clamp sits between the multiplication and this addition)
      }
      w[t] = __byte_perm(__byte_perm(__float_as_uint(q[0]), __float_as_uint(q[1]), 0x0040), __byte_perm(__float_as_uint(q[2]), __float_as_uint(q[3]), 0x0040), 0x5410);
    }
    sts128(stage_piece(sp, 0), u);
  } else {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint4 u;
      if (RES) {
        u = lds128(stage_piece(sp, q));
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float2 f = OUT == DT_F16 ? __half22float2(((const __half2*)&u)[t]) : __bfloat1622float2(((const __nv_bfloat162*)&u)[t]);
          fadd2_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1], f.x, f.y);   // v[] comes out of an addition here
        }
      }
      // ReLU after packing, two values per instruction: rounding is monotonic and keeps the sign; without a ReLU the
      // floor is -inf and the maximum changes nothing
      if (OUT == DT_F16) {
        __half2* h = (__half2*)&u;
        const __half2 fl = *(const __half2*)&relu_floor;
#pragma unroll
        for (int t = 0; t < 4; ++t) h[t] = __hmax2(__floats2half2_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1]), fl);
      } else {
        __nv_bfloat162* h = (__nv_bfloat162*)&u;
        const __nv_bfloat162 fl = *(const __nv_bfloat162*)&relu_floor;
#pragma unroll
        for (int t = 0; t < 4; ++t) h[t] = __hmax2(__floats2bfloat162_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1]), fl);
      }
      sts128(stage_piece(sp, q), u);
    }
  }
}
// One box's share of chunks for one epilogue warp, straight-line form.
template <int OUT, int ACC, bool RES>
__device__ __forceinline__ void box_fast(const UmmaParams& p, uint32_t taddr, int first, int last, int step, int n0, int bx, int chunks_per_box, StagePos sp,
                                         float lo, uint32_t relu_floor) {
  const float res_scale = p.ep.res_scale, out_inv = p.ep.out_inv;
  const float* mulv = p.ep.mul;
  const float* addv = p.ep.add1 ? p.ep.add1 : p.ep.add2;
  const int j_shift = OUT == DT_S8 ? 0 : 1;   // 16 columns are one (int8) or two (16-bit types) 16-byte pieces
#pragma unroll 1
  for (int ch = first; ch < last; ch += step) {
    const int col0 = n0 + ch * 16;
    if (col0 >= p.K_out) break;
    uint32_t r[16];
    tmem_ld16(taddr + (uint32_t)(ch * 16), r);
    tmem_ld_wait_regs<16>(r);
    sp.j0 = (ch - bx * chunks_per_box) << j_shift;
    chunk_fast<OUT, ACC, RES>(r, mulv + col0, addv + col0, res_scale, out_inv, lo, relu_floor, sp);
  }
}

// The Darknet layer form as straight-line code (MODE 3): fp32 accumulators, one per-channel addend, LeakyReLU with a
// slope in [0, 1], then (optionally) the residual tile, two-byte outputs.  For such a slope x < 0 ? fl(a*x) : x equals
// max(x, fl(a*x)): the product rounds monotonically and keeps the sign.
// GELU (erf form) without branches, used only where the result is rounded to a two-byte type right after (the
// library erff takes two different paths by magnitude, which a warp's 32 rows then both execute):
//   x Phi(x) = x / 2 + |x| (1/2 - Phi(-|x|)),   Phi(-a) = 2^P(a),
// with P of degree 8, the minimax fit (a linear programme over the error of 2^P) of log2 Phi(-a) on [0, 5.7]: 7.6e-9 in Phi.  P stays
// below -26 beyond and goes to minus infinity, so infinities and NaN come out as from the formula.  Largest error against 64 bits
// 3.4e-7, the roundings of fp32 included (4.7e-7 for erf as a polynomial in 1 / (1 + 0.33 |z|), which takes a reciprocal more).
// A feed-forward layer's epilogue is bound by instruction issue: this is 13 packed and 4 scalar instructions for two values; BERT-base
// of 64 x 128 1707 -> 1664 us in fp16 against the reciprocal's form, 1687 with scalar instructions.
__device__ __forceinline__ void ffma2(float& a0, float& a1, float b0, float b1, float c0, float c1) {   // a = a * b + c
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tmov.b64 z, {%4, %5};\n\tfma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void gelu_erf_two_byte_pair(float& t0, float& t1) {
  const float a0 = fabsf(t0), a1 = fabsf(t1);
  float p0 = a0, p1 = a1;
  ffma2(p0, p1, -2.772033213e-06f, -2.772033213e-06f, 3.862057201e-05f, 3.862057201e-05f);
  constexpr float kP[7] = {-1.825468353e-04f, -1.458717888e-04f, 7.075473666e-03f, -5.250503123e-02f, -4.592049122e-01f, -1.151105762f, -1.0f};
#pragma unroll
  for (int i = 0; i < 7; ++i) ffma2(p0, p1, a0, a1, kP[i], kP[i]);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(p0));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(p1));
  ffma2(p0, p1, -1.f, -1.f, 0.5f, 0.5f);
  fmul2_rn(t0, t1, 0.5f, 0.5f);
  ffma2(p0, p1, a0, a1, t0, t1);
  t0 = p0; t1 = p1;
}
// The form for results that are requantised: erf by Abramowitz & Stegun 7.1.26 (the whole expression within 5e-7).  A value next to a
// rounding boundary moves by a whole step with any other last bits, and twelve layers carry such steps to 2 % of the output; the
// shorter form above would save 3 % of an int8 BERT-base at that price.
__device__ __forceinline__ void gelu_erf_requantised_pair(float& t0, float& t1) {
  float z0 = t0, z1 = t1;
  fmul2_rn(z0, z1, 0.70710678118654752440f, 0.70710678118654752440f);
  const float a0 = fabsf(z0), a1 = fabsf(z1);
  float d0 = a0, d1 = a1;
  ffma2(d0, d1, 0.3275911f, 0.3275911f, 1.0f, 1.0f);
  const float k0 = __fdividef(1.0f, d0), k1 = __fdividef(1.0f, d1);
  float p0 = k0, p1 = k1;
  ffma2(p0, p1, 1.061405429f, 1.061405429f, -1.453152027f, -1.453152027f);
  ffma2(p0, p1, k0, k1, 1.421413741f, 1.421413741f);
  ffma2(p0, p1, k0, k1, -0.284496736f, -0.284496736f);
  ffma2(p0, p1, k0, k1, 0.254829592f, 0.254829592f);
  fmul2_rn(p0, p1, -k0, -k1);                       // -(polynomial * k)
  float e0 = a0, e1 = a1;
  fmul2_rn(e0, e1, a0, a1);
  fmul2_rn(e0, e1, -1.4426950408889634f, -1.4426950408889634f);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e0));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e1));
  ffma2(p0, p1, e0, e1, 1.0f, 1.0f);                // 1 - polynomial * k * exp(-z^2)
  p0 = copysignf(p0, z0); p1 = copysignf(p1, z1);
  fadd2_rn(p0, p1, 1.0f, 1.0f);
  fmul2_rn(t0, t1, 0.5f, 0.5f);
  fmul2_rn(t0, t1, p0, p1);
}
// ACTF 0: LeakyReLU, 1: GELU (erf form)
template <int OUT, int ACTF, bool RES>
__device__ __forceinline__ void chunk_leaky(const uint32_t (&r)[16], const float* __restrict__ addv, float slope, const StagePos& sp) {
  float v[16], cv[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
#pragma unroll
  for (int q = 0; q < 4; ++q) { const float4 f = __ldg((const float4*)addv + q); cv[4 * q] = f.x; cv[4 * q + 1] = f.y; cv[4 * q + 2] = f.z; cv[4 * q + 3] = f.w; }
#pragma unroll
  for (int j = 0; j < 16; j += 2) {
    fadd2_rn(v[j], v[j + 1], cv[j], cv[j + 1]);
    if (ACTF == 0) {
      float t0 = v[j], t1 = v[j + 1];
      fmul2_rn(t0, t1, slope, slope);
      v[j] = fmaxf(v[j], t0); v[j + 1] = fmaxf(v[j + 1], t1);   // (a maximum between the product and any later sum: nothing to contract)
    } else {
      gelu_erf_two_byte_pair(v[j], v[j + 1]);
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint4 u;
    if (RES) {
      u = lds128(stage_piece(sp, q));
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 f = OUT == DT_F16 ? __half22float2(((const __half2*)&u)[t]) : __bfloat1622float2(((const __nv_bfloat162*)&u)[t]);
        fadd2_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1], f.x, f.y);
      }
    }
    if (OUT == DT_F16) {
      __half2* h = (__half2*)&u;
#pragma unroll
      for (int t = 0; t < 4; ++t) h[t] = __floats2half2_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1]);
    } else {
      __nv_bfloat162* h = (__nv_bfloat162*)&u;
#pragma unroll
      for (int t = 0; t < 4; ++t) h[t] = __floats2bfloat162_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1]);
    }
    sts128(stage_piece(sp, q), u);
  }
}
template <int OUT, int ACTF, bool RES>
__device__ __forceinline__ void box_leaky(const UmmaParams& p, uint32_t taddr, int first, int last, int step, int n0, int bx, int chunks_per_box, StagePos sp) {
  const float slope = p.ep.act_a;
  const float* addv = p.ep.add1 ? p.ep.add1 : p.ep.add2;
#pragma unroll 1
  for (int ch = first; ch < last; ch += step) {
    const int col0 = n0 + ch * 16;
    if (col0 >= p.K_out) break;
    uint32_t r[16];
    tmem_ld16(taddr + (uint32_t)(ch * 16), r);
    tmem_ld_wait_regs<16>(r);
    sp.j0 = (ch - bx * chunks_per_box) << 1;
    chunk_leaky<OUT, ACTF, RES>(r, addv + col0, slope, sp);
  }
}

// The int8 form of a transformer's first feed-forward layer: int32 accumulators, per-channel multiplier and addend,
// GELU, requantisation by multiplication to int8.  ACC as in chunk_fast (1: conversion, 2: exact integer-add form).
template <int ACC>
__device__ __forceinline__ void chunk_gelu_s8(const uint32_t (&r)[16], const float* __restrict__ mulv, const float* __restrict__ addv, float out_inv, const StagePos& sp) {
  float v[16], cv[16];
  if (ACC == 2) {
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      v[j] = __uint_as_float(r[j] + kMagicBits); v[j + 1] = __uint_as_float(r[j + 1] + kMagicBits);
      fadd2_rn(v[j], v[j + 1], -kMagic, -kMagic);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = (float)(int32_t)r[j];
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) { const float4 f = __ldg((const float4*)mulv + q); cv[4 * q] = f.x; cv[4 * q + 1] = f.y; cv[4 * q + 2] = f.z; cv[4 * q + 3] = f.w; }
#pragma unroll
  for (int j = 0; j < 16; j += 2) fmul2_rn(v[j], v[j + 1], cv[j], cv[j + 1]);
#pragma unroll
  for (int q = 0; q < 4; ++q) { const float4 f = __ldg((const float4*)addv + q); cv[4 * q] = f.x; cv[4 * q + 1] = f.y; cv[4 * q + 2] = f.z; cv[4 * q + 3] = f.w; }
#pragma unroll
  for (int j = 0; j < 16; j += 2) {   // scalar sums after a packed product (see fadd2_rn)
    v[j] = __fadd_rn(v[j], cv[j]); v[j + 1] = __fadd_rn(v[j + 1], cv[j + 1]);
    gelu_erf_requantised_pair(v[j], v[j + 1]);
  }
  uint4 u;
  uint32_t* w = (uint32_t*)&u;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    float q[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) q[b] = __fadd_rn(fminf(fmaxf(__fmul_rn(v[t * 4 + b], out_inv), -128.f), 127.f), kMagic);
    w[t] = __byte_perm(__byte_perm(__float_as_uint(q[0]), __float_as_uint(q[1]), 0x0040), __byte_perm(__float_as_uint(q[2]), __float_as_uint(q[3]), 0x0040), 0x5410);
  }
  sts128(stage_piece(sp, 0), u);
}
template <int ACC>
__device__ __forceinline__ void box_gelu_s8(const UmmaParams& p, uint32_t taddr, int first, int last, int step, int n0, int bx, int chunks_per_box, StagePos sp) {
  const float out_inv = p.ep.out_inv;
  const float* mulv = p.ep.mul;
  const float* addv = p.ep.add1 ? p.ep.add1 : p.ep.add2;
#pragma unroll 1
  for (int ch = first; ch < last; ch += step) {
    const int col0 = n0 + ch * 16;
    if (col0 >= p.K_out) break;
    uint32_t r[16];
    tmem_ld16(taddr + (uint32_t)(ch * 16), r);
    tmem_ld_wait_regs<16>(r);
    sp.j0 = ch - bx * chunks_per_box;
    chunk_gelu_s8<ACC>(r, mulv + col0, addv + col0, out_inv, sp);
  }
}

// The products of one k-block: 32 bytes of K per instruction; `la`, `lb` are the low words of the operands' descriptors.
// Everything that does not change from instruction to instruction is decided outside -- the issuing lane's instruction
// stream is what the tensor pipe waits for.
__device__ __forceinline__ uint64_t desc64(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
template <bool PAIR, bool INT>
__device__ __forceinline__ void issue_one(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accum) {
  if constexpr (PAIR && INT) umma_i8_pair(d, da, db, idesc, accum);
  else if constexpr (PAIR) umma_f16_pair(d, da, db, idesc, accum);
  else if constexpr (INT) umma_i8(d, da, db, idesc, accum);
  else umma_f16(d, da, db, idesc, accum);
}
// (a pair's commit arrives on the barrier at this offset in both CTAs once the MMAs issued so far have completed)
template <bool PAIR> __device__ __forceinline__ void commit_at(uint32_t bar) {
  if constexpr (PAIR)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// The products of one k-block of umma_split_kernel.
__device__ __forceinline__ void issue_kblock(const UmmaParams& p, uint32_t d, uint32_t la, uint32_t lb, int ksteps, uint32_t accum) {
  if (ksteps == 4 && !p.acc_int && p.b_kstep == 2) {
#pragma unroll
    for (int k = 0; k < 4; ++k) issue_one<false, false>(d, desc64(la + 2 * k, p.desc_hi), desc64(lb + 2 * k, p.desc_hi), p.idesc, k ? 1u : accum);
    return;
  }
  for (int k = 0; k < ksteps; ++k) {
    if (p.acc_int) issue_one<false, true>(d, desc64(la + 2 * k, p.desc_hi), desc64(lb + 2 * k, p.desc_hi), p.idesc, accum);
    else issue_one<false, false>(d, desc64(la + 2 * k, p.desc_hi), desc64(lb + (uint32_t)(p.b_kstep * k), p.desc_hi), p.idesc, accum);
    accum = 1;
  }
}
// Row and column of a tile; consecutive tiles of a unit lie tile_step apart.
template <bool V> struct BoolConst { static constexpr bool value = V; };
struct TileWalk {
  int mi, ni;
  __device__ __forceinline__ TileWalk(const UmmaParams& p, int tile) { ni = tile / p.m_tiles; mi = tile - ni * p.m_tiles; }
  __device__ __forceinline__ bool next(const UmmaParams& p, int step) {   // true when the column changed
    mi += step;
    const bool wrapped = mi >= p.m_tiles;
    while (mi >= p.m_tiles) { mi -= p.m_tiles; ++ni; }
    return wrapped;
  }
};

// --------------------------------------------------------------------- kernel ----
// MODE 3: staged epilogue, further straight-line forms: LeakyReLU before the optional residual (Darknet) or GELU, two-byte
//         outputs (box_leaky); int8 operands, GELU, requantised int8 output (box_gelu_s8).
// MODE 0: direct epilogue (any output type, rows written straight to global memory).
// MODE 1: staged epilogue, straight-line forms (box_fast): activation none / ReLU after the residual, one per-channel
//         addend, int8 requantisation by multiplication.
// MODE 2: staged epilogue, general form: every activation, activation before the residual, division requantisation,
//         any combination of per-channel vectors, a ragged last chunk.
// PAIR: CTA-pair variant (its cta_group::2 instructions make the kernel launchable only as clusters of two).
template <int OUT, int MODE, bool PAIR>
__global__ void __launch_bounds__(EpiCfg<MODE != 0>::kThreads, 1)
umma_conv_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmY,
                 const __grid_constant__ CUtensorMap tmR, const UmmaParams p) {
  constexpr bool STAGED = MODE != 0;
  constexpr int kPair = PAIR ? 1 : 0;
  constexpr int kEpilogueWarps = EpiCfg<STAGED>::kWarps, kFilterWarp = EpiCfg<STAGED>::kFilterWarp, kStorerWarp = EpiCfg<STAGED>::kStorerWarp;
  constexpr int CW = EpiCfg<STAGED>::kChunk;
  extern __shared__ uint8_t smem_raw[];
  if (threadIdx.x == 0) TS(7);
  // operand stages start on a 1024-byte boundary (the 128-byte swizzle repeats every 1024 bytes)
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int stage_bytes = p.bps * (BM + p.bn_load) * p.kb_bytes;
  uint8_t* staging = smem + (size_t)p.stages * stage_bytes;   // 1024-byte aligned: stage sizes are multiples of 2 KiB
  uint8_t* ctrl = staging + (size_t)p.ring_boxes * 16384;
  uint64_t* full_bar = (uint64_t*)ctrl;            // [stages]
  uint64_t* empty_bar = full_bar + 16;             // [stages]
  uint64_t* tfull_bar = empty_bar + 16;            // [2]
  uint64_t* tempty_bar = tfull_bar + 2;            // [2]
  uint64_t* box_full = tempty_bar + 2;             // [ring] box is armed: free, and its residual (if any) has landed
  uint64_t* box_done = box_full + kMaxRing;        // [ring] every epilogue warp that owns part of the box has written it
  uint32_t* tmem_slot = (uint32_t*)(box_done + kMaxRing);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // A lane per barrier: 52 initialisations in a row would be on every launch's way.
  if (warp == 0) {
    constexpr int kTempty = 34, kBoxes = 36, kAll = kBoxes + 2 * kMaxRing;
    for (int i = lane; i < kAll; i += 32) {
      // full (both producers have armed the stage and every byte has landed), empty, accumulator full, accumulator empty (in pair mode the
      // epilogue warps of both CTAs release it on the first CTA's barrier), box armed, box done
      const uint32_t count = i < 16 ? 2u : i < kTempty ? 1u : i < kBoxes ? (uint32_t)(kEpilogueWarps << kPair) : i < kBoxes + kMaxRing ? 1u : (uint32_t)p.box_arrivals;
      mbar_init(&full_bar[i], count);
    }
    if (lane == 0) *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kStorerWarp && lane == 0) {
    prefetch_map(&tmA);
    prefetch_map(&tmB);
    if (STAGED) prefetch_map(&tmY);
    if (p.res_tma) prefetch_map(&tmR);
  }
  if constexpr (PAIR) {   // the peer's barriers exist before anything of this CTA can reach them
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (PAIR) {  // the same warp of both CTAs allocates the same columns in both tensor memories
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)p.tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)p.tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  if constexpr (PAIR) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Programmatic dependent launch: everything above overlapped the previous kernel's tail.  Only the threads that touch
  // tensors other kernels write or read wait for that kernel (grid_dependency_wait): the producer of A, the storer and direct
  // epilogues.  The producer of B does not when its boxes come from constants: they are on the way early.
  if (threadIdx.x == 0) TS(0);

  const uint32_t a_box = (uint32_t)(BM * p.kb_bytes), b_box = (uint32_t)(p.bn_load * p.kb_bytes);
  // Tile walk: a unit (a CTA, or a CTA pair) takes every `tile_step`-th tile; in pair mode a tile is 256 rows and
  // this CTA owns the half given by its rank in the cluster.
  const int rank = PAIR ? (int)cluster_ctarank() : 0;
  const int tile_first = (int)(blockIdx.x >> kPair), tile_step = (int)(gridDim.x >> kPair);
  if (warp == 0) {
    // ------------------------------------------------------------ producer of A ----
    // One lane; its instruction rate bounds the rate of stages.  The pixel a tile starts at is carried from tile to tile.
    if (elect_one()) {
      grid_dependency_wait();
      asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the next kernel may start its own prologue now
      const uint32_t bytes_kb = PAIR ? 2u * a_box : a_box;              // the first CTA's barrier counts the bytes of both
      const uint32_t sa0 = smem_u32(smem), full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
      const uint32_t land0 = PAIR ? map_to_cta(full0, 0) : full0;       // the barriers the copies signal
      auto produce = [&](auto im2col_mode) {
        constexpr bool IM2COL = decltype(im2col_mode)::value;
        const uint32_t full_end = full0 + 8u * (uint32_t)p.stages, to_empty = empty0 - full0, to_land = land0 - full0;
        const int bps = p.bps, kbe = p.kbe, C = p.C, R = p.R, S = p.S;
        const bool hook = p.test_skip_stage && blockIdx.x == 0;
        bool ok = true;
        uint32_t bar = full0, ph = 1, sa_stage = sa0;   // a stage is free when its phase differs: the first round passes at once
        TileWalk at(p, tile_first);
        int img = 0, op = 0, oq = 0, d_img = 0, d_op = 0, d_oq = 0;
        auto locate = [&](int pix, int& i, int& r, int& c) { const int pq = p.P * p.Q; i = pix / pq; pix -= i * pq; r = pix / p.Q; c = pix - r * p.Q; };
        if (IM2COL) {
          locate(((at.mi << kPair) + rank) * BM, img, op, oq);
          locate((tile_step << kPair) * BM, d_img, d_op, d_oq);
        }
        for (int tile = tile_first; tile < p.total_tiles && ok; tile += tile_step) {
          const int m0 = ((at.mi << kPair) + rank) * BM;
          const int w0 = oq * p.stride_w - p.pad_l, h0 = op * p.stride_h - p.pad_t;
          int fr = 0, fs = 0, c0 = 0, left = p.num_kb;
          while (left > 0) {
            if (!mbar_try_wait_at(bar + to_empty, ph) && !mbar_wait(empty_bar + ((bar - full0) >> 3), ph, abort_flag, p.status, 1, p.spin_limit)) { ok = false; break; }
            const int nb = min(left, bps);
            left -= nb;
            // Test hook (never set by the planner): this stage is neither armed nor loaded, so its barrier can never
            // complete and the MMA lane's bounded wait reports a timeout; nothing faults and nothing spins for ever.
            const bool skip = !PAIR && hook && tile == tile_first && left == 0;
            if (!skip && (!PAIR || rank == 0)) mbar_expect_tx_at(bar, (uint32_t)nb * bytes_kb);
            const uint32_t land = bar + to_land;
            uint32_t sa = sa_stage;
            for (int j = skip ? nb : 0; j < nb; ++j) {
              if (IM2COL) load_im2col_at<PAIR>(sa, &tmA, land, c0, w0, h0, img, (uint16_t)fs, (uint16_t)fr);
              else load_2d_at<PAIR>(sa, &tmA, land, c0, m0);
              sa += a_box;
              c0 += kbe;
              if (c0 >= C) {
                c0 = 0;
                if (IM2COL && ++fs == S) { fs = 0; if (++fr == R) fr = 0; }   // the next filter term walks the window again
              }
            }
            sa_stage += (uint32_t)stage_bytes;
            bar += 8;
            if (bar == full_end) { bar = full0; ph ^= 1; sa_stage = sa0; }
          }
          const bool wrapped = at.next(p, tile_step);
          if (IM2COL) {
            if (wrapped) locate(((at.mi << kPair) + rank) * BM, img, op, oq);
            else {
              oq += d_oq; if (oq >= p.Q) { oq -= p.Q; ++op; }
              op += d_op; if (op >= p.P) { op -= p.P; ++img; }
              img += d_img;
            }
          }
        }
        if (!ok) await_stages(full_bar, p.stages, (int)(bar - full0) >> 3, ph);
      };
      if (p.im2col) produce(BoolConst<true>{}); else produce(BoolConst<false>{});
    }
  } else if (warp == kFilterWarp) {
    // ------------------------------------------------------------ producer of B ----
    if (elect_one()) {
      if (!p.b_constant) grid_dependency_wait();
      const uint32_t bytes_kb = PAIR ? 2u * b_box : b_box;
      const uint32_t sb0 = smem_u32(smem) + (uint32_t)p.bps * a_box, full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
      const uint32_t land0 = PAIR ? map_to_cta(full0, 0) : full0;
      const uint32_t full_end = full0 + 8u * (uint32_t)p.stages, to_empty = empty0 - full0, to_land = land0 - full0;
      const int bps = p.bps, kbe = p.kbe, C = p.C, batched = p.rows_per_batch;
      bool ok = true;
      uint32_t bar = full0, ph = 1, sb_stage = sb0;
      TileWalk at(p, tile_first);
      for (int tile = tile_first; tile < p.total_tiles && ok; tile += tile_step, at.next(p, tile_step)) {
        const int n0 = at.ni * p.BN + (PAIR ? rank * p.bn_load : 0);
        const int bidx = p.rows_per_batch ? ((at.mi << kPair) + rank) * BM / p.rows_per_batch : 0;
        int c0 = 0, tap = 0, left = p.num_kb;
        while (left > 0) {
          if (!mbar_try_wait_at(bar + to_empty, ph) && !mbar_wait(empty_bar + ((bar - full0) >> 3), ph, abort_flag, p.status, 8, p.spin_limit)) { ok = false; break; }
          const int nb = min(left, bps);
          left -= nb;
          if (!PAIR || rank == 0) mbar_expect_tx_at(bar, (uint32_t)nb * bytes_kb);
          const uint32_t land = bar + to_land;
          uint32_t sb = sb_stage;
          for (int j = 0; j < nb; ++j) {
            if (batched) load_3d_at<PAIR>(sb, &tmB, land, p.b_n_major ? n0 : c0, p.b_n_major ? c0 : n0, bidx);
            else load_3d_at<PAIR>(sb, &tmB, land, c0, tap, n0);
            sb += b_box;
            c0 += kbe;
            if (c0 >= C) { c0 = 0; ++tap; }
          }
          sb_stage += (uint32_t)stage_bytes;
          bar += 8;
          if (bar == full_end) { bar = full0; ph ^= 1; sb_stage = sb0; }
        }
      }
      if (!ok) await_stages(full_bar, p.stages, (int)(bar - full0) >> 3, ph);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer ----
    if (rank == 0 && elect_one()) {  // in pair mode the first CTA's lane issues for both
      // Everything that does not change from stage to stage is decided here: the pipe has about two products queued when the lane comes
      // back for the next stage, so that its instructions until then are time in which the tensor cores have nothing to do.  (One look at the
      // next stage's barrier between two products costs more than it hides: YOLOv3 of 16 pictures + 8 %.  This loop and the producers'
      // without index arithmetic: 1572 -> 1496 us, ResNet-50 of 45 images 843 -> 828.)
      auto walk = [&](auto int_is, auto four_is, auto one_is) {
        constexpr bool INT = decltype(int_is)::value, FOUR = decltype(four_is)::value, ONE = decltype(one_is)::value;   // int8; 128-byte k-blocks; one a stage
        const int ksteps = FOUR ? 4 : p.kb_bytes >> 5;  // 32 bytes of K per instruction
        const uint32_t bstep = FOUR ? 2u : (uint32_t)p.b_kstep, hi = p.desc_hi, idesc = p.idesc, BN = (uint32_t)p.BN;
        // low descriptor words of the current stage's first boxes (addresses in 16-byte units; shared memory ends below 2^18)
        const uint32_t lo0 = (1u << 16) | (smem_u32(smem) >> 4), lo_stage = (uint32_t)stage_bytes >> 4, lo_b = ((uint32_t)p.bps * a_box) >> 4;
        const uint32_t full0 = smem_u32(full_bar), full_end = full0 + 8u * (uint32_t)p.stages, to_empty = smem_u32(empty_bar) - full0, tfull0 = smem_u32(tfull_bar);
        const int num_kb = p.num_kb, bps = p.bps, total = p.total_tiles;
        uint32_t full = full0, ph = 0, tcount = 0, lo = lo0;
        for (int tile = tile_first; tile < total; tile += tile_step, ++tcount) {
          const uint32_t acc = tcount & 1, acc_ph = (tcount >> 1) & 1;
          if (!mbar_wait(&tempty_bar[acc], acc_ph ^ 1, abort_flag, p.status, 2, p.spin_limit)) return;
          tc_fence_after();
          const uint32_t tmem_d = tmem_base + acc * BN;
          uint32_t accum = 0;
          for (int left = num_kb; left > 0; left -= ONE ? 1 : bps) {
            if (!mbar_try_wait_at(full, ph) && !mbar_wait(full_bar + ((full - full0) >> 3), ph, abort_flag, p.status, 3, p.spin_limit)) return;
            tc_fence_after();
            uint32_t la = lo, lb = lo + lo_b;
            for (int j = ONE ? 1 : min(left, bps); j > 0; --j) {
              if constexpr (FOUR) {
#pragma unroll
                for (int k = 0; k < 4; ++k) issue_one<PAIR, INT>(tmem_d, desc64(la + 2 * k, hi), desc64(lb + 2 * k, hi), idesc, k ? 1u : accum);
              } else {
                for (int k = 0; k < ksteps; ++k) { issue_one<PAIR, INT>(tmem_d, desc64(la + 2 * k, hi), desc64(lb + bstep * k, hi), idesc, accum); accum = 1; }
              }
              accum = 1;
              la += a_box >> 4;
              lb += b_box >> 4;
            }
            commit_at<PAIR>(full + to_empty);  // frees the stage once these MMAs have read it
            lo += lo_stage;
            full += 8;
            if (full == full_end) { full = full0; ph ^= 1; lo = lo0; }
          }
          commit_at<PAIR>(tfull0 + 8u * acc);  // accumulator complete
          if (tcount == 0) TS(3);
        }
      };
      using Yes = BoolConst<true>;
      using No = BoolConst<false>;
      const bool four = p.kb_bytes == 128 && p.b_kstep == 2, one = p.bps == 1;
      if (!four) { if (p.acc_int) walk(Yes{}, No{}, No{}); else walk(No{}, No{}, No{}); }
      else if (p.acc_int) { if (one) walk(Yes{}, Yes{}, Yes{}); else walk(Yes{}, Yes{}, No{}); }
      else { if (one) walk(No{}, Yes{}, Yes{}); else walk(No{}, Yes{}, No{}); }
    }
  } else if (warp == kStorerWarp) {
    // -------------------------- staging ring: store finished boxes, arm them again (residual loads) ----
    if (STAGED && elect_one()) {
      grid_dependency_wait();   // earlier kernels may still read what the stores overwrite, and write the residual
      const int cols_per_box = 128 / p.out_esz;
      const uint32_t staging_u32 = smem_u32(staging);
      // Arming runs ring_boxes ahead of storing: a box is armed for its next use as soon as its store has read it.
      int a_tile = tile_first, a_bx = 0, a_slot = 0;
      uint32_t a_ph = 1;   // (as if waiting for boxes to be empty)
      TileWalk a_at(p, tile_first);
      auto arm = [&]() {
        if (a_tile >= p.total_tiles) return;
        if (p.res_tma) {
          mbar_expect_tx(box_full + a_slot, 16384u);
          tma_load_2d(staging + a_slot * 16384, &tmR, box_full + a_slot, a_at.ni * p.BN + a_bx * cols_per_box, ((a_at.mi << kPair) + rank) * BM);
        } else {
          mbar_arrive(box_full + a_slot);
        }
        if (++a_slot == p.ring_boxes) { a_slot = 0; a_ph ^= 1; }
        if (++a_bx == p.stage_boxes || a_at.ni * p.BN + a_bx * cols_per_box >= p.K_out) { a_bx = 0; a_tile += tile_step; a_at.next(p, tile_step); }
      };
      for (int b = 0; b < p.ring_boxes; ++b) arm();
      int slot = 0;
      bool unread = false;   // the newest store may still be reading its box
      uint32_t ph = 0;
      bool ok = true;
      TileWalk at(p, tile_first);
      for (int tile = tile_first; tile < p.total_tiles && ok; tile += tile_step, at.next(p, tile_step)) {
        const int m0 = ((at.mi << kPair) + rank) * BM, n0 = at.ni * p.BN;
        for (int bx = 0; bx < p.stage_boxes; ++bx) {
          const int x0 = n0 + bx * cols_per_box;
          if (x0 >= p.K_out) break;
          // Nothing to send yet: use the wait to let the last store finish reading its box and hand that box back,
          // so that the next tile's epilogue never waits for this tile's boxes to be stored.
          if (!mbar_try_wait(box_done + slot, ph)) {
            if (unread) {
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
              arm();
              unread = false;
            }
            if (!mbar_wait(box_done + slot, ph, abort_flag, p.status, 7, p.spin_limit)) { ok = false; break; }
          }
          if (p.store_mode == 0) {
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"((uint64_t)&tmY),
                         "r"(staging_u32 + (uint32_t)slot * 16384u), "r"(x0), "r"(m0)
                         : "memory");
          } else {
            // the 128 rows of the box are one run of sequence positions of one batch element; its columns one head
            const int g = m0 / p.store_S, s0 = m0 - g * p.store_S;
            int c1, c2, c3;
            if (p.store_mode == 1) { c1 = s0; c2 = x0 / cols_per_box; c3 = g; }                                   // [B][NH][S][D]
            else { const int b = g / p.store_NH; c1 = g - b * p.store_NH; c2 = s0; c3 = b; }                      // [B][S][NH][D]
            asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"((uint64_t)&tmY),
                         "r"(staging_u32 + (uint32_t)slot * 16384u), "r"(0), "r"(c1), "r"(c2), "r"(c3)
                         : "memory");
          }
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          if (unread) {
            asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // every store but the newest has read its box
            arm();
          }
          unread = true;
          if (++slot == p.ring_boxes) { slot = 0; ph ^= 1; }
        }
      }
      if (!ok && p.res_tma) await_stages(box_full, p.ring_boxes, a_slot, a_ph);
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // stores complete before shared memory is released
    }
  } else {
    // ---------------------------------------------------------------- epilogue ----
    const int quarter = warp & 3;  // the TMEM lanes this warp may read: 32*quarter .. +31
    const int cgroup = (warp - 2) >> 2;  // the warps of a quarter take the 32-column chunks round-robin
    uint32_t tcount = 0;
    bool ok = true;
    constexpr int kGroups = kEpilogueWarps / 4;            // warps per TMEM lane quarter
    constexpr int kChunksPerWarp = 8 / kGroups;            // BN <= 256 -> at most 8 chunks of 32 columns
    const int r_in_tile = quarter * 32 + lane;
    const uint32_t staging_u32 = smem_u32(staging);
    if constexpr (STAGED) {
      // Per output tile the staging ring supplies stage_boxes boxes of 128 rows x 128 bytes; the
      // storer warp has already had the residual put there, this warp overwrites its part of the box
      // with the result and the storer warp sends the box out.
      const int cols_per_box = 128 / p.out_esz, chunks_per_box = cols_per_box / CW;
      // Which 16-column chunks of a tile the four warps of a group (one per lane quarter) take: either a
      // contiguous run, so that a group fills and hands over a box (or its share of one) on its own while the
      // other groups work on other boxes, or every fourth chunk, so that all groups finish box after box together.
      const int n_chunks = p.BN / CW, per_group = n_chunks / kGroups;  // per group: 1, 2 or 4 chunks
      const int ch_lo = cgroup * per_group, ch_hi = ch_lo + per_group;
      int slot = 0;
      uint32_t ph = 0;
      // ReLU of the straight-line forms: the lower clamp of an int8 output, a packed floor for 16-bit outputs
      const bool fast_relu = p.ep.act == ACT_RELU;
      const float fast_lo = fast_relu ? 0.f : -128.f;
      const uint32_t fast_floor = fast_relu ? 0u : (OUT == DT_F16 ? 0xFC00FC00u : 0xFF80FF80u);
      TileWalk at(p, tile_first);
      for (int tile = tile_first; tile < p.total_tiles && ok; tile += tile_step, ++tcount, at.next(p, tile_step)) {
        const uint32_t acc = tcount & 1, acc_ph = (tcount >> 1) & 1;
        const int n0 = at.ni * p.BN;
        if (!mbar_wait(&tfull_bar[acc], acc_ph, abort_flag, p.status, 4, p.spin_limit)) { ok = false; break; }
        tc_fence_after();
        if (tcount == 0 && threadIdx.x == 64) TS(4);
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * (uint32_t)p.BN;
        for (int bx = 0; bx < p.stage_boxes && ok; ++bx) {
          if (n0 + bx * cols_per_box >= p.K_out) break;
          int first, last, step;
          if (p.epi_interleave) { first = bx * chunks_per_box + cgroup; last = min((bx + 1) * chunks_per_box, n_chunks); step = kGroups; }
          else { first = max(ch_lo, bx * chunks_per_box); last = min(ch_hi, (bx + 1) * chunks_per_box); step = 1; }
          if (first < last) {
            if (!mbar_wait(box_full + slot, ph, abort_flag, p.status, 6, p.spin_limit)) { ok = false; break; }
            StagePos sp;
            sp.row_addr = staging_u32 + (uint32_t)slot * 16384u + (uint32_t)r_in_tile * 128u;
            sp.rxor = r_in_tile & 7;
            if constexpr (MODE == 1) {
              // straight-line forms, chosen once per launch on the host (p.fast_variant = ACC * 2 + RES)
              switch (p.fast_variant) {
                case 0: box_fast<OUT, 0, false>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp, fast_lo, fast_floor); break;
                case 1: box_fast<OUT, 0, true>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp, fast_lo, fast_floor); break;
                case 2: box_fast<OUT, 1, false>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp, fast_lo, fast_floor); break;
                case 3: box_fast<OUT, 1, true>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp, fast_lo, fast_floor); break;
                case 4: box_fast<OUT, 2, false>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp, fast_lo, fast_floor); break;
                default: box_fast<OUT, 2, true>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp, fast_lo, fast_floor); break;
              }
            } else if constexpr (MODE == 3) {
              if constexpr (OUT == DT_S8) {
                if (p.ep.acc_small) box_gelu_s8<2>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp);
                else box_gelu_s8<1>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp);
              }
              if constexpr (OUT == DT_F16 || OUT == DT_BF16) {
                if (p.ep.act == ACT_GELU_ERF) box_leaky<OUT, 1, false>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp);
                else if (p.ep.res) box_leaky<OUT, 0, true>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp);
                else box_leaky<OUT, 0, false>(p, taddr, first, last, step, n0, bx, chunks_per_box, sp);
              }
            } else {
#pragma unroll 1
            for (int ch = first; ch < last; ch += step) {
              const int col0 = n0 + ch * CW;
              if (col0 >= p.K_out) break;  // columns past K_out inside a chunk are computed and then clipped by the store
              uint32_t r[CW];
              tmem_ld<CW>(taddr + (uint32_t)(ch * CW), r);
              tmem_ld_wait_regs<CW>(r);
              float v[CW];
              if (p.acc_int) {
                if (p.ep.acc_small) {
#pragma unroll
                  for (int j = 0; j < CW; j += 2) {
                    v[j] = __uint_as_float(r[j] + kMagicBits); v[j + 1] = __uint_as_float(r[j + 1] + kMagicBits);
                    fadd2_rn(v[j], v[j + 1], -kMagic, -kMagic);
                  }
                } else {
#pragma unroll
                  for (int j = 0; j < CW; ++j) v[j] = (float)(int32_t)r[j];
                }
              } else {
#pragma unroll
                for (int j = 0; j < CW; ++j) v[j] = __uint_as_float(r[j]);
              }
              sp.j0 = ((ch - bx * chunks_per_box) * CW * p.out_esz) >> 4;
              epilogue_chunk_staged<OUT, true>(p, v, col0, sp);
            }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the bulk-copy engine must see these writes
            __syncwarp();
            if (lane == 0) mbar_arrive(box_done + slot);
          }
          if (++slot == p.ring_boxes) { slot = 0; ph ^= 1; }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { if (PAIR && rank) mbar_arrive_cluster(map_to_cta(smem_u32(&tempty_bar[acc]), 0)); else mbar_arrive(&tempty_bar[acc]); }
        if (tcount == 0 && threadIdx.x == 64) TS(5);
      }
    } else {
      // Direct epilogue: rows go straight to global memory.  Residual rows can be fetched before the
      // accumulator is ready: they only depend on the tile.
      grid_dependency_wait();
      const bool res_vec = p.ep.res && (p.K_out & 15) == 0 && (p.ep.res_dt == DT_F16 || p.ep.res_dt == DT_BF16 || p.ep.res_dt == DT_S8);
      const int res_q = p.ep.res_dt == DT_S8 ? 2 : 4;       // 16-byte pieces per 32 channels
      const int res_esz = p.ep.res_dt == DT_S8 ? 1 : 2;
      for (int tile = tile_first; tile < p.total_tiles && ok; tile += tile_step, ++tcount) {
        const uint32_t acc = tcount & 1, acc_ph = (tcount >> 1) & 1;
        const int m0 = (((tile % p.m_tiles) << kPair) + rank) * BM, n0 = (tile / p.m_tiles) * p.BN;
        const int64_t row = (int64_t)m0 + r_in_tile;
        uint4 pre[kChunksPerWarp][4] = {};
        bool pre_ok[kChunksPerWarp] = {};
#pragma unroll
        for (int i = 0; i < kChunksPerWarp; ++i) {
          const int c = (cgroup + kGroups * i) * 32, col0 = n0 + c;
          pre_ok[i] = res_vec && c < p.BN && row < p.M_total && col0 + 32 <= p.K_out;
          if (pre_ok[i]) {
            const uint4* rp = (const uint4*)((const char*)p.ep.res + (row * p.K_out + col0) * res_esz);
#pragma unroll
            for (int q = 0; q < 4; ++q) if (q < res_q) pre[i][q] = __ldg(rp + q);
          }
        }
        if (!mbar_wait(&tfull_bar[acc], acc_ph, abort_flag, p.status, 4, p.spin_limit)) { ok = false; break; }
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * (uint32_t)p.BN;
#pragma unroll
        for (int i = 0; i < kChunksPerWarp; ++i) {
          const int c = (cgroup + kGroups * i) * 32, col0 = n0 + c;
          if (c >= p.BN || col0 >= p.K_out) break;  // uniform across the warp
          uint32_t r[32];
          tmem_ld32(taddr + (uint32_t)c, r);
          tmem_ld_wait();
          const int ncols = min(32, p.K_out - col0);
          if (p.ep.out_dt == DT_S32) {
            if (row < p.M_total) {
              int32_t* out = (int32_t*)p.y + row * p.K_out + col0;
#pragma unroll
              for (int j = 0; j < 32; ++j) if (j < ncols) out[j] = (int32_t)r[j];
            }
          } else if (row < p.M_total) {
            float v[32];
            if (p.acc_int) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = (float)(int32_t)r[j];
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            }
            StagePos sp = {0, 0, 0};
            epilogue_chunk<OUT, false, 32>(p, v, row, col0, ncols, pre[i], pre_ok[i], sp, false);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { if (PAIR && rank) mbar_arrive_cluster(map_to_cta(smem_u32(&tempty_bar[acc]), 0)); else mbar_arrive(&tempty_bar[acc]); }
      }
    }
  }
  // ------------------------------------------------------------------ teardown ----
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) TS(6);
  if constexpr (PAIR) cluster_sync_all();  // neither CTA leaves (or frees tensor memory) while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols) : "memory");
  }
}

// ------------------------------------------------------- few tiles: split reductions ----
// A launch whose tiles leave most of the chip idle (a batch of one, the deep layers of a few images, a classifier) is bound by
// the serial walk of each tile over its k-blocks, not by any throughput.  Here the 2 to 8 CTAs of a cluster share a tile of 64
// or 128 rows by 16 to 64 columns: each walks a contiguous share of the k-blocks, leaves its 32-bit partial tile in its own
// shared memory, and after a cluster barrier adds up, finishes and stores a share of the rows, reading its peers' partials in
// rank order, so that the result does not depend on timing (int32 partial sums are exact).  Residuals are fetched while the
// products run.
constexpr int kSplitThreads = 352, kSplitEpiWarps = 8;   // producer of A, MMA issuer, eight warps that empty tensor memory, producer of B
constexpr int kSplitRows = 4;                             // rows one thread finishes, at most (128 rows x 16 pieces / 2 CTAs / 256 threads)
struct SplitShared { uint64_t full[8], empty[8], done; uint32_t tmem; int abort; };
static_assert(offsetof(SplitShared, empty) == 64 && offsetof(SplitShared, done) == 128, "the barriers are initialised as one array");

// What four neighbouring columns need from the epilogue's per-channel vectors; one thread keeps the same columns for all its rows.
struct FourColumns { float mul[4], add1[4], add2[4]; };
__device__ __forceinline__ void load_four_columns(const Epilogue& ep, int col, FourColumns& f) {
  auto vec = [&](const float* src, float (&o)[4]) { const float4 v = __ldg((const float4*)(src + col)); o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; };
  if (ep.mul) vec(ep.mul, f.mul);
  if (ep.add1) vec(ep.add1, f.add1);
  if (ep.add2) vec(ep.add2, f.add2);
}
// The residual of four neighbouring results as it lies in memory (up to 16 bytes).
__device__ __forceinline__ uint4 load_four_residuals(const Epilogue& ep, int64_t at) {
  uint4 u = make_uint4(0, 0, 0, 0);
  if (ep.res_dt == DT_F16 || ep.res_dt == DT_BF16) { const uint2 t = *(const uint2*)((const uint16_t*)ep.res + at); u.x = t.x; u.y = t.y; }
  else if (ep.res_dt == DT_S8) u.x = *(const uint32_t*)((const int8_t*)ep.res + at);
  else u = *(const uint4*)((const float*)ep.res + at);
  return u;
}
// Finishes and stores four neighbouring results of one row, with the arithmetic of epilogue_value (every step rounded by itself).
__device__ __forceinline__ void finish_four(const UmmaParams& p, float (&v)[4], int64_t row, int col, const FourColumns& f, const uint4& res) {
  const Epilogue& ep = p.ep;
  if (ep.mul) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __fmul_rn(v[j], f.mul[j]);
  }
  if (ep.alpha != 1.f) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __fmul_rn(v[j], ep.alpha);
  }
  if (ep.add1) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __fadd_rn(v[j], f.add1[j]);
  }
  if (ep.add2) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __fadd_rn(v[j], f.add2[j]);
  }
  if (ep.act_first) apply_act_all<4>(ep.act, v, ep.act_a, ep.act_b);
  if (ep.res) {
    const uint32_t w[4] = {res.x, res.y, res.z, res.w};
    float r[4];
    if (ep.res_dt == DT_F16 || ep.res_dt == DT_BF16) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const float2 h = ep.res_dt == DT_F16 ? __half22float2(*(const __half2*)&w[t]) : __bfloat1622float2(*(const __nv_bfloat162*)&w[t]);
        r[2 * t] = h.x; r[2 * t + 1] = h.y;
      }
    } else if (ep.res_dt == DT_S8) {
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = __fmul_rn((float)(signed char)(w[0] >> (8 * j)), ep.res_scale);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = __uint_as_float(w[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __fadd_rn(v[j], r[j]);
  }
  if (!ep.act_first) apply_act_all<4>(ep.act, v, ep.act_a, ep.act_b);
  const int64_t at = row * p.y_ld + col;
  if (ep.out_dt == DT_F16 || ep.out_dt == DT_BF16) {
    uint2 u;
    uint32_t* w = (uint32_t*)&u;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (ep.out_dt == DT_F16) { const __half2 h = __floats2half2_rn(v[2 * t], v[2 * t + 1]); w[t] = *(const uint32_t*)&h; }
      else { const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * t], v[2 * t + 1]); w[t] = *(const uint32_t*)&h; }
    }
    *(uint2*)((uint16_t*)p.y + at) = u;
  } else if (ep.out_dt == DT_S8) {
    uint32_t q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = (uint32_t)rne_sat_s8(ep.out_multiply ? __fmul_rn(v[j], ep.out_inv) : __fdiv_rn(v[j], ep.out_scale));
    *(uint32_t*)((int8_t*)p.y + at) = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
  } else {
    *(float4*)((float*)p.y + at) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// The form nearly every layer of a two-byte network has: fp32 sums, one per-channel addend, a residual of the result's type, ReLU or LeakyReLU
// (p.split_plain, decided when planning).  The same steps as finish_four, without its twenty decisions on the way of every result.
template <bool BF16>
__device__ __forceinline__ void finish_plain(const UmmaParams& p, float (&v)[4], int64_t row, int col, const float4& add, const uint4& res) {
  const Epilogue& ep = p.ep;
  const float a[4] = {add.x, add.y, add.z, add.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = __fadd_rn(v[j], a[j]);
  if (ep.act == ACT_LEAKY && ep.act_first) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = apply_act(ACT_LEAKY, v[j], ep.act_a, 0.f);
  }
  if (ep.res) {
    const uint32_t w[2] = {res.x, res.y};
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const float2 h = BF16 ? __bfloat1622float2(*(const __nv_bfloat162*)&w[t]) : __half22float2(*(const __half2*)&w[t]);
      v[2 * t] = __fadd_rn(v[2 * t], h.x);
      v[2 * t + 1] = __fadd_rn(v[2 * t + 1], h.y);
    }
  }
  if (ep.act == ACT_RELU) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = apply_act(ACT_RELU, v[j], 0.f, 0.f);
  } else if (ep.act == ACT_LEAKY && !ep.act_first) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = apply_act(ACT_LEAKY, v[j], ep.act_a, 0.f);
  }
  uint2 u;
  uint32_t* w = (uint32_t*)&u;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    if (BF16) { const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * t], v[2 * t + 1]); w[t] = *(const uint32_t*)&h; }
    else { const __half2 h = __floats2half2_rn(v[2 * t], v[2 * t + 1]); w[t] = *(const uint32_t*)&h; }
  }
  *(uint2*)((uint16_t*)p.y + row * p.y_ld + col) = u;
}

__global__ void __launch_bounds__(kSplitThreads, 2)
umma_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const UmmaParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int stage_bytes = p.bps * (p.bm + p.bn_load) * p.kb_bytes;
  SplitShared& sh = *(SplitShared*)(smem + p.split_data_bytes);
  volatile int* abort_flag = &sh.abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int swz = p.BN >= 32 ? 7 : 3;   // a row of the partial tile has BN / 4 pieces, at least 4
  const int rank = (int)blockIdx.x % p.splits, tile = (int)blockIdx.x / p.splits;
  if (warp == 0) {   // a lane per barrier
    if (lane < 17) mbar_init(&sh.full[lane], lane < 8 ? 2u : 1u);
    if (lane == 0) { sh.abort = 0; prefetch_map(&tmA); prefetch_map(&tmB); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)), "r"((uint32_t)p.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;
  const uint32_t a_box = (uint32_t)(p.bm * p.kb_bytes), b_box = (uint32_t)(p.bn_load * p.kb_bytes);
  const int ni = tile / p.m_tiles, m0 = (tile - ni * p.m_tiles) * p.bm, n0 = ni * p.BN;
  const int kb_lo = (int)((int64_t)p.num_kb * rank / p.splits), kb_hi = (int)((int64_t)p.num_kb * (rank + 1) / p.splits);
  // A thread's place in the final pass: four columns, the same for all its rows (the pass's 256 threads span whole rows).
  const int per_row = p.BN >> 2, t = (int)threadIdx.x - 64, c4 = t & (per_row - 1), col = n0 + 4 * c4, row_step = (kSplitEpiWarps * 32) / per_row;
  const int rows = min(p.bm, p.M_total - m0), r_lo = rows * rank / p.splits, r_hi = rows * (rank + 1) / p.splits;
  const bool vec = (p.K_out & 3) == 0, finisher = warp >= 2 && warp < 2 + kSplitEpiWarps && col < p.K_out;
  FourColumns fc;
  float4 plain_add = make_float4(0.f, 0.f, 0.f, 0.f);
  uint4 res[kSplitRows];
  if (warp == 0 || warp == 2 + kSplitEpiWarps) {
    // ------------------------------------------------------------ producers of A and B ----
    if (elect_one()) {
      const bool do_a = warp == 0;
      if (do_a || !p.b_constant) grid_dependency_wait();
      if (do_a) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
      int w0 = 0, h0 = 0, img = 0;
      if (do_a && p.im2col) {
        const int pq = p.P * p.Q;
        img = m0 / pq;
        const int rem = m0 - img * pq, op = rem / p.Q, oq = rem - op * p.Q;
        w0 = oq * p.stride_w - p.pad_l;
        h0 = op * p.stride_h - p.pad_t;
      }
      const int bidx = p.rows_per_batch ? m0 / p.rows_per_batch : 0;
      int tap = kb_lo / p.chunks_per_tap, c0 = (kb_lo - tap * p.chunks_per_tap) * p.kbe;
      int fr = (tap % (p.R * p.S)) / p.S, fs = tap % p.S, left = kb_hi - kb_lo, s = 0;
      uint32_t ph = 1;
      const uint32_t first = smem_u32(smem) + (do_a ? 0u : (uint32_t)p.bps * a_box), box = do_a ? a_box : b_box;
      uint32_t at_stage = first;
      bool ok = true;
      while (left > 0) {
        if (!mbar_wait(&sh.empty[s], ph, abort_flag, p.status, do_a ? 21 : 23, p.spin_limit)) { ok = false; break; }
        const int nb = left < p.bps ? left : p.bps;
        left -= nb;
        const bool skip = do_a && p.test_skip_stage && blockIdx.x == 0 && left == 0;   // (the test hook of the persistent kernel)
        const uint32_t land = smem_u32(&sh.full[s]);
        if (!skip) mbar_expect_tx_at(land, (uint32_t)nb * box);
        uint32_t dst = at_stage;
        for (int j = skip ? nb : 0; j < nb; ++j) {
          if (!do_a) {
            if (p.rows_per_batch) load_3d_at<false>(dst, &tmB, land, p.b_n_major ? n0 : c0, p.b_n_major ? c0 : n0, bidx);
            else load_3d_at<false>(dst, &tmB, land, c0, tap, n0);
          } else if (p.im2col) load_im2col_at<false>(dst, &tmA, land, c0, w0, h0, img, (uint16_t)fs, (uint16_t)fr);
          else load_2d_at<false>(dst, &tmA, land, c0, m0);
          dst += box;
          c0 += p.kbe;
          if (c0 >= p.C) { c0 = 0; ++tap; if (++fs == p.S) { fs = 0; if (++fr == p.R) fr = 0; } }
        }
        at_stage += (uint32_t)stage_bytes;
        if (++s == p.stages) { s = 0; ph ^= 1; at_stage = first; }
      }
      if (!ok) await_stages(sh.full, p.stages, s, ph);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      int s = 0, left = kb_hi - kb_lo;
      uint32_t ph = 0, accum = 0;
      const int ksteps = p.kb_bytes >> 5;
      const uint32_t lo0 = (1u << 16) | (smem_u32(smem) >> 4), lo_stage = (uint32_t)stage_bytes >> 4, lo_b = ((uint32_t)p.bps * a_box) >> 4;
      uint32_t lo = lo0;
      bool ok = true;
      while (left > 0) {
        if (!mbar_wait(&sh.full[s], ph, abort_flag, p.status, 22, p.spin_limit)) { ok = false; break; }
        tc_fence_after();
        const int nb = left < p.bps ? left : p.bps;
        left -= nb;
        uint32_t la = lo, lb = lo + lo_b;
        for (int j = 0; j < nb; ++j) {
          issue_kblock(p, tmem, la, lb, ksteps, accum);
          accum = 1;
          la += a_box >> 4;
          lb += b_box >> 4;
        }
        umma_commit(&sh.empty[s]);
        lo += lo_stage;
        if (++s == p.stages) { s = 0; ph ^= 1; lo = lo0; }
      }
      if (ok) umma_commit(&sh.done);
    }
  } else {
    if (finisher && p.split_plain) plain_add = __ldg((const float4*)((p.ep.add1 ? p.ep.add1 : p.ep.add2) + col));
    else if (finisher && vec) load_four_columns(p.ep, col, fc);
    grid_dependency_wait();   // residuals are read, and tensors earlier kernels may still read overwritten, from here on
    if (finisher && vec && p.ep.res) {
#pragma unroll
      for (int i = 0; i < kSplitRows; ++i) {
        const int r = r_lo + t / per_row + i * row_step;
        if (r < r_hi) res[i] = load_four_residuals(p.ep, ((int64_t)m0 + r) * p.K_out + col);
      }
    }
    // the accumulators go to shared memory as 16-byte pieces, row r's piece c at c ^ (r & 7): rows apart by whole bank cycles
    // are then written, and neighbouring pieces of a row read, without conflicts
    // (64-row products occupy the first 16 lanes of every quarter of tensor memory)
    const int quarter = warp & 3, r = p.bm == 64 ? quarter * 16 + (lane & 15) : quarter * 32 + lane;
    const bool lane_ok = p.bm == 128 || lane < 16;
    if (mbar_wait(&sh.done, 0, abort_flag, p.status, 24, p.spin_limit)) {
      tc_fence_after();
      const uint32_t row_at = smem_u32(smem) + (uint32_t)(r * p.BN * 4);
      for (int c = (warp - 2) >> 2; c < p.BN / 16; c += kSplitEpiWarps / 4) {
        uint32_t v[16];
        tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(c * 16), v);
        tmem_ld_wait_regs<16>(v);
        if (lane_ok) {
#pragma unroll
          for (int q = 0; q < 4; ++q) sts128(row_at + (uint32_t)(((4 * c + q) ^ (r & swz)) << 4), make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)p.tmem_cols) : "memory");
  }
  if (finisher) {
    const uint32_t base = smem_u32(smem);
#pragma unroll
    for (int i = 0; i < kSplitRows; ++i) {
      const int r = r_lo + t / per_row + i * row_step;
      if (r >= r_hi) break;
      const uint32_t at = base + (uint32_t)(r * p.BN * 4) + (uint32_t)((c4 ^ (r & swz)) << 4);
      const int64_t row = (int64_t)m0 + r;
      uint4 u[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < p.splits)
          asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u[k].x), "=r"(u[k].y), "=r"(u[k].z), "=r"(u[k].w) : "r"(map_to_cta(at, (uint32_t)k)) : "memory");
      float v[4];
      if (p.acc_int) {
        int4 a = make_int4((int)u[0].x, (int)u[0].y, (int)u[0].z, (int)u[0].w);
#pragma unroll
        for (int k = 1; k < 8; ++k) if (k < p.splits) { a.x += (int)u[k].x; a.y += (int)u[k].y; a.z += (int)u[k].z; a.w += (int)u[k].w; }
        if (p.ep.out_dt == DT_S32) {
          const int raw[4] = {a.x, a.y, a.z, a.w};
          for (int j = 0; j < 4 && col + j < p.K_out; ++j) ((int32_t*)p.y)[row * p.K_out + col + j] = raw[j];
          continue;
        }
        v[0] = (float)a.x; v[1] = (float)a.y; v[2] = (float)a.z; v[3] = (float)a.w;
      } else {
        v[0] = __uint_as_float(u[0].x); v[1] = __uint_as_float(u[0].y); v[2] = __uint_as_float(u[0].z); v[3] = __uint_as_float(u[0].w);
#pragma unroll
        for (int k = 1; k < 8; ++k)
          if (k < p.splits) { v[0] += __uint_as_float(u[k].x); v[1] += __uint_as_float(u[k].y); v[2] += __uint_as_float(u[k].z); v[3] += __uint_as_float(u[k].w); }
      }
      if (p.split_plain) { if (p.ep.out_dt == DT_BF16) finish_plain<true>(p, v, row, col, plain_add, res[i]); else finish_plain<false>(p, v, row, col, plain_add, res[i]); }
      else if (vec && !p.ep.add_full) finish_four(p, v, row, col, fc, res[i]);
      else
        for (int j = 0; j < 4 && col + j < p.K_out; ++j) store_from_float(p.y, p.ep.out_dt, row * p.y_ld + col + j, epilogue_value(p.ep, v[j], row, col + j, p.K_out));
    }
  }
  cluster_sync_all();   // nobody leaves while a peer may still read its partial tile
}

// ------------------------------------------------------------ fused attention ----
// softmax(scale * Q K^T) V for heads of 64 channels and any number of positions (two-byte types).  One CTA works on one
// block of 128 query rows of one head at a time and keeps the scores of 128 x 128 (query, key) pairs in tensor memory -- they
// never reach global memory.  Roles: warp 0 brings Q, K, V in with TMA and sends the result out, warp 1 issues the two
// products, warps 2-5 (one TMEM lane quarter each, a thread per query row) do the soft-max between them and the final
// scaling.  Shared memory holds one block (no double buffer) and is reused inside it -- the probabilities overwrite K
// (and Q when it is not needed again), the result accumulates over the scores' tensor memory columns, the result box overwrites
// V -- so that four (three) CTAs share an SM and fill each other's gaps.  The probabilities go to the second product
// unnormalised (exp(s - max), rounded to the two-byte type) and the row sums divide the result, as in any online soft-max.
//
// MULTI = false: up to 128 positions, one key block.  MULTI = true: the key blocks of a row follow one another; each block's
// product is read back and added to the row's 64 running results in registers, which are rescaled when the maximum moves.
// A sequence that does not fill its last block needs no padding anywhere: TMA zero-fills loads and clips stores past the
// last position, the products shrink to the next multiple of 16 keys and the soft-max masks the rest.
struct AttnParams {
  int tiles, NH, S, q_tiles, k_blocks;   // query blocks in all; heads per batch element; positions; blocks per head
  int qkv_rows;                  // 0: q, k, v lie [B][NH][S][D]; 1: heads are 64-column groups of [B * S] rows
  int merge;                     // 1: the result is stored [B][S][NH][D], 0: [B][NH][S][D]
  float scale_log2e;             // scale * log2(e)
  uint32_t idesc_s, idesc_s_last, idesc_o, desc_hi;   // (the last key block's scores product may be narrower)
  int last_keys, last_ksteps;    // keys in the last block, and 16-key steps of its second product
  uint32_t spin_limit;
  int* status;
};
constexpr int kAttnS = 128, kAttnD = 64, kAttnThreads = 192;
constexpr uint32_t kAttnBox = 16384;   // 128 rows x 128 bytes

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(dst)),
               "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}

template <bool BF16, bool MULTI>
__global__ void __launch_bounds__(kAttnThreads, MULTI ? 3 : 4)
attn_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
            const __grid_constant__ CUtensorMap tmY, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;                 // [128 rows][64] K-major
  uint8_t* sK = sQ + kAttnBox;        // [128 keys][64] K-major
  uint8_t* sP = MULTI ? sK : sQ;      // two k-blocks of [128 rows][64 keys], written once the first product has read its operands
  uint8_t* sV = sP + 2 * kAttnBox;    // [128 keys][64 channels]: the second product reads it MN-major
  uint8_t* sY = sV;                   // result box, written once the last second product has read V
  uint64_t* bars = (uint64_t*)(sV + kAttnBox);
  uint64_t *b_full = bars, *b_s = bars + 1, *b_p = bars + 2, *b_o = bars + 3, *b_e = bars + 4;
  uint32_t* tmem_slot = (uint32_t*)(bars + 8);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(b_full, 1); mbar_init(b_s, 1); mbar_init(b_p, 4); mbar_init(b_o, 1); mbar_init(b_e, 4);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(128u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem_s = tmem_base, tmem_o = tmem_base;   // the result's 64 columns replace the first 64 of the scores
  const int k_blocks = MULTI ? p.k_blocks : 1;
  // `n` counts key blocks over all of this CTA's query blocks: its parity is the phase of every barrier

  if (warp == 0) {
    // ------------------------------------------------ loads and the result's store ----
    if (elect_one()) {
      uint32_t n = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
        const int head = MULTI ? tile / p.q_tiles : tile, q0 = MULTI ? (tile - head * p.q_tiles) * kAttnS : 0;
        const int b = head / p.NH, h = head - b * p.NH;
        auto load = [&](uint8_t* dst, const CUtensorMap* map, int s0) {
          if (p.qkv_rows) tma_load_4d(dst, map, b_full, 0, h, s0, b); else tma_load_4d(dst, map, b_full, 0, s0, h, b);
        };
        for (int kb = 0; kb < k_blocks; ++kb, ++n) {
          // the previous block's products have finished reading Q, K, V and P
          if (n > 0 && !mbar_wait(b_o, (n - 1) & 1, abort_flag, p.status, 11, p.spin_limit)) { ok = false; break; }
          mbar_expect_tx(b_full, (kb == 0 ? 3u : 2u) * kAttnBox);
          if (kb == 0) load(sQ, &tmQ, q0);
          load(sK, &tmK, kb * kAttnS);
          load(sV, &tmV, kb * kAttnS);
        }
        // (a wait may lag one phase behind, not two: with b_o of the last block complete, b_e of the one before it is as well)
        if (!ok || (MULTI && !mbar_wait(b_o, (n - 1) & 1, abort_flag, p.status, 11, p.spin_limit))) break;
        if (!mbar_wait(b_e, (n - 1) & 1, abort_flag, p.status, 12, p.spin_limit)) break;
        if (p.merge)
          asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"((uint64_t)&tmY), "r"(smem_u32(sY)), "r"(0),
                       "r"(h), "r"(q0), "r"(b)
                       : "memory");
        else
          asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"((uint64_t)&tmY), "r"(smem_u32(sY)), "r"(0),
                       "r"(q0), "r"(h), "r"(b)
                       : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the box is V again: the next loads are issued by this thread
      }
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
      if (*abort_flag && n > 0) await_landing(b_full, (n - 1) & 1);   // (armed but never consumed)
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------- the two products ----
    if (elect_one()) {
      const uint64_t fixed = ((uint64_t)p.desc_hi << 32) | (1ull << 16);
      const uint64_t dq = fixed | (uint64_t)((smem_u32(sQ) & 0x3FFFF) >> 4), dk = fixed | (uint64_t)((smem_u32(sK) & 0x3FFFF) >> 4);
      const uint64_t dv = fixed | (uint64_t)((smem_u32(sV) & 0x3FFFF) >> 4), dp = fixed | (uint64_t)((smem_u32(sP) & 0x3FFFF) >> 4);
      uint32_t n = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x)
        for (int kb = 0; kb < k_blocks; ++kb, ++n) {
          const bool last = kb + 1 == k_blocks;
          if (!mbar_wait(b_full, n & 1, abort_flag, p.status, 13, p.spin_limit)) { ok = false; break; }
          // the previous block's result has been read from the columns the scores go to
          if (MULTI && n > 0 && !mbar_wait(b_e, (n - 1) & 1, abort_flag, p.status, 17, p.spin_limit)) { ok = false; break; }
          tc_fence_after();
          const uint32_t idesc_s = last ? p.idesc_s_last : p.idesc_s;
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16(tmem_s, dq + 2 * k, dk + 2 * k, idesc_s, k ? 1u : 0u);        // S = Q K^T, 64 deep
          umma_commit(b_s);
          if (!mbar_wait(b_p, n & 1, abort_flag, p.status, 14, p.spin_limit)) { ok = false; break; }
          tc_fence_after();
          const int ksteps = last ? p.last_ksteps : 8;
          for (int k = 0; k < ksteps; ++k)   // O = P V: P advances 32 bytes per step inside a k-block, V sixteen rows
            umma_f16(tmem_o, dp + (uint64_t)((k >> 2) * (kAttnBox >> 4) + 2 * (k & 3)), dv + (uint64_t)(128 * k), p.idesc_o, k ? 1u : 0u);
          umma_commit(b_o);
        }
    }
  } else {
    // ------------------------------------------------ soft-max and the final scaling ----
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t p_row = smem_u32(sP) + (uint32_t)row * 128u, y_row = smem_u32(sY) + (uint32_t)row * 128u;
    const int rx = row & 7;
    uint32_t n = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
      // a warp whose 32 rows all lie past the last position has nothing to compute: what it leaves in shared memory only
      // reaches rows that the store clips
      const bool live = (MULTI ? (tile % p.q_tiles) * kAttnS : 0) + quarter * 32 < p.S;
      float run_max = -3.402823466e+38f, sum = 0.f;
      float o[MULTI ? kAttnD : 1];
      if (MULTI) {
#pragma unroll
        for (int j = 0; j < (MULTI ? kAttnD : 1); ++j) o[j] = 0.f;
      }
      for (int kb = 0; kb < k_blocks; ++kb, ++n) {
        const bool last = kb + 1 == k_blocks;
        const int keys = last ? p.last_keys : kAttnS, chunks = (keys + 15) >> 4;
        if (!mbar_wait(b_s, n & 1, abort_flag, p.status, 15, p.spin_limit)) { ok = false; break; }
        tc_fence_after();
        float corr = 0.f;
        if (live) {
          float mx = run_max;
#pragma unroll 1
          for (int c = 0; c < chunks; ++c) {
            uint32_t r[16];
            tmem_ld16(tmem_s + lane_addr + (uint32_t)(c * 16), r);
            tmem_ld_wait_regs<16>(r);
            if (c * 16 + 16 <= keys) {
#pragma unroll
              for (int j = 0; j < 16; ++j) mx = fmaxf(mx, __uint_as_float(r[j]) * p.scale_log2e);
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) if (c * 16 + j < keys) mx = fmaxf(mx, __uint_as_float(r[j]) * p.scale_log2e);
            }
          }
          if (MULTI) {
            corr = run_max - mx;   // 1 when the maximum has not moved, 0 for the first block
            asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(corr));
            sum *= corr;
            run_max = mx;
          }
#pragma unroll 1
          for (int c = 0; c < chunks; ++c) {
            uint32_t r[16];
            tmem_ld16(tmem_s + lane_addr + (uint32_t)(c * 16), r);
            tmem_ld_wait_regs<16>(r);
            float e[16];
            const bool whole = c * 16 + 16 <= keys;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              e[j] = fmaf(__uint_as_float(r[j]), p.scale_log2e, -mx);
              asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e[j]));
              if (!whole && c * 16 + j >= keys) e[j] = 0.f;
              sum += e[j];
            }
            // keys c*16 .. c*16+15 are pieces (c & 3) * 2, +1 of this row in k-block c >> 2
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              uint4 u;
              uint32_t* w = (uint32_t*)&u;
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                if (BF16) { __nv_bfloat162 h = __floats2bfloat162_rn(e[q * 8 + 2 * t], e[q * 8 + 2 * t + 1]); w[t] = *(uint32_t*)&h; }
                else { __half2 h = __floats2half2_rn(e[q * 8 + 2 * t], e[q * 8 + 2 * t + 1]); w[t] = *(uint32_t*)&h; }
              }
              sts128(p_row + (uint32_t)(c >> 2) * kAttnBox + (uint32_t)(((((c & 3) << 1) + q) ^ rx) << 4), u);
            }
          }
        }
        tc_fence_before();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tensor cores read P through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(b_p);
        const float inv = last ? __fdividef(1.0f, sum) : 1.f;
        if (!mbar_wait(b_o, n & 1, abort_flag, p.status, 16, p.spin_limit)) { ok = false; break; }
        tc_fence_after();
        if (live) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t r[16];
            tmem_ld16(tmem_o + lane_addr + (uint32_t)(c * 16), r);
            tmem_ld_wait_regs<16>(r);
            if (MULTI) {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                float& acc = o[MULTI ? c * 16 + j : 0];
                acc = fmaf(acc, corr, __uint_as_float(r[j]));
                r[j] = __float_as_uint(acc);
              }
            }
            if (!MULTI || last) {
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                uint4 u;
                uint32_t* w = (uint32_t*)&u;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                  const float a = __uint_as_float(r[q * 8 + 2 * t]) * inv, b = __uint_as_float(r[q * 8 + 2 * t + 1]) * inv;
                  if (BF16) { __nv_bfloat162 h = __floats2bfloat162_rn(a, b); w[t] = *(uint32_t*)&h; }
                  else { __half2 h = __floats2half2_rn(a, b); w[t] = *(uint32_t*)&h; }
                }
                sts128(y_row + (uint32_t)((((c << 1) + q) ^ rx) << 4), u);
              }
            }
          }
        }
        tc_fence_before();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(b_e);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(128u) : "memory");
  }
}

// ------------------------------------------------------------- host: tensor maps ----
int elem_bytes(int dt) { return dt == DT_S8 ? 1 : 2; }
int storage_size_of(int dt) { return dt == DT_S8 || dt == DT_U8 ? 1 : (dt == DT_F16 || dt == DT_BF16 ? 2 : (dt == DT_S64 ? 8 : 4)); }
int pick_kb_bytes(int c_bytes) { return c_bytes > 64 ? 128 : (c_bytes > 32 ? 64 : 32); }
int pick_bn(int k_out) { return k_out <= 64 ? 64 : (k_out <= 128 ? 128 : 256); }

}  // namespace

struct UmmaLaunch {
  CUtensorMap tmA, tmB, tmY, tmR;
  UmmaParams p;
  int grid;
  size_t smem;
};

bool umma_conv_supported(const UmmaConv& c) {
  if (c.in_dt != DT_F16 && c.in_dt != DT_BF16 && c.in_dt != DT_S8) return false;
  int es = elem_bytes(c.in_dt);
  if (((int64_t)c.C * es) % 16 != 0) return false;   // TMA strides and channel coordinates must be 16-byte multiples
  if (c.C * es < 32) return false;
  if (c.K < 1 || c.R < 1 || c.S < 1 || c.R * c.S * (c.w_terms > 1 ? c.w_terms : 1) > 4096) return false;
  if (c.w_terms > 1 && c.w_batches > 0) return false;
  if (c.stride_h < 1 || c.stride_w < 1 || c.stride_h > 8 || c.stride_w > 8) return false;
  if (c.pad_t > 127 || c.pad_l > 127 || c.R > 128 || c.S > 128) return false;  // im2col corners are 8-bit
  if ((int64_t)c.N * c.P * c.Q >= (1ll << 31)) return false;
  if (c.H < 1 || c.W < 1 || c.P < 1 || c.Q < 1) return false;
  if (c.w_batches > 0 && (c.R != 1 || c.S != 1 || c.rows_per_batch <= 0 || c.rows_per_batch % 128 != 0)) return false;
  if (c.w_n_major && (c.w_batches <= 0 || es != 2 || c.K != 64 || c.C % 64 != 0)) return false;
  return true;
}

bool umma_store_perm_ok(const UmmaConv& c, const Epilogue& ep, const void* y) {
  if (c.store_mode != 1 && c.store_mode != 2) return false;
  const int oes = storage_size_of(ep.out_dt);
  if (!(ep.out_dt == DT_F16 || ep.out_dt == DT_BF16 || ep.out_dt == DT_S8) || c.store_D * oes != 128) return false;  // one head = one 128-byte box
  if (ep.res || ep.add_full || (uintptr_t)y % 16 != 0 || getenv("ODLA_B200_DIRECT_EPILOGUE")) return false;
  if (c.store_S <= 0 || c.store_S % 128 != 0 || c.store_NH <= 0 || c.R != 1 || c.S != 1) return false;
  const long long M = (long long)c.N * c.P * c.Q;
  if (c.store_mode == 1) return M % c.store_S == 0 && c.K == c.store_NH * c.store_D;
  return M % ((long long)c.store_S * c.store_NH) == 0 && c.K == c.store_D;
}

constexpr int kLongReduction = 12;   // k-blocks from which a tile's time is its operands' and MMAs', not its epilogue's

// Whether the CTAs of a cluster share each tile's reduction (umma_split_kernel), and over which tiles.  How many share it
// changes the order in which floating-point sums are taken, so that number is decided from the rows of the whole recorded
// batch and not from this launch's share of them: a row's result does not depend on how a batch is cut over GPUs or
// sub-batches.  The tile's shape then follows the launch's own rows.  In clocks, measured on 3x3 layers of one image with 9 to
// 144 k-blocks: one takes 176 of a persistent CTA's walk, 200 of a cluster's, whose barriers and slower way out cost 4500.
// 7 x 7 x 512 -> 512: 22.4 -> 13.7 us.
void choose_split(const UmmaConv& c, int sms, UmmaParams& p) {
  p.splits = 1;
  p.bm = BM;
  if (c.store_mode != 0 || getenv("ODLA_B200_NO_SPLIT")) return;
  auto tiles = [](int64_t n, int64_t t) { return (n + t - 1) / t; };
  const int64_t rows_full = std::max<int64_t>(c.rows_full, p.M_total);
  double best = 176.0 * p.num_kb;
  for (int n = 2; n <= 8 && n <= p.num_kb; n *= 2) {
    // enough SMs for clusters over 64-column tiles of the whole batch
    if (tiles(rows_full, BM) * tiles(c.K, 64) * n > sms) break;
    const double cost = 200.0 * tiles(p.num_kb, n) + 4500.0;
    if (cost < best) { best = cost; p.splits = n; }
  }
  if (p.splits == 1) return;
  // the smallest tiles that still find an SM each: fewer bytes per k-block and CTA
  best = -1;
  for (int bm = BM; bm >= 64; bm /= 2)
    for (int bn = 64; bn >= 16; bn /= 2) {
      if (c.w_batches > 0 && (bm != BM || (c.w_n_major && bn != 64))) continue;   // B boxes of a batched GEMM follow 128-row tiles
      const int64_t ctas = tiles(p.M_total, bm) * tiles(c.K, bn) * p.splits;
      const double cost = (double)tiles(ctas, sms) * std::max((bm + bn) * p.kb_bytes / 80.0, 200.0);
      if (best < 0 || cost < best) { best = cost; p.bm = bm; p.BN = bn; }
    }
  p.bn_load = p.BN;
  p.m_tiles = (int)tiles(p.M_total, p.bm);
  p.n_tiles = (int)tiles(c.K, p.BN);
  p.total_tiles = p.m_tiles * p.n_tiles;
}

// The tile of a persistent launch whose p.BN is at least 128: how many columns, and whether CTA pairs (tcgen05 cta_group::2)
// share it.  A pair computes 256 rows x BN columns and each CTA loads only half of the filter tile.  That pays where
// operand traffic into shared memory is the limit -- two-byte operands and a long reduction (measured: 12 or more k-blocks,
// e.g. a 768-deep transformer projection; at 8 a ResNet layer loses) -- and costs where the epilogue is, because the pair's
// CTAs then wait for each other's accumulators.  Needs an even grid.
// Long reductions also choose their columns: a launch takes whole rounds of tiles, and 96 tiles of 256 columns on 74 pairs
// are two rounds as long as 148 would be.  192 columns make them 128 shorter ones.  In clocks, from the walk's own
// timing: a k-block of 256, 192, 128 columns takes 560, 430, 390 on pairs and 600, 470, 415 on single CTAs, a tile 1200 to
// start, the last tile's epilogue 20 a column and a pair's setting up 400.  3x3 512 -> 1024 at 13 x 13 x 16: 43 -> 35 us, a
// 3072 -> 768 projection of 8192 rows with a residual: 49 -> 45 us.  (192 columns are one and a half boxes of one-byte results: not there.)  The clocks are those of
// k-blocks of 128 bytes, measured on the layers named here; shorter k-blocks are given the same, which only scales both sides.
void choose_tile(const UmmaConv& c, const Epilogue& ep, int sms, UmmaParams& p) {
  p.pair = 0;
  p.bn_load = p.BN;
  if (p.BN < 128 && !getenv("ODLA_B200_PAIR_MIN_BN")) return;
  // (the thresholds can be moved through the environment, which the tests use to run every shape on pairs)
  const int pair_min_bn = getenv("ODLA_B200_PAIR_MIN_BN") ? atoi(getenv("ODLA_B200_PAIR_MIN_BN")) : 128;
  const int pair_min_kb = getenv("ODLA_B200_PAIR_MIN_KB") ? atoi(getenv("ODLA_B200_PAIR_MIN_KB")) : kLongReduction;
  const bool pairs = (c.in_dt != DT_S8 || getenv("ODLA_B200_PAIR_S8")) && p.num_kb >= pair_min_kb && sms >= 2 && c.w_batches == 0 &&
                     (c.store_mode == 0 || p.M_total % (2 * BM) == 0);
  auto tiles = [](int64_t n, int64_t t) { return (n + t - 1) / t; };
  const bool choose = p.num_kb >= kLongReduction && p.BN >= 128 && c.w_batches == 0;
  const int out_esz = storage_size_of(ep.out_dt);
  double best = -1;
  int best_bn = p.BN, best_pair = 0;
  for (int bn = choose ? pick_bn(c.K) : p.BN; bn >= (choose ? 128 : p.BN); bn -= 64) {
    if (bn == 192 && (out_esz != 2 || p.kb_bytes != 128)) continue;
    for (int pair = pairs && bn >= pair_min_bn ? 1 : 0; pair >= 0; --pair) {
      const double kb = bn > 192 ? (pair ? 560 : 600) : (bn > 128 ? (pair ? 430 : 470) : (pair ? 390 : 415));
      const int64_t rounds = tiles(tiles(p.M_total, BM << pair) * tiles(c.K, bn), pair ? sms / 2 : sms);
      const double cost = (double)rounds * (p.num_kb * kb + 1200.0) + 20.0 * bn + 400.0 * pair;
      if (best < 0 || cost < best) { best = cost; best_bn = bn; best_pair = pair; }
      if (pair && !choose) break;   // (only tests come here: short reductions on pairs)
    }
  }
  p.BN = best_bn;
  p.pair = best_pair;
  p.bn_load = p.BN >> p.pair;
  p.m_tiles = (int)tiles(p.M_total, BM << p.pair);
  p.n_tiles = (int)tiles(c.K, p.BN);
  p.total_tiles = p.m_tiles * p.n_tiles;
}

UmmaLaunch* umma_conv_prepare(const UmmaConv& c, const void* x, const void* w, void* y, const Epilogue& ep, int* status, int sms) {
  if (!umma_conv_supported(c) || !load_driver_entry_points()) return nullptr;
  auto* L = new UmmaLaunch();
  UmmaParams& p = L->p;
  const int es = elem_bytes(c.in_dt);
  p.M_total = c.N * c.P * c.Q; p.K_out = c.K; p.C = c.C; p.R = c.R; p.S = c.S; p.P = c.P; p.Q = c.Q;
  p.stride_h = c.stride_h; p.stride_w = c.stride_w; p.pad_t = c.pad_t; p.pad_l = c.pad_l;
  p.im2col = !(c.R == 1 && c.S == 1 && c.stride_h == 1 && c.stride_w == 1 && c.pad_t == 0 && c.pad_l == 0 && c.P == c.H && c.Q == c.W);
  p.kb_bytes = pick_kb_bytes(c.C * es);
  p.kbe = p.kb_bytes / es;
  p.chunks_per_tap = (c.C + p.kbe - 1) / p.kbe;
  const int terms = c.w_terms > 1 ? c.w_terms : 1;
  p.num_kb = c.R * c.S * terms * p.chunks_per_tap;
  p.BN = pick_bn(c.K);
  p.m_tiles = (p.M_total + BM - 1) / BM;
  // Few rows (small batches, the classifier): narrower tiles put more SMs to work on the same reduction; a tile's time
  // is dominated by its k-blocks, not by its width.
  // (a staged tile leaves in whole 128-byte boxes, so one-byte outputs keep at least 128 columns)
  if (!getenv("ODLA_B200_NO_BN_SHRINK")) {
    const int min_bn = storage_size_of(ep.out_dt) == 1 ? 128 : 64;
    while (p.BN > min_bn && 2 * p.m_tiles * ((c.K + p.BN - 1) / p.BN) <= sms) p.BN /= 2;
  }
  p.n_tiles = (c.K + p.BN - 1) / p.BN;
  p.total_tiles = p.m_tiles * p.n_tiles;
  choose_split(c, sms, p);
  if (p.splits == 1) choose_tile(c, ep, sms, p);
  // Several k-blocks share one pipeline stage (one mbarrier round trip) when they are small: up to
  // 48 KB per stage, balanced over the tile's k-blocks.
  const int box_bytes = (p.bm + p.bn_load) * p.kb_bytes;
  int bps_max = (48 * 1024) / box_bytes;
  if (bps_max < 1) bps_max = 1;
  if (bps_max > 8) bps_max = 8;
  const int share_kb = (p.num_kb + p.splits - 1) / p.splits;   // k-blocks one CTA walks
  const int iters = (share_kb + bps_max - 1) / bps_max;
  p.bps = (share_kb + iters - 1) / iters;
  p.num_it = (p.num_kb + p.bps - 1) / p.bps;
  const int stage_bytes = p.bps * box_bytes;
  // Staged epilogue: the output tile goes through shared memory (128-byte-swizzled boxes of 128 rows)
  // and leaves with TMA stores; the residual tile arrives the same way when its element size equals
  // the output's.  Needs 16-byte-multiple rows in global memory and a 1/2-byte output type.
  p.out_esz = storage_size_of(ep.out_dt);
  // The residual of a staged launch always comes through the staging box, so it must have the output's type.
  const bool res_ok = !ep.res || (ep.res_dt == ep.out_dt && (uintptr_t)ep.res % 16 == 0);
  const int64_t y_cols = c.y_pitch > 0 ? c.y_pitch : c.K;  // row pitch of y in elements
  p.y_ld = (int)y_cols;
  p.staged = p.splits == 1 && (ep.out_dt == DT_F16 || ep.out_dt == DT_BF16 || ep.out_dt == DT_S8) && (y_cols * p.out_esz) % 16 == 0 && !ep.add_full && res_ok &&
             (c.y_pitch == 0 || (c.y_pitch >= c.K && !ep.res && c.store_mode == 0)) &&
             ((uintptr_t)y % 16 == 0) && !getenv("ODLA_B200_DIRECT_EPILOGUE");
  p.stage_boxes = p.staged ? (p.BN * p.out_esz + 127) / 128 : 0;
  p.res_tma = p.staged && ep.res;
  const bool plain_act = !ep.act_first && (ep.act == ACT_NONE || ep.act == ACT_RELU) && (ep.out_dt != DT_S8 || (ep.out_multiply && ep.out_inv > 0.f));
  // what the straight-line epilogue assumes (see chunk_fast); everything else takes the general staged form
  const bool fast_ok = plain_act && c.K % 16 == 0 && ep.alpha == 1.f && ((ep.add1 != nullptr) != (ep.add2 != nullptr)) &&
                       ((ep.mul != nullptr) == (c.in_dt == DT_S8)) && (ep.out_dt != DT_S8 || c.in_dt == DT_S8) && !getenv("ODLA_B200_GENERAL_EPILOGUE");
  // the Darknet form (see chunk_leaky): LeakyReLU with a slope in [0, 1] straight after the per-channel addend, a
  // residual (if any) after the activation, fp32 accumulators, two-byte outputs
  // (the same kernel carries the GELU form of a transformer's first feed-forward layer: no residual there)
  const bool act_form = (ep.act == ACT_LEAKY && ep.act_a >= 0.f && ep.act_a <= 1.f && (!ep.res || ep.act_first)) ||
                        (ep.act == ACT_GELU_ERF && !ep.res && !getenv("ODLA_B200_EXACT_ERF"));
  const bool leaky_ok = act_form && c.K % 16 == 0 && ep.alpha == 1.f &&
                        ((ep.add1 != nullptr) != (ep.add2 != nullptr)) && !ep.mul && c.in_dt != DT_S8 && (ep.out_dt == DT_F16 || ep.out_dt == DT_BF16) &&
                        !getenv("ODLA_B200_GENERAL_EPILOGUE");
  // ... and its int8 form: int8 operands, multiplier + addend, GELU, requantised int8 output
  const bool gelu_s8_ok = ep.act == ACT_GELU_ERF && !ep.res && c.in_dt == DT_S8 && ep.out_dt == DT_S8 && ep.mul && ep.out_multiply && ep.out_inv > 0.f &&
                          c.K % 16 == 0 && ep.alpha == 1.f && ((ep.add1 != nullptr) != (ep.add2 != nullptr)) &&
                          !getenv("ODLA_B200_EXACT_ERF") && !getenv("ODLA_B200_GENERAL_EPILOGUE");
  p.epi_mode = !p.staged ? 0 : (fast_ok ? 1 : ((leaky_ok || gelu_s8_ok) ? 3 : 2));
  p.fast_variant = (c.in_dt == DT_S8 ? (ep.acc_small ? 2 : 1) : 0) * 2 + (ep.res ? 1 : 0);
  // Shared memory: pipeline stages first (up to 4, or what one tile needs), then as many staging
  // boxes as fit (at least one tile's worth, at most 8) so residual loads run ahead of the epilogue
  // and stores drain behind it; what is left goes back to the pipeline.
  // A memory-bound layer needs enough bytes in flight per SM to cover the latency of HBM (about 64 KB at 6.5 TB/s
  // over 148 SMs): boxes armed ahead carry the residual loads, stages armed ahead the operand loads, so neither is
  // limited to what one tile needs.
  const int budget = 224 * 1024;
  int want_stages = p.num_it + 1 < 4 ? p.num_it + 1 : 4;
  if (want_stages < 2) want_stages = 2;
  p.ring_boxes = 0;
  if (p.staged) {
    int ring_want = ep.res ? 4 * p.stage_boxes : 2 * p.stage_boxes;
    if (ring_want < 4) ring_want = 4;
    if (getenv("ODLA_B200_RING")) ring_want = atoi(getenv("ODLA_B200_RING"));
    p.ring_boxes = (budget - want_stages * stage_bytes) / 16384;
    if (p.ring_boxes > kMaxRing) p.ring_boxes = kMaxRing;
    if (p.ring_boxes > ring_want) p.ring_boxes = ring_want;
    int ring_min = p.stage_boxes;
    // Long reductions are bound by how many operand bytes are on their way: a stage is 1400 clocks from its request to its
    // MMAs and 700 more to its next request, in which the tensor cores take in 130 KB of a 256 x 256 pair tile's operands.
    // Their epilogues have time, so two boxes go round (one being written, one being stored), a tile's worth where a residual
    // is fetched ahead and four stages remain.  3x3 256 -> 512 at 26 x 26 x 16: 40.7 -> 36.7 us, 1024 -> 256 at 14 x 14 x 256: 40.8 -> 36.9 us, a
    // 3072-deep projection of 8192 rows: 48.7 -> 45.0 us.
    if (p.num_kb >= kLongReduction) {
      ring_min = ep.res && budget - p.stage_boxes * 16384 >= 4 * stage_bytes ? p.stage_boxes : 2;
      if (p.ring_boxes > ring_min) p.ring_boxes = ring_min;
    }
    if (p.ring_boxes < ring_min) p.ring_boxes = ring_min;
    if (p.ring_boxes < 2) p.ring_boxes = 2;  // the store of box i frees box i-1
  }
  {
    // 16 epilogue warps = 4 groups; a group owns BN/64 consecutive 16-column chunks, a box holds 128/out_esz/16
    const int per_group = std::max(p.BN / 64, 1), per_box = 128 / p.out_esz / 16;
    const int groups_per_box = per_box / per_group < 4 ? per_box / per_group : 4;
    p.box_arrivals = 4 * (groups_per_box < 1 ? 1 : groups_per_box);
    // Contiguous runs let the groups work on different boxes at once; finishing box after box gets the first store out sooner,
    // which only still pays for the long arithmetic of MODE 3 (LeakyReLU, GELU) with a residual or few tiles: a feed-forward layer of
    // 8192 x 768 -> 3072 in int8 takes 31.6 us box after box and 32.6 in runs, its Q, K and V product 20.6 and 18.3; ResNet-50 of 45
    // images 819 and 805, of 256 in int8 3330 and 3290.
    p.epi_interleave = p.epi_mode == 3 && (ep.res != nullptr || (p.total_tiles << p.pair) < 16 * sms);
    if (getenv("ODLA_B200_EPI_INTERLEAVE")) p.epi_interleave = atoi(getenv("ODLA_B200_EPI_INTERLEAVE"));
    // In runs a group waits only for its own boxes, by the parity of the box's phase, so the use of the same box one
    // turn of the ring earlier has to have been full by then.  That use lies in the tile before, at or below the group's
    // own box there (ring of at least a tile's boxes; every tile with all its boxes; groups whole to a box, which 192 columns are
    // not) -- and boxes without a residual fill in order.  Residuals land in any order: there it has to be the group's own box
    // (ring of exactly a tile) or lie two tiles back, which every group has left before the accumulator could be reused.
    const bool whole_tiles = p.K_out > (p.n_tiles - 1) * p.BN + (p.stage_boxes - 1) * (128 / p.out_esz);
    const bool in_order = !ep.res || p.ring_boxes == p.stage_boxes || p.ring_boxes >= 2 * p.stage_boxes;
    if (p.ring_boxes < p.stage_boxes || p.BN == 192 || !whole_tiles || !in_order) p.epi_interleave = 1;
    if (p.epi_interleave) p.box_arrivals = 16;
  }
  p.stages = (budget - p.ring_boxes * 16384) / stage_bytes;
  if (p.stages > 8) p.stages = 8;
  {
    // stages beyond one tile's worth let the producer run into the following tiles (the stage ring spans tiles)
    int cap = p.num_it + 1 > 6 ? p.num_it + 1 : 6;
    if (getenv("ODLA_B200_STAGE_CAP")) cap = atoi(getenv("ODLA_B200_STAGE_CAP")) + p.num_it;
    if (p.stages > cap) p.stages = cap;
  }
  if (p.stages < 2) p.stages = 2;
  p.acc_int = c.in_dt == DT_S8;
  p.store_mode = c.store_mode; p.store_S = c.store_S; p.store_NH = c.store_NH;
  if (p.store_mode && (!p.staged || !umma_store_perm_ok(c, ep, y))) { delete L; return nullptr; }
  if (c.y_pitch > 0 && !p.staged && (p.splits == 1 || ep.res)) { delete L; return nullptr; }  // the direct epilogue writes rows of K elements
  p.rows_per_batch = c.w_batches > 0 ? c.rows_per_batch : 0;
  p.tmem_cols = p.splits > 1 ? std::max(p.BN, 32) : (p.BN > 128 ? 512 : 2 * p.BN);  // 32 to 512: powers of two
  const uint32_t fmt = c.in_dt == DT_BF16 ? 1u : (c.in_dt == DT_S8 ? 1u : 0u);      // bf16 / signed 8-bit / f16
  const uint32_t cfmt = p.acc_int ? 2u : 1u;                                        // s32 / f32 accumulators
  p.idesc = (cfmt << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.BN >> 3) << 17) | ((uint32_t)((p.bm << p.pair) >> 4) << 24);
  // B stored [k][n]: the instruction reads it MN-major (descriptor bit 16).  A box is then 64 k-rows of 128 bytes: the
  // 8-row group pitch (SBO) is the same 1024 bytes, and 32 bytes of K are 16 rows = 2048 bytes further on.
  p.b_n_major = c.w_n_major ? 1 : 0;
  p.b_kstep = p.b_n_major ? (16 * 128) >> 4 : 2;
  if (p.b_n_major) {
    if (p.BN != 64 || p.kb_bytes != 128 || p.pair) { delete L; return nullptr; }
    p.idesc |= 1u << 16;
  }
  const uint32_t layout = p.kb_bytes == 128 ? 2u : (p.kb_bytes == 64 ? 4u : 6u);    // swizzle mode of the operand tiles
  const uint32_t sbo = (uint32_t)(8 * p.kb_bytes) >> 4;                             // 8-row group pitch, 16-byte units
  p.desc_hi = sbo | (1u << 14) | (layout << 29);                                    // bits 32-45 SBO, 46-47 version 1, 61-63 layout
  p.y = y; p.status = status; p.ep = ep;
  p.spin_limit = kSpinLimit;
  p.test_skip_stage = 0;
  // Test hooks for the time-out path (tests/test_conv_umma_gpu.py): a short limit and one deliberately unarmed stage.
  if (const char* e = getenv("ODLA_B200_TEST_SPIN_LIMIT")) { const long v = atol(e); if (v >= 64 && v <= (1l << 18)) p.spin_limit = (uint32_t)v; }
  if (getenv("ODLA_B200_TEST_SKIP_STAGE") && !p.pair) p.test_skip_stage = 1;
  p.b_constant = c.w_constant;
  L->grid = p.pair ? (2 * p.total_tiles < (sms & ~1) ? 2 * p.total_tiles : (sms & ~1)) : (p.total_tiles < sms ? p.total_tiles : sms);
  L->smem = (size_t)p.stages * stage_bytes + (size_t)p.ring_boxes * 16384 + 1024 /*alignment slack*/ + 1024 /*barriers*/;
  if (p.splits > 1) {
    p.stages = std::max(1, std::min({200 * 1024 / stage_bytes, 8, (share_kb + p.bps - 1) / p.bps}));
    p.split_data_bytes = (std::max(p.stages * stage_bytes, p.bm * p.BN * 4) + 1023) / 1024 * 1024;
    p.split_plain = !p.acc_int && c.K % 4 == 0 && !ep.mul && ep.alpha == 1.f && ((ep.add1 != nullptr) != (ep.add2 != nullptr)) && !ep.add_full &&
                    (ep.act == ACT_NONE || (ep.act == ACT_RELU && !ep.act_first) || ep.act == ACT_LEAKY) && (ep.out_dt == DT_F16 || ep.out_dt == DT_BF16) &&
                    (!ep.res || ep.res_dt == ep.out_dt);
    L->grid = p.total_tiles * p.splits;
    L->smem = (size_t)p.split_data_bytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
  }
  if (L->smem > 227 * 1024) { delete L; return nullptr; }

  const CUtensorMapDataType dt = c.in_dt == DT_S8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : (c.in_dt == DT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
  const CUtensorMapSwizzle sw = p.kb_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (p.kb_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
  CUresult r;
  if (p.im2col) {
    cuuint64_t dims[4] = {(cuuint64_t)c.C, (cuuint64_t)c.W, (cuuint64_t)c.H, (cuuint64_t)c.N};
    cuuint64_t strides[3] = {(cuuint64_t)c.C * es, (cuuint64_t)c.W * c.C * es, (cuuint64_t)c.H * c.W * c.C * es};
    if (c.x_w_stride) { strides[0] = (cuuint64_t)c.x_w_stride; strides[1] = (cuuint64_t)c.x_h_stride; strides[2] = (cuuint64_t)c.x_n_stride; }
    // The box of filter-window origins: from -pad to the last origin that still yields an output.
    int lower[2] = {-c.pad_l, -c.pad_t};
    // The last origin is (Q-1)*stride - pad; the upper corner is that position relative to W-1 (H-1).
    int upper[2] = {(c.Q - 1) * c.stride_w - c.pad_l - (c.W - 1), (c.P - 1) * c.stride_h - c.pad_t - (c.H - 1)};
    if (upper[0] < -128 || upper[0] > 127 || upper[1] < -128 || upper[1] > 127) { delete L; return nullptr; }
    cuuint32_t estr[4] = {1, (cuuint32_t)c.stride_w, (cuuint32_t)c.stride_h, 1};
    r = g_encode_im2col(&L->tmA, dt, 4, (void*)x, dims, strides, lower, upper, (cuuint32_t)p.kbe, (cuuint32_t)p.bm, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS) {
      // Drivers up to 13.1 encode small im2col tensors (< 128 KiB) with a flag that makes the load
      // misbehave; CUTLASS clears bit 21 of the second descriptor word in that case
      // (cute/atom/copy_traits_sm90_im2col.hpp), and so does this library.
      int drv = 0;
      cudaDriverGetVersion(&drv);
      const int64_t span = c.x_w_stride ? (int64_t)c.N * c.x_n_stride : (int64_t)c.N * c.H * c.W * c.C * es;
      if (drv <= 13010 && span < 131072) ((uint64_t*)&L->tmA)[1] &= ~(1ull << 21);
    }
  } else {
    cuuint64_t dims[2] = {(cuuint64_t)c.C, (cuuint64_t)p.M_total};
    cuuint64_t strides[1] = {(cuuint64_t)c.C * es};
    cuuint32_t box[2] = {(cuuint32_t)p.kbe, (cuuint32_t)p.bm};
    cuuint32_t estr[2] = {1, 1};
    r = g_encode_tiled(&L->tmA, dt, 2, (void*)x, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (r != CUDA_SUCCESS) {
    if (!c.x_w_stride) fprintf(stderr, "[odla_b200] tensor map (A) encode failed: %d\n", (int)r);  // overlapping strides are an optional fast path
    delete L;
    return nullptr;
  }
  {
    cuuint64_t dims[3] = {(cuuint64_t)c.C, (cuuint64_t)(c.R * c.S * terms), (cuuint64_t)c.K};
    cuuint64_t strides[2] = {(cuuint64_t)c.C * es, (cuuint64_t)c.R * c.S * terms * c.C * es};
    cuuint32_t box[3] = {(cuuint32_t)p.kbe, 1, (cuuint32_t)p.bn_load};
    if (c.w_batches > 0) {  // [batches][K][C]: the box spans BN rows of one matrix
      dims[1] = (cuuint64_t)c.K; dims[2] = (cuuint64_t)c.w_batches;
      strides[1] = (cuuint64_t)c.K * c.C * es;
      box[1] = (cuuint32_t)p.BN; box[2] = 1;
    }
    if (c.w_n_major) {      // [batches][C][K]: the box spans kbe rows (of the reduction) by all 64 columns
      dims[0] = (cuuint64_t)c.K; dims[1] = (cuuint64_t)c.C;
      strides[0] = (cuuint64_t)c.K * es;
      box[0] = (cuuint32_t)c.K; box[1] = (cuuint32_t)p.kbe;
    }
    cuuint32_t estr[3] = {1, 1, 1};
    r = g_encode_tiled(&L->tmB, dt, 3, (void*)w, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (r != CUDA_SUCCESS) { fprintf(stderr, "[odla_b200] tensor map (B) encode failed: %d\n", (int)r); delete L; return nullptr; }
  if (p.staged) {
    const CUtensorMapDataType odt = p.out_esz == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16;
    cuuint64_t dims[2] = {(cuuint64_t)y_cols, (cuuint64_t)p.M_total};
    cuuint64_t strides[1] = {(cuuint64_t)y_cols * p.out_esz};
    cuuint32_t box[2] = {(cuuint32_t)(128 / p.out_esz), (cuuint32_t)BM};
    cuuint32_t estr[2] = {1, 1};
    if (p.store_mode) {
      const cuuint64_t D = (cuuint64_t)c.store_D, S = (cuuint64_t)c.store_S, NH = (cuuint64_t)c.store_NH;
      const cuuint64_t Bn = (cuuint64_t)p.M_total / (S * (p.store_mode == 1 ? 1 : NH));
      cuuint64_t d4[4] = {D, p.store_mode == 1 ? S : NH, p.store_mode == 1 ? NH : S, Bn};
      cuuint64_t s4[3] = {D * p.out_esz, d4[1] * D * p.out_esz, d4[1] * d4[2] * D * p.out_esz};
      cuuint32_t b4[4] = {(cuuint32_t)D, p.store_mode == 1 ? (cuuint32_t)BM : 1u, p.store_mode == 1 ? 1u : (cuuint32_t)BM, 1};
      cuuint32_t e4[4] = {1, 1, 1, 1};
      r = g_encode_tiled(&L->tmY, odt, 4, y, d4, s4, b4, e4, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else
    r = g_encode_tiled(&L->tmY, odt, 2, y, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS && p.res_tma)
      r = g_encode_tiled(&L->tmR, odt, 2, (void*)ep.res, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { fprintf(stderr, "[odla_b200] tensor map (output/residual) encode failed: %d\n", (int)r); delete L; return nullptr; }
  }
  if (!p.staged) L->tmY = L->tmA;
  if (!p.res_tma) L->tmR = L->tmA;
  static bool attr_set[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 16 && !attr_set[dev]) {
#define B2_SMEM(O, M)                                                                                                              \
  (cudaFuncSetAttribute(umma_conv_kernel<O, M, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess && \
   cudaFuncSetAttribute(umma_conv_kernel<O, M, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess)
    bool ok = B2_SMEM(DT_F16, 1) && B2_SMEM(DT_BF16, 1) && B2_SMEM(DT_S8, 1) && B2_SMEM(DT_F16, 2) && B2_SMEM(DT_BF16, 2) && B2_SMEM(DT_S8, 2) && B2_SMEM(DT_F16, 3) && B2_SMEM(DT_BF16, 3) && B2_SMEM(DT_S8, 3) && B2_SMEM(-1, 0);
#undef B2_SMEM
    ok = ok && cudaFuncSetAttribute(umma_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess;
    if (!ok) { cudaGetLastError(); delete L; return nullptr; }
    attr_set[dev] = true;
  }
  return L;
}

int umma_conv_run(UmmaLaunch* L, cudaStream_t stream) {
  if (!L) return -1;
  if (L->p.total_tiles <= 0) return 0;
  const UmmaParams& p = L->p;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)L->grid);
  cfg.blockDim = dim3(p.splits > 1 ? kSplitThreads : p.staged ? EpiCfg<true>::kThreads : EpiCfg<false>::kThreads);
  cfg.dynamicSmemBytes = L->smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  static const bool pdl = !getenv("ODLA_B200_NO_PDL");
  int na = 0;
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (p.pair || p.splits > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.pair ? 2 : (unsigned)p.splits;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t le;
#define B2_LAUNCH(O, M)                                                                                   \
  le = p.pair ? cudaLaunchKernelEx(&cfg, umma_conv_kernel<O, M, true>, L->tmA, L->tmB, L->tmY, L->tmR, p) \
              : cudaLaunchKernelEx(&cfg, umma_conv_kernel<O, M, false>, L->tmA, L->tmB, L->tmY, L->tmR, p)
  if (p.splits > 1) le = cudaLaunchKernelEx(&cfg, umma_split_kernel, L->tmA, L->tmB, p);
  else if (p.epi_mode == 0) B2_LAUNCH(-1, 0);
  else if (p.epi_mode == 1) { if (p.ep.out_dt == DT_F16) B2_LAUNCH(DT_F16, 1); else if (p.ep.out_dt == DT_BF16) B2_LAUNCH(DT_BF16, 1); else B2_LAUNCH(DT_S8, 1); }
  else if (p.epi_mode == 3) { if (p.ep.out_dt == DT_F16) B2_LAUNCH(DT_F16, 3); else if (p.ep.out_dt == DT_BF16) B2_LAUNCH(DT_BF16, 3); else B2_LAUNCH(DT_S8, 3); }
  else { if (p.ep.out_dt == DT_F16) B2_LAUNCH(DT_F16, 2); else if (p.ep.out_dt == DT_BF16) B2_LAUNCH(DT_BF16, 2); else B2_LAUNCH(DT_S8, 2); }
#undef B2_LAUNCH
  if (le != cudaSuccess) { fprintf(stderr, "[odla_b200] umma_conv launch failed: %s\n", cudaGetErrorString(le)); cudaGetLastError(); return -2; }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { fprintf(stderr, "[odla_b200] umma_conv launch failed: %s\n", cudaGetErrorString(e)); return -2; }
  return 0;
}
void umma_conv_destroy(UmmaLaunch* L) { delete L; }

// ---- fused attention: host side ----
struct AttnLaunch {
  CUtensorMap tmQ, tmK, tmV, tmY;
  AttnParams p;
  int grid;
  size_t smem;
  bool bf16, multi;
};
bool attn_supported(int dt, int64_t S, int64_t D) { return (dt == DT_F16 || dt == DT_BF16) && S >= 1 && S <= 65536 && D == kAttnD; }
AttnLaunch* attn_prepare(const AttnShape& a, const void* q, const void* k, const void* v, void* y, int* status, int sms) {
  const int64_t S = a.positions, q_tiles = (S + kAttnS - 1) / kAttnS, batch = a.batch, heads = a.heads, ld = a.qkv_row_elems;
  if (!attn_supported(a.dt, S, kAttnD) || batch * heads <= 0 || batch * heads * q_tiles >= (1ll << 31) || batch * S >= (1ll << 31) || !load_driver_entry_points()) return nullptr;
  if ((uintptr_t)q % 16 || (uintptr_t)k % 16 || (uintptr_t)v % 16 || (uintptr_t)y % 16 || ld % 8) return nullptr;
  auto* L = new AttnLaunch();
  AttnParams& p = L->p;
  p.NH = (int)heads; p.S = (int)S; p.q_tiles = (int)q_tiles; p.k_blocks = (int)q_tiles;
  p.tiles = (int)(batch * heads * q_tiles);
  p.qkv_rows = ld > 0 ? 1 : 0; p.merge = a.merge_heads ? 1 : 0;
  p.scale_log2e = a.scale * 1.4426950408889634f;
  L->bf16 = a.dt == DT_BF16; L->multi = q_tiles > 1;
  p.last_keys = (int)(S - (q_tiles - 1) * kAttnS);
  p.last_ksteps = (p.last_keys + 15) / 16;
  const uint32_t fmt = a.dt == DT_BF16 ? 1u : 0u, common = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(128 >> 4) << 24);
  p.idesc_s = common | ((uint32_t)(kAttnS >> 3) << 17);
  p.idesc_s_last = common | ((uint32_t)(2 * p.last_ksteps) << 17);                 // as many keys as are left, in sixteens
  p.idesc_o = common | (1u << 16) | ((uint32_t)(kAttnD >> 3) << 17);               // B (= V) is MN-major
  p.desc_hi = ((uint32_t)(8 * 128) >> 4) | (1u << 14) | (2u << 29);
  p.spin_limit = kSpinLimit;
  p.status = status;
  const int per_sm = L->multi ? 3 : 4;
  L->grid = p.tiles < per_sm * sms ? p.tiles : per_sm * sms;
  L->smem = (L->multi ? 4 : 3) * (size_t)kAttnBox + 1024 /*alignment slack*/ + 256 /*barriers*/;
  const CUtensorMapDataType tdt = a.dt == DT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  // heads inside rows: (channel, head, position, batch); heads outside: (channel, position, head, batch)
  auto encode = [&](CUtensorMap* m, const void* base, bool rows, int64_t row_elems, CUtensorMapL2promotion l2) {
    const cuuint64_t D = (cuuint64_t)kAttnD, hs = (cuuint64_t)heads, ps = (cuuint64_t)S, bs = (cuuint64_t)batch, re = (cuuint64_t)row_elems * 2;
    cuuint64_t dr[4] = {D, hs, ps, bs}, sr[3] = {D * 2, re, ps * re}, dh[4] = {D, ps, hs, bs}, sh[3] = {D * 2, ps * D * 2, hs * ps * D * 2};
    cuuint32_t br[4] = {(cuuint32_t)kAttnD, 1, (cuuint32_t)kAttnS, 1}, bh[4] = {(cuuint32_t)kAttnD, (cuuint32_t)kAttnS, 1, 1}, e[4] = {1, 1, 1, 1};
    return g_encode_tiled(m, tdt, 4, (void*)base, rows ? dr : dh, rows ? sr : sh, rows ? br : bh, e, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, l2,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = CUDA_SUCCESS;
  const void* src[3] = {q, k, v};
  CUtensorMap* maps[3] = {&L->tmQ, &L->tmK, &L->tmV};
  for (int i = 0; i < 3 && r == CUDA_SUCCESS; ++i) r = encode(maps[i], src[i], ld > 0, ld, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
  if (r == CUDA_SUCCESS) r = encode(&L->tmY, y, a.merge_heads, heads * kAttnD, CU_TENSOR_MAP_L2_PROMOTION_NONE);
  if (r != CUDA_SUCCESS) { fprintf(stderr, "[odla_b200] tensor map (attention) encode failed: %d\n", (int)r); delete L; return nullptr; }
  auto* fn = L->multi ? (L->bf16 ? attn_kernel<true, true> : attn_kernel<false, true>) : (L->bf16 ? attn_kernel<true, false> : attn_kernel<false, false>);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L->smem) != cudaSuccess) { cudaGetLastError(); delete L; return nullptr; }
  return L;
}
int attn_run(AttnLaunch* L, cudaStream_t stream) {
  if (!L) return -1;
  if (L->p.tiles <= 0) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)L->grid);
  cfg.blockDim = dim3(kAttnThreads);
  cfg.dynamicSmemBytes = L->smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  static const bool pdl = !getenv("ODLA_B200_NO_PDL");
  int na = 0;
  if (pdl) { attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[na].val.programmaticStreamSerializationAllowed = 1; ++na; }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  auto* fn = L->multi ? (L->bf16 ? attn_kernel<true, true> : attn_kernel<false, true>) : (L->bf16 ? attn_kernel<true, false> : attn_kernel<false, false>);
  const cudaError_t le = cudaLaunchKernelEx(&cfg, fn, L->tmQ, L->tmK, L->tmV, L->tmY, L->p);
  if (le != cudaSuccess) { fprintf(stderr, "[odla_b200] attention launch failed: %s\n", cudaGetErrorString(le)); cudaGetLastError(); return -2; }
  return 0;
}
void attn_destroy(AttnLaunch* L) { delete L; }

}  // namespace b200
