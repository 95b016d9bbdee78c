// fp32 convolutions (NHWC, one group) and products with constant weights on the tensor cores.
//
//   D[M, N] = A[M, R*S*C] * W[N, R*S*C]^T      M = pixels (rows of a product), A gathered by im2col-mode TMA as in kernels_umma.cu
//
// The tensor cores have no fp32 operand type, but an fp32 value is exactly the sum of three bf16 values (8 + 8 + 8 bits of
// mantissa, the same exponent range): a = a1 + a2 + a3, each the leading bits of what the ones before leave.  The product a * w is then
// a1 w1 + (a1 w2 + a2 w1) + (a1 w3 + a2 w2 + a3 w1), six bf16 products that are exact in fp32; what the other three add up to is at most
// 1.5 * 2^-24 of a * w, 2^-26.5 rms (a rounding to fp32: 2^-24, 2^-25.3).  Six of them at
// 4096 a clock and SM are 683 fp32 products against the FMA pipe's 128, of which the tiles of kernels_f32.cu reach a third.
// CUDA cores -> here: ResNet-50 of 8 images 2759 -> 1007 us, YOLOv3 of one 416 x 416 picture 3130 -> 1595, BERT of 2 x 128 2476 -> 1683, each call
// waited for; a 3x3 layer of 8 x 28 x 28 x 128 -> 128, its launch bracketed, 64 -> 27, of 2 x 52 x 52 x 128 -> 256 101 -> 35.  What bounds it: half a stage of 64 columns takes some 800 clocks
// where its products take 400 (the splitting warps' chain of load, split, store and signal), one of 128 columns 1100 where they take
// 770; short reductions their first loads and the finishing of the tile.
//
// Precision.  The tensor cores add into their accumulators without rounding to nearest, so that a long reduction kept there
// drifts.  The leading products a1 w1 of 64 values therefore go to an accumulator of their own, two of which take turns, and are
// added up in registers with ordinary fp32 additions while the other fills; the five small products, a 2^-8th of the result, share
// one accumulator for the whole tile, where the drift is a 2^-8th as well.  Against float64 (rms error over rms result, products of 64 to
// 4608 values) N(0, 1) operands have 7e-8 to 1.4e-7, on the CUDA cores 1.1e-7 to 3.1e-7; after a ReLU 5e-8 to 1.3e-7 and 8e-8 to 2.3e-7.  Only where
// both operands have one sign throughout is the drift the larger part: 8.5e-8 to 1.1e-7 and 5.8e-8 to 9.0e-8.
// Values for which the split does not hold -- an infinity among the operands, a sum that overflows on the way, results so small that bits
// of A below the smallest bf16 count -- show up in the sum (not finite, or not zero and below p.least) and such results are computed
// again: from the infinities' signs where there are any, else as an fp32 FMA chain (replay) from the operands, A as it lies, W as the sum
// of its three parts, which it is exactly.  A NaN in the row needs nothing: its sums are NaN.  An FMA chain takes a hundred times as long as
// the tensor cores, so that it has to be rare: hence p.least as low as the layer's weights allow.  ResNet-50 of 8 images, waited for after
// each call: 1007 us, with an image of NaN 1018, of infinities 1111, of 1e-40 1299, all of them of 1e-40 2661.
//
// One CTA per SM walks tiles of 128 rows x BN columns, 64 values of the reduction a stage:
//   warp 0       TMA: fp32 rows of A as they lie, the three planes of W (split once on the host)
//   warps 2-5    split A: a thread reads its row from shared memory and writes the three planes to tensor memory, from where the
//                products take their left operand -- read from shared memory, operands alone would need its whole bandwidth
//   warp 1       issues the 24 tcgen05.mma of a stage
//   warps 6-13   add up the accumulators in registers and finish the tile: the common forms straight into boxes that TMA stores (and
//                has filled with the residual), the others through shared memory in whole rows of 16-byte pieces
// With few tiles over a long reduction the CTAs of a cluster share it, as in kernels_umma.cu; partial tiles meet through distributed
// shared memory in rank order.
#include <cstddef>
#include <cstdio>
#include <cstdlib>

#include <algorithm>

#include "epilogue.cuh"
#include "tensor_maps.h"
#include "umma_ptx.cuh"

namespace b200 {
namespace {

constexpr int kRows = 128, kDepth = 64, kHalf = 32;   // rows of a tile, values of the reduction in a stage and in a split part of it
constexpr int kSplitWarps = 4, kSumWarps = 8, kFirstSplitter = 2, kFirstSummer = kFirstSplitter + kSplitWarps;
constexpr int kThreads = 32 * (kFirstSummer + kSumWarps);
constexpr int kMaxStages = 8;
constexpr uint32_t kBox = 16384;                       // 128 rows x 32 columns

struct F32UmmaParams {
  int M, N, C, H, W, R, S, P, Q, stride_h, stride_w, pad_t, pad_l;
  int im2col, chunks, tail_halves, num_kb, splits, m_tiles, total_tiles, stages;
  int plain;                 // fp32 results in rows of whole 16-byte pieces, at most one addend, no activation or a last ReLU
  int boxed;                 // ... which leave (and residuals arrive) through boxes of 128 rows x 32 columns by TMA
  int64_t a_row, a_img, a_h, a_w;   // floats from row to row of a product's A, from image to image, line to line and pixel to pixel of a convolution's
  uint32_t spin_limit;
  float least;               // results below this, zero apart, are computed again
  int test_skip_stage;       // test hook, as in kernels_umma.cu: the last stage of CTA 0's first tile is neither armed nor loaded
  const float* A;
  const uint16_t* planes;    // [num_kb][3][N][32]
  void* y;
  int* status;
  Epilogue ep;
};
struct SharedState { uint64_t full[kMaxStages], empty[kMaxStages], split[4], slot_empty[4], sum_empty[2], low_empty, res_full; uint32_t tmem; int abort; };
static_assert(offsetof(SharedState, split) == 16 * kMaxStages && offsetof(SharedState, sum_empty) == 16 * kMaxStages + 64 && offsetof(SharedState, res_full) == 16 * kMaxStages + 88,
              "the barriers are initialised as one array");

template <int BN> struct Tile {
  static constexpr uint32_t kABytes = kRows * kDepth * 4, kPlane = BN * kDepth * 2, kStage = kABytes + 3 * kPlane, kOut = kRows * BN * 4;
  static constexpr int kSlots = BN == 128 ? 2 : 4;            // split half stages of A in tensor memory
  static constexpr uint32_t kLow = 2 * BN, kSlot0 = 3 * BN;   // columns: two accumulators of leading products, one of small products, the slots
  static_assert(kSlot0 + kSlots * 48 <= 512, "tensor memory");
};

// Issued by the one lane of a converged warp whose `lead` is set: in a region that a single lane enters, the compiler moves every
// operand from vector to uniform registers in front of its product, and the tensor pipe waits for that (12 products of 64 columns take
// 770 clocks that way and 390 this way).
template <bool ACCUMULATE> __device__ __forceinline__ void umma_bf16_tmem_a(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "n"(ACCUMULATE ? 1 : 0), "r"(lead)
      : "memory");
}
__device__ __forceinline__ void umma_commit_at(uint32_t bar, uint32_t lead) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(lead) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
      "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float4 lds4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// The upper halves of two values (x at the lower address), which are bf16 values; the rest of both replaces them.  (After a first part that
// was rounded, cutting off leaves 8 + 8 + 8 bits as rounding does.)
__device__ __forceinline__ uint32_t split_off(float& x, float& y) {
  const uint32_t a = __float_as_uint(x), b = __float_as_uint(y);
  x = __fsub_rn(x, __uint_as_float(a & 0xffff0000u));
  y = __fsub_rn(y, __uint_as_float(b & 0xffff0000u));
  return __byte_perm(a, b, 0x7632);
}
// The first parts, rounded to nearest: the rests are half as large as with bits cut off, and of either sign, so that the small products' sums
// stay small where all operands have one sign (4608 of them: rms error 1.7e-7 -> 1.1e-7; ResNet-50 of 8 images 988 -> 1005 us).  Subnormals
// have none: a value of 2^-133 or less, rounded up here and away from zero below, could end as zero.  Above 3.396e38 they are infinite, and such
// results computed again.
__device__ __forceinline__ uint32_t split_first(float& x, float& y) {
  float a, b;
  uint32_t w;
  asm("mul.ftz.f32 %0, %1, 0f3F800000;" : "=f"(a) : "f"(x));
  asm("mul.ftz.f32 %0, %1, 0f3F800000;" : "=f"(b) : "f"(y));
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(b), "f"(a));
  x = __fsub_rn(x, __uint_as_float(w << 16));
  y = __fsub_rn(y, __uint_as_float(w & 0xffff0000u));
  return w;
}
// The third parts.  They are all that is left of a value of 2^-110 or more.  Of a smaller one bits below bf16's smallest, 2^-133, would be cut
// off, and nothing be left of many: it is rounded away from zero instead, so that a result of such values does not become a zero that
// hides among the true ones.  (`one` is 1, which the compiler does not know: a multiply-add has a pipe that stands idle here, an addition
// would queue with the other integer instructions.  ResNet-50 of 8 images 964 us without either, 976 and 979 with.)
__device__ __forceinline__ uint32_t split_last(float x, float y, uint32_t one) {
  uint32_t a, b;
  asm("mad.lo.u32 %0, %1, %2, 65535;" : "=r"(a) : "r"(__float_as_uint(x)), "r"(one));
  asm("mad.lo.u32 %0, %1, %2, 65535;" : "=r"(b) : "r"(__float_as_uint(y)), "r"(one));
  return __byte_perm(a, b, 0x7632);
}
// How many halves of a stage hold values: the last stage of a tap may have one.
__device__ __forceinline__ int halves_of(const F32UmmaParams& p, int chunk) { return chunk + 1 == p.chunks ? p.tail_halves : 2; }
__device__ __forceinline__ int next_chunk(const F32UmmaParams& p, int chunk) { return chunk + 1 == p.chunks ? 0 : chunk + 1; }
template <bool V> struct Const { static constexpr bool value = V; };
__device__ __forceinline__ void summers_sync() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(32 * kSumWarps) : "memory");
}

// Where the values of block kb of a row lie, and how many there are; null in the padding.
__device__ __forceinline__ const float* values_at(const F32UmmaParams& p, int row, int kb, int& count) {
  const int tap = kb / p.chunks, c0 = (kb - tap * p.chunks) * kDepth;
  count = min(kDepth, p.C - c0);
  if (!p.im2col) return p.A + (int64_t)row * p.a_row + c0;
  const int pq = p.P * p.Q, img = row / pq, op = (row - img * pq) / p.Q, oq = row - img * pq - op * p.Q;
  const int h = op * p.stride_h - p.pad_t + tap / p.S, w = oq * p.stride_w - p.pad_l + tap % p.S;
  if ((unsigned)h >= (unsigned)p.H || (unsigned)w >= (unsigned)p.W) return nullptr;
  return p.A + img * p.a_img + h * p.a_h + w * p.a_w + c0;
}
// What a row's values are: all finite, infinities among them (in blocks [first, last]), or a NaN, which makes every result NaN.
enum { ROW_FINITE, ROW_INFINITE, ROW_NAN };
struct RowKind { int kind, first, last; };
__device__ __noinline__ RowKind look_at_row(const F32UmmaParams& p, int row) {
  RowKind k{ROW_FINITE, 0, 0};
  for (int kb = 0; kb < p.num_kb; ++kb) {
    int count;
    const float* a = values_at(p, row, kb, count);
    if (!a) continue;
    uint32_t top = 0;
#pragma unroll 4
    for (int c = 0; c < count; c += 4) {
      const uint4 v = *(const uint4*)(a + c);
      top = max(max(max(top, v.x & 0x7fffffffu), v.y & 0x7fffffffu), max(v.z & 0x7fffffffu, v.w & 0x7fffffffu));
    }
    if (top > 0x7f800000u) { k.kind = ROW_NAN; return k; }
    if (top == 0x7f800000u) {
      if (k.kind == ROW_FINITE) { k.kind = ROW_INFINITE; k.first = kb; }
      k.last = kb;
    }
  }
  return k;
}
// The result of a row with infinities: they alone decide it.  Random signs meet within a few of them, where the walk ends.
__device__ __noinline__ float infinite_sum(const F32UmmaParams& p, int row, int col, int first, int last) {
  uint32_t sign = 2;   // none so far
  for (int kb = first; kb <= last; ++kb) {
    int count;
    const float* a = values_at(p, row, kb, count);
    if (!a) continue;
    const uint16_t* w1 = p.planes + ((int64_t)kb * 3 * p.N + col) * kDepth;   // (zero where the weight is, and of its sign)
    for (int c = 0; c < count; ++c) {
      const uint32_t v = __float_as_uint(a[c]);
      if ((v & 0x7fffffffu) != 0x7f800000u) continue;
      const uint32_t w = w1[c], here = (v >> 31) ^ (w >> 15);
      if ((w & 0x7fffu) == 0 || (sign != 2 && sign != here)) return __int_as_float(0x7fffffff);
      sign = here;
    }
  }
  return __uint_as_float(sign << 31 | 0x7f800000u);
}
// Two results of a row from the operands as they are: values in memory order, FMAs, padding left out.  Bound by its loads' latency; four
// chains at a time with loads ahead take half as long, but the registers of the call then cost the kernel 2 % on its ordinary way.
__device__ __noinline__ float2 replay(const F32UmmaParams& p, int row, int col0, int col1) {
  float sum[2] = {};
  const int64_t at[2] = {(int64_t)col0 * kDepth, (int64_t)col1 * kDepth};
  for (int kb = 0; kb < p.num_kb; ++kb) {
    int count;
    const float* a = values_at(p, row, kb, count);
    if (!a) continue;
    const uint16_t* w = p.planes + (int64_t)kb * 3 * p.N * kDepth;   // [3][p.N][64]
#pragma unroll 1
    for (int c = 0; c < count; c += 4) {
      const float4 v = *(const float4*)(a + c);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint2 u[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) u[i] = __ldg((const uint2*)(w + (int64_t)i * p.N * kDepth + at[j] + c));
        auto part = [&](int i, int k) { const uint32_t h = k < 2 ? u[i].x : u[i].y; return __uint_as_float(k & 1 ? h & 0xffff0000u : h << 16); };
        auto weight = [&](int k) { return part(0, k) + (part(1, k) + part(2, k)); };   // (both sums are exact)
        sum[j] = fmaf(v.x, weight(0), sum[j]);
        sum[j] = fmaf(v.y, weight(1), sum[j]);
        sum[j] = fmaf(v.z, weight(2), sum[j]);
        sum[j] = fmaf(v.w, weight(3), sum[j]);
      }
    }
  }
  return make_float2(sum[0], sum[1]);
}
__device__ __forceinline__ bool doubtful(const F32UmmaParams& p, float v) { return !(fabsf(v) < __int_as_float(0x7f800000)) || (v != 0.f && fabsf(v) < p.least); }
// Beside a tiny result a zero is doubtful as well: the coarse last parts of subnormals may have cancelled.
__device__ __forceinline__ bool any_tiny(const F32UmmaParams& p, const float* v, int n) {
  bool tiny = false;
  for (int j = 0; j < n; ++j) tiny = tiny || (v[j] != 0.f && fabsf(v[j]) < p.least);
  return tiny;
}
// Whether any of N is, in short independent chains: twice the bits less one is least for the smallest value that is not zero, and
// zero times a value is not zero where it is not finite.
template <int N> __device__ __forceinline__ bool any_doubtful(const F32UmmaParams& p, const float (&v)[N]) {
  constexpr int kChains = N < 4 ? N : 4;
  uint32_t least[kChains];
  float zero[kChains];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint32_t u = 2u * __float_as_uint(v[j]) - 1u;
    least[j % kChains] = j < kChains ? u : min(least[j % kChains], u);
    zero[j % kChains] = __fmaf_rn(v[j], 0.f, j < kChains ? 0.f : zero[j % kChains]);
  }
#pragma unroll
  for (int c = 1; c < kChains; ++c) { least[0] = min(least[0], least[c]); zero[0] = __fadd_rn(zero[0], zero[c]); }
  return least[0] < 2u * __float_as_uint(p.least) - 1u || !(zero[0] == 0.f);
}

// A tile's result lies in shared memory at `out`, row r's 16-byte piece c at c ^ (r & 7); with a shared reduction every CTA of the
// cluster has its part there.
template <int BN> __device__ __forceinline__ uint32_t result_at(uint32_t out, int r, int c) {
  return out + (uint32_t)(r * BN * 4) + (uint32_t)((((c >> 2) ^ (r & 7)) << 4) + (c & 3) * 4);
}
template <int BN, int W> __device__ __forceinline__ void read_result(const F32UmmaParams& p, uint32_t out, int r, int c, float (&x)[W]) {
  const uint32_t at = result_at<BN>(out, r, c);
  if (p.splits == 1) {
    if constexpr (W == 4) asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(at) : "memory");
    else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x[0]) : "r"(at) : "memory");
    return;
  }
#pragma unroll
  for (int j = 0; j < W; ++j) x[j] = 0.f;
  for (int k = 0; k < p.splits; ++k) {
    float u[W];
    if constexpr (W == 4)
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(u[0]), "=f"(u[1]), "=f"(u[2]), "=f"(u[3]) : "r"(map_to_cta(at, (uint32_t)k)) : "memory");
    else asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(u[0]) : "r"(map_to_cta(at, (uint32_t)k)) : "memory");
#pragma unroll
    for (int j = 0; j < W; ++j) x[j] = __fadd_rn(x[j], u[j]);
  }
}
// `n` sums of one row, of columns from `col` on, the doubtful ones among them computed again -- these alone: a result may not depend on
// which others lie beside it, as the width of the tiles follows this launch's share of the batch (32 columns are together in either).
// `beside_tiny`: there is a tiny one among those 32.
__device__ __noinline__ void sum_doubtful(const F32UmmaParams& p, float* sums, int n, int row, int col, bool beside_tiny) {
  if (row >= p.M) return;
  RowKind k{-1, 0, 0};
  bool tiny = beside_tiny;
  int held = -1;   // two are computed at a time
  for (int j = 0; j < n && col + j < p.N; ++j) {
    if (!beside_tiny && j % 32 == 0) tiny = any_tiny(p, sums + j, min(n - j, 32));
    if (!doubtful(p, sums[j]) && !(tiny && sums[j] == 0.f)) continue;
    if (k.kind < 0) k = look_at_row(p, row);
    if (k.kind == ROW_NAN) return;   // (they are NaN)
    if (k.kind == ROW_INFINITE) sums[j] = infinite_sum(p, row, col + j, k.first, k.last);
    else if (held < 0) held = j;
    else {
      const float2 s = replay(p, row, col + held, col + j);
      sums[held] = s.x;
      sums[j] = s.y;
      held = -1;
    }
  }
  if (held >= 0) sums[held] = replay(p, row, col + held, col + held).x;
}
// The doubtful ones among a thread's results, stored again where that changes anything.
template <int BN, int W>
__device__ __noinline__ void finish_doubtful(const F32UmmaParams& p, uint32_t out, int m0, int n0, int r_lo, int r_hi, int t) {
  const int c = t % (BN / W) * W, r0 = r_lo + t / (BN / W);
  if (n0 + c >= p.N) return;
  for (int r = r0; r < r_hi; r += 32 * kSumWarps * W / BN) {
    float x[W], again[W];
    read_result<BN, W>(p, out, r, c, x);
    bool zero = false, tiny = false;
    for (int j = 0; j < W; ++j) { again[j] = x[j]; zero = zero || x[j] == 0.f; }
    for (int k = c & ~31; zero && !tiny && k < (c | 31); k += 4) {
      float beside[4];
      read_result<BN, 4>(p, out, r, k, beside);
      tiny = any_tiny(p, beside, 4);
    }
    sum_doubtful(p, again, W, m0 + r, n0 + c, tiny);
    const int64_t row = (int64_t)m0 + r;
    for (int j = 0; j < W; ++j)
      if (__float_as_uint(again[j]) != __float_as_uint(x[j])) store_from_float(p.y, p.ep.out_dt, row * p.N + n0 + c + j, epilogue_value(p.ep, again[j], row, n0 + c + j, p.N));
  }
}
// Rows [r_lo, r_hi) of the tile that starts at (m0, n0): the epilogue (every step rounded by itself) and the store.  A thread keeps W
// columns, whose addends it reads once, and has several rows' residuals and results on the way at a time.  Returns whether any is doubtful.
template <int BN, int W>
__device__ __forceinline__ bool finish_rows(const F32UmmaParams& p, bool f32_io, uint32_t out, int m0, int n0, int r_lo, int r_hi, int t) {
  constexpr int kPerRow = BN / W, kStep = 32 * kSumWarps / kPerRow, kAhead = W == 4 ? 4 : 8;
  const Epilogue& ep = p.ep;
  const int c = t % kPerRow * W, col = n0 + c;
  if (col >= p.N) return false;
  float a1[W], a2[W];
#pragma unroll
  for (int j = 0; j < W; ++j) {
    a1[j] = f32_io && ep.add1 ? __ldg(ep.add1 + col + j) : 0.f;
    a2[j] = f32_io && ep.add2 ? __ldg(ep.add2 + col + j) : 0.f;
  }
  bool again = false;
  for (int r0 = r_lo + t / kPerRow; r0 < r_hi; r0 += kAhead * kStep) {
    float res[kAhead][W], x[kAhead][W] = {};
    const int64_t at0 = ((int64_t)m0 + r0) * p.N + col;
    if (f32_io && ep.res) {
#pragma unroll
      for (int i = 0; i < kAhead; ++i)
        if (r0 + i * kStep < r_hi) {
          const float* src = (const float*)ep.res + at0 + (int64_t)i * kStep * p.N;
          if constexpr (W == 4) { const float4 f = *(const float4*)src; res[i][0] = f.x; res[i][1] = f.y; res[i][2] = f.z; res[i][3] = f.w; }
          else res[i][0] = *src;
        }
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (r0 + i * kStep < r_hi) read_result<BN, W>(p, out, r0 + i * kStep, c, x[i]);
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      bool bad = false;
#pragma unroll
      for (int j = 0; j < W; ++j) {
        bad = bad || doubtful(p, x[i][j]);
        if (ep.alpha != 1.f) x[i][j] = __fmul_rn(x[i][j], ep.alpha);
        if (ep.add1) x[i][j] = __fadd_rn(x[i][j], a1[j]);
        if (ep.add2) x[i][j] = __fadd_rn(x[i][j], a2[j]);
      }
      again = again || (bad && r0 + i * kStep < r_hi);
    }
    if (f32_io) {
      float (&flat)[kAhead * W] = *(float (*)[kAhead * W])x;
      if (ep.act_first) apply_act_all<kAhead * W>(ep.act, flat, ep.act_a, ep.act_b);
      if (ep.res) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
#pragma unroll
          for (int j = 0; j < W; ++j) x[i][j] = __fadd_rn(x[i][j], res[i][j]);
      }
      if (!ep.act_first) apply_act_all<kAhead * W>(ep.act, flat, ep.act_a, ep.act_b);
#pragma unroll
      for (int i = 0; i < kAhead; ++i)
        if (r0 + i * kStep < r_hi) {
          float* dst = (float*)p.y + at0 + (int64_t)i * kStep * p.N;
          if constexpr (W == 4) *(float4*)dst = make_float4(x[i][0], x[i][1], x[i][2], x[i][3]);
          else *dst = x[i][0];
        }
    } else {
#pragma unroll 1
      for (int r = r0; r < min(r_hi, r0 + kAhead * kStep); r += kStep) {
        float v[W];
        read_result<BN, W>(p, out, r, c, v);
#pragma unroll
        for (int j = 0; j < W; ++j) store_from_float(p.y, ep.out_dt, ((int64_t)m0 + r) * p.N + col + j, epilogue_value(ep, v[j], (int64_t)m0 + r, col + j, p.N));
      }
    }
  }
  return again;
}
// The plain form (p.plain) of a shared reduction, with nothing left to decide for a result.
template <int BN>
__device__ __forceinline__ bool finish_plain_rows(const F32UmmaParams& p, uint32_t out, int m0, int n0, int r_lo, int r_hi, int t) {
  constexpr int kPerRow = BN / 4, kStep = 32 * kSumWarps / kPerRow;
  const Epilogue& ep = p.ep;
  const int c = t % kPerRow * 4, col = n0 + c;
  if (col >= p.N) return false;
  const float* addv = ep.add1 ? ep.add1 : ep.add2;
  const float4 add = addv ? __ldg((const float4*)(addv + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float* res = (const float*)ep.res;
  float* y = (float*)p.y;
  bool again = false;
#pragma unroll 2
  for (int r = r_lo + t / kPerRow; r < r_hi; r += kStep) {
    const int64_t at = ((int64_t)m0 + r) * p.N + col;
    const float4 f = res ? *(const float4*)(res + at) : make_float4(0.f, 0.f, 0.f, 0.f);
    float x[4];
    read_result<BN, 4>(p, out, r, c, x);
#pragma unroll
    for (int j = 0; j < 4; ++j) again = again || doubtful(p, x[j]);
    if (addv) { x[0] = __fadd_rn(x[0], add.x); x[1] = __fadd_rn(x[1], add.y); x[2] = __fadd_rn(x[2], add.z); x[3] = __fadd_rn(x[3], add.w); }
    if (res) { x[0] = __fadd_rn(x[0], f.x); x[1] = __fadd_rn(x[1], f.y); x[2] = __fadd_rn(x[2], f.z); x[3] = __fadd_rn(x[3], f.w); }
    if (ep.act == ACT_RELU) {
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = apply_act(ACT_RELU, x[j], 0.f, 0.f);
    }
    *(float4*)(y + at) = make_float4(x[0], x[1], x[2], x[3]);
  }
  return again;
}
// COLS columns of one row, straight from their sums into the row's places in the boxes of 32 columns that start at `at` (128-byte swizzle:
// 16-byte piece j of a row at j ^ (row & 7)); the residual lies there already.  Columns past N hold anything: the store clips them.
template <int COLS>
__device__ __forceinline__ void finish_in_boxes(const F32UmmaParams& p, float (&acc)[COLS], uint32_t at, int row, int m0, int col0) {
  const Epilogue& ep = p.ep;
  if (__any_sync(0xffffffffu, any_doubtful<COLS>(p, acc))) {   // (one branch for the warp, and through a copy: the sums themselves stay in registers)
    float copy[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) copy[j] = acc[j];
    sum_doubtful(p, copy, COLS, m0 + row, col0, false);
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] = copy[j];
  }
  const float* addv = ep.add1 ? ep.add1 : ep.add2;
#pragma unroll
  for (int q0 = 0; q0 < COLS / 4; q0 += 4) {
    float4 a[4];
    if (addv) {
#pragma unroll
      for (int q = 0; q < 4; ++q) a[q] = __ldg((const float4*)(addv + min(col0 + 4 * (q0 + q), p.N - 4)));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float* x = acc + 4 * (q0 + q);
        x[0] = __fadd_rn(x[0], a[q].x); x[1] = __fadd_rn(x[1], a[q].y); x[2] = __fadd_rn(x[2], a[q].z); x[3] = __fadd_rn(x[3], a[q].w);
      }
    }
    auto place = [&](int q) { return at + (uint32_t)((q0 + q) / 8) * kBox + (uint32_t)((((q0 + q) & 7) ^ (row & 7)) << 4); };
    if (ep.res) {
#pragma unroll
      for (int q = 0; q < 4; ++q) a[q] = lds4(place(q));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float* x = acc + 4 * (q0 + q);
        x[0] = __fadd_rn(x[0], a[q].x); x[1] = __fadd_rn(x[1], a[q].y); x[2] = __fadd_rn(x[2], a[q].z); x[3] = __fadd_rn(x[3], a[q].w);
      }
    }
    if (ep.act == ACT_RELU) {
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[4 * q0 + j] = apply_act(ACT_RELU, acc[4 * q0 + j], 0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float* x = acc + 4 * (q0 + q);
      asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(place(q)), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]) : "memory");
    }
  }
}
template <int BN>
__device__ __forceinline__ void finish_tile(const F32UmmaParams& p, uint32_t out, int m0, int n0, int r_lo, int r_hi, int t) {
  const Epilogue& ep = p.ep;
  const bool f32_io = !ep.mul && !ep.add_full && (!ep.res || ep.res_dt == DT_F32) && ep.out_dt == DT_F32, four = p.plain || (f32_io && (p.N & 3) == 0);
  const bool again = p.plain ? finish_plain_rows<BN>(p, out, m0, n0, r_lo, r_hi, t)
                     : four  ? finish_rows<BN, 4>(p, true, out, m0, n0, r_lo, r_hi, t)
                             : finish_rows<BN, 1>(p, f32_io, out, m0, n0, r_lo, r_hi, t);
  if (__any_sync(0xffffffffu, again)) {   // (over what was just stored; 32 columns of a row are one warp's, so that zeros beside a tiny result come along)
    if (four) finish_doubtful<BN, 4>(p, out, m0, n0, r_lo, r_hi, t);
    else finish_doubtful<BN, 1>(p, out, m0, n0, r_lo, r_hi, t);
  }
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
f32_umma_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmY,
                const __grid_constant__ CUtensorMap tmR, const __grid_constant__ F32UmmaParams p) {
  using T = Tile<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t base = smem_u32(smem), out = base + (uint32_t)p.stages * T::kStage;
  SharedState& sh = *(SharedState*)(smem + (size_t)p.stages * T::kStage + T::kOut);
  volatile int* abort_flag = &sh.abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)blockIdx.x % p.splits, first = (int)blockIdx.x / p.splits, step = (int)gridDim.x / p.splits;
  const int kb_lo = (int)((int64_t)p.num_kb * rank / p.splits), kb_hi = (int)((int64_t)p.num_kb * (rank + 1) / p.splits);
  const int tiles = first < p.total_tiles ? (p.total_tiles - first + step - 1) / step : 0, its = tiles * (kb_hi - kb_lo);
  if (warp == 0) {   // a lane per barrier
    constexpr int kSplit = 2 * kMaxStages, kSum = kSplit + 8;
    if (lane < kSum + 4) mbar_init(&sh.full[lane], lane >= kSplit && lane < kSplit + 4 ? kSplitWarps : lane >= kSum && lane < kSum + 3 ? kSumWarps : 1);
    if (lane == 0) { sh.abort = 0; prefetch_map(&tmA); prefetch_map(&tmB); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;

  if (warp == 0) {
    // ---------------------------------------------------------------------- loads ----
    if (elect_one()) {
      // A and W are walked separately: the weights of the first stages are constants and do not wait for the kernel in front
      int a_tile = first, a_kb = kb_lo, chunk = 0, c0 = 0, fr = 0, fs = 0, m0 = 0, w0 = 0, h0 = 0, img = 0, b_tile = first, b_kb = kb_lo;
      const int skip_tile = p.test_skip_stage && blockIdx.x == 0 ? first : -1;
      auto load_a = [&](int s) {
        if (a_kb == kb_lo) {
          m0 = (a_tile % p.m_tiles) * kRows;
          const int tap = kb_lo / p.chunks, pq = p.P * p.Q;
          chunk = kb_lo - tap * p.chunks; c0 = chunk * kDepth; fr = tap / p.S; fs = tap - fr * p.S;
          img = m0 / pq;
          const int rem = m0 - img * pq, op = rem / p.Q;
          h0 = op * p.stride_h - p.pad_t;
          w0 = (rem - op * p.Q) * p.stride_w - p.pad_l;
        }
        const uint32_t dst = base + (uint32_t)s * T::kStage, bar = smem_u32(&sh.full[s]);
        const int halves = halves_of(p, chunk);
        const bool skip = a_tile == skip_tile && a_kb + 1 == kb_hi;
        if (!skip) mbar_expect_tx(&sh.full[s], 3 * T::kPlane + (uint32_t)halves * (T::kABytes / 2));
        for (int i = skip ? halves : 0; i < halves; ++i) {   // (128 bytes of every row each; what lies past C arrives as zeros)
          if (p.im2col) load_im2col_at<false>(dst + (uint32_t)i * (T::kABytes / 2), &tmA, bar, c0 + i * kHalf, w0, h0, img, (uint16_t)fs, (uint16_t)fr);
          else load_2d_at<false>(dst + (uint32_t)i * (T::kABytes / 2), &tmA, bar, c0 + i * kHalf, m0);
        }
        chunk = next_chunk(p, chunk);
        c0 = chunk * kDepth;
        if (chunk == 0 && ++fs == p.S) { fs = 0; ++fr; }
        if (++a_kb == kb_hi) { a_kb = kb_lo; a_tile += step; }
      };
      auto load_b = [&](int s) {
        load_3d_at<false>(base + (uint32_t)s * T::kStage + T::kABytes, &tmB, smem_u32(&sh.full[s]), 0, (b_tile / p.m_tiles) * BN, 3 * b_kb);
        if (++b_kb == kb_hi) { b_kb = kb_lo; b_tile += step; }
      };
      const int early = min(p.stages, its);
      for (int s = 0; s < early; ++s) load_b(s);   // (their barriers are armed with A's loads)
      grid_dependency_wait();
      asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
      for (int s = 0; s < early; ++s) load_a(s);
      bool ok = true;
      int s = 0;
      uint32_t ph = 0;
      for (int it = early; it < its; ++it) {
        if (!mbar_wait(&sh.empty[s], ph, abort_flag, p.status, 31, p.spin_limit)) { ok = false; break; }
        load_a(s);
        load_b(s);
        if (++s == p.stages) { s = 0; ph ^= 1; }
      }
      if (!ok) await_stages(sh.full, p.stages, s, ph);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------- products ----
    const uint32_t lead = elect_one() ? 1u : 0u;
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);   // bf16 operands, fp32 sums
    constexpr uint32_t kDescHi = ((8u * 128u) >> 4) | (1u << 14) | (2u << 29);   // rows of 128 bytes, 128-byte swizzle, eight rows 1024 bytes apart
    const uint32_t lo0 = (1u << 16) | ((base + T::kABytes) >> 4), empty0 = smem_u32(sh.empty), slot0 = smem_u32(sh.slot_empty);
    uint32_t lo = lo0, ph = 0, slot_ph = 0, folds = 0;
    int s = 0, slot = 0;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, p.status, code, p.spin_limit)) != 0;
    };
    // The twelve products of half a stage; FIRST: the small ones start their sums.
    auto issue = [&](auto half_is, auto first_is, uint32_t high) {
      constexpr uint32_t kAt = decltype(half_is)::value ? 4u : 0u;
      constexpr bool kFirst = decltype(first_is)::value;
      const uint32_t a = tmem + T::kSlot0 + (uint32_t)slot * 48u, low = tmem + T::kLow;
      auto b_at = [&](int plane, int k) {
        uint64_t v;
        asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo + kAt + (uint32_t)((plane * (int)T::kPlane) >> 4) + 2u * (uint32_t)k), "r"(kDescHi));
        return v;
      };
      umma_bf16_tmem_a<(kAt > 0)>(high, a, b_at(0, 0), kIdesc, lead);
      umma_bf16_tmem_a<true>(high, a + 8u, b_at(0, 1), kIdesc, lead);
      umma_bf16_tmem_a<!kFirst>(low, a + 32u, b_at(0, 0), kIdesc, lead);   // the smallest first: a3 w1, a2 w2, a2 w1, a1 w3, a1 w2
      umma_bf16_tmem_a<true>(low, a + 40u, b_at(0, 1), kIdesc, lead);
#pragma unroll
      for (int k = 0; k < 2; ++k) umma_bf16_tmem_a<true>(low, a + 16u + 8u * k, b_at(1, k), kIdesc, lead);
#pragma unroll
      for (int k = 0; k < 2; ++k) umma_bf16_tmem_a<true>(low, a + 16u + 8u * k, b_at(0, k), kIdesc, lead);
#pragma unroll
      for (int k = 0; k < 2; ++k) umma_bf16_tmem_a<true>(low, a + 8u * k, b_at(2, k), kIdesc, lead);
#pragma unroll
      for (int k = 0; k < 2; ++k) umma_bf16_tmem_a<true>(low, a + 8u * k, b_at(1, k), kIdesc, lead);
      umma_commit_at(slot0 + 8u * slot, lead);
      if (++slot == T::kSlots) { slot = 0; slot_ph ^= 1; }
    };
    for (int n = 0; n < tiles && ok; ++n) {
      if (n > 0) ok = wait(&sh.low_empty, (uint32_t)(n - 1) & 1, 32);
      int chunk = kb_lo % p.chunks;
      for (int kb = kb_lo; kb < kb_hi && ok; ++kb, ++folds) {
        const int halves = halves_of(p, chunk);
        chunk = next_chunk(p, chunk);
        const uint32_t d = folds & 1, high = tmem + d * (uint32_t)BN;
        if (!(ok = wait(&sh.sum_empty[d], ((folds >> 1) & 1) ^ 1, 33))) break;
        if (!(ok = wait(&sh.full[s], ph, 34))) break;
        if (!(ok = wait(&sh.split[slot], slot_ph, 35))) break;
        tc_fence_after();
        if (kb == kb_lo) issue(Const<false>{}, Const<true>{}, high);
        else issue(Const<false>{}, Const<false>{}, high);
        if (halves == 2) {
          if (!(ok = wait(&sh.split[slot], slot_ph, 35))) break;
          tc_fence_after();
          issue(Const<true>{}, Const<false>{}, high);
        }
        umma_commit_at(empty0 + 8u * s, lead);   // (the sums of these products are complete as well)
        lo += T::kStage >> 4;
        if (++s == p.stages) { s = 0; ph ^= 1; lo = lo0; }
      }
    }
  } else if (warp < kFirstSummer) {
    // ------------------------------------------------------------------- splits A ----
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t one = (uint32_t)min(p.stages, 1), rx = (uint32_t)(row & 7), lane_addr = (uint32_t)(quarter * 32) << 16;
    int s = 0, slot = 0;
    uint32_t ph = 0, slot_ph = 1;   // (the first round of slots is free)
    bool ok = true;   // (a lane's own: whatever becomes of the waits, the warp stays together for its collective stores)
    for (int it = 0, left = 0, chunk = 0; it < its; ++it, --left) {
      if (left == 0) { left = kb_hi - kb_lo; chunk = kb_lo % p.chunks; }   // the next tile
      const int halves = halves_of(p, chunk);
      chunk = next_chunk(p, chunk);
      for (int half = 0; half < halves; ++half) {
        if (ok) ok = mbar_wait(&sh.full[s], ph, abort_flag, p.status, 36, p.spin_limit);
        const uint32_t at = base + (uint32_t)s * T::kStage + (uint32_t)half * (T::kABytes / 2) + (uint32_t)row * 128u;
        uint32_t w1[16], w2[16], w3[16];
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q) {
          float4 v = lds4(at + ((q ^ rx) << 4));
          w1[2 * q] = split_first(v.x, v.y); w1[2 * q + 1] = split_first(v.z, v.w);
          w2[2 * q] = split_off(v.x, v.y); w2[2 * q + 1] = split_off(v.z, v.w);
          w3[2 * q] = split_last(v.x, v.y, one); w3[2 * q + 1] = split_last(v.z, v.w, one);
        }
        if (ok) ok = mbar_wait(&sh.slot_empty[slot], slot_ph, abort_flag, p.status, 37, p.spin_limit);
        tc_fence_after();
        const uint32_t dst = tmem + lane_addr + T::kSlot0 + (uint32_t)slot * 48u;
        tmem_st16(dst, w1);
        tmem_st16(dst + 16u, w2);
        tmem_st16(dst + 32u, w3);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.split[slot]);
        if (++slot == T::kSlots) { slot = 0; slot_ph ^= 1; }
      }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
  } else {
    // ---------------------------------------------------------------------- sums ----
    const int half = (warp - kFirstSummer) >> 2, quarter = warp & 3, row = quarter * 32 + lane, t = (int)threadIdx.x - 32 * kFirstSummer;
    const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * (BN / 2));
    uint32_t folds = 0, ph = 0;
    int s = 0;
    bool ok = true;   // (after a wait that ran out the walk goes on without waiting: every warp has to meet the others' barriers)
    grid_dependency_wait();   // residuals are read, and tensors earlier kernels may still read overwritten, from here on
    auto ask_for_residual = [&](int tile) {   // one thread
      const int m0 = (tile % p.m_tiles) * kRows, n0 = (tile / p.m_tiles) * BN, boxes = min(BN / 32, (p.N - n0 + 31) / 32);
      mbar_expect_tx(&sh.res_full, (uint32_t)boxes * kBox);
      for (int b = 0; b < boxes; ++b) load_2d_at<false>(out + (uint32_t)b * kBox, &tmR, smem_u32(&sh.res_full), n0 + 32 * b, m0);
    };
    if (t == 0 && p.boxed) {
      prefetch_map(&tmY);
      if (p.ep.res && tiles > 0) ask_for_residual(first);
    }
    for (int n = 0, tile = first; n < tiles; ++n, tile += step) {
      float acc[BN / 2];
#pragma unroll
      for (int j = 0; j < BN / 2; ++j) acc[j] = 0.f;
      auto add = [&](uint32_t at) {
#pragma unroll
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[16];
          tmem_ld16(at + 16u * c, r);
          tmem_ld_wait_regs<16>(r);
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[16 * c + j] = __fadd_rn(acc[16 * c + j], __uint_as_float(r[j]));
        }
      };
      for (int kb = kb_lo; kb < kb_hi; ++kb, ++folds) {
        const uint32_t d = folds & 1;
        if (ok) ok = mbar_wait(&sh.empty[s], ph, abort_flag, p.status, 38, p.spin_limit);   // (this stage's products are complete)
        if (++s == p.stages) { s = 0; ph ^= 1; }
        tc_fence_after();
        add(taddr + d * (uint32_t)BN);
        if (kb + 1 == kb_hi) add(taddr + T::kLow);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&sh.sum_empty[d]);
          if (kb + 1 == kb_hi) mbar_arrive(&sh.low_empty);
        }
      }
      const int m0 = (tile % p.m_tiles) * kRows, n0 = (tile / p.m_tiles) * BN;
      if (p.boxed) {
        // the row's columns are finished in their box, over the residual that TMA has put there
        if (p.ep.res) ok &= mbar_wait(&sh.res_full, (uint32_t)n & 1, abort_flag, p.status, 40, p.spin_limit);   // (always: it lands whatever became of the products)
        else if (n > 0) {
          if (t == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          summers_sync();   // the stores of the tile before have read the boxes
        }
        finish_in_boxes<BN / 2>(p, acc, out + (uint32_t)(half * (BN / 64)) * kBox + (uint32_t)row * 128u, row, m0, n0 + half * (BN / 2));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        summers_sync();
        if (t == 0) {
          for (int b = 0; b < BN / 32 && n0 + 32 * b < p.N; ++b)
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"((uint64_t)&tmY), "r"(out + (uint32_t)b * kBox), "r"(n0 + 32 * b), "r"(m0) : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          if (p.ep.res && n + 1 < tiles) {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            ask_for_residual(tile + step);
          }
        }
        continue;
      }
      const uint32_t at = out + (uint32_t)(row * BN * 4);
#pragma unroll
      for (int q = 0; q < BN / 8; ++q) {
        const uint32_t piece = (uint32_t)(half * (BN / 8) + q) ^ (uint32_t)(row & 7);
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at + (piece << 4)), "f"(acc[4 * q]), "f"(acc[4 * q + 1]), "f"(acc[4 * q + 2]), "f"(acc[4 * q + 3]) : "memory");
      }
      if (p.splits == 1) {
        summers_sync();
        finish_tile<BN>(p, out, m0, n0, 0, min(kRows, p.M - m0), t);
        summers_sync();   // the next tile overwrites what others may still read
      }
    }
    if (t == 0 && p.boxed) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // stores complete before shared memory is released
  }
  __syncwarp();
  tc_fence_before();
  if (p.splits > 1) {
    cluster_sync_all();
    if (warp >= kFirstSummer && tiles > 0) {
      const int m0 = (first % p.m_tiles) * kRows, rows = min(kRows, p.M - m0);
      finish_tile<BN>(p, out, m0, (first / p.m_tiles) * BN, rows * rank / p.splits, rows * (rank + 1) / p.splits, (int)threadIdx.x - 32 * kFirstSummer);
    }
    cluster_sync_all();   // nobody leaves while a peer may still read its partial tile
  } else {
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

template <int BN> size_t smem_bytes() { return (size_t)(BN == 128 ? 2 : 3) * Tile<BN>::kStage + Tile<BN>::kOut + 1024 /*alignment slack*/ + sizeof(SharedState); }
template <int BN> bool allow_smem() {
  static bool set[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 16 && set[dev]) return true;
  if (cudaFuncSetAttribute(f32_umma_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) { cudaGetLastError(); return false; }
  if (dev >= 0 && dev < 16) set[dev] = true;
  return true;
}
// How many clusters of n CTAs run at a time: they have to find their SMs inside one part of the chip each, which leaves some over.
int clusters_at_once(int n, int sms) {
  static int cache[16][9] = {};
  int dev = 0;
  if (n == 1 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return std::max(1, sms / n);
  if (cache[dev][n]) return cache[dev][n];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(sms / n * n));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem_bytes<64>();
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)n; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int fit = 0;
  if (!allow_smem<64>() || cudaOccupancyMaxActiveClusters(&fit, f32_umma_kernel<64>, &cfg) != cudaSuccess || fit <= 0) { cudaGetLastError(); fit = std::max(1, sms / n); }
  return cache[dev][n] = fit;
}

// How many CTAs share a tile's reduction, from the rows of the whole recorded batch alone (it is the order of the sums, see
// choose_split in kernels_umma.cu), and how many columns this launch's tiles have (which changes no sum).  In clocks: half a stage
// takes 12 products of 66 (128 columns) or 42; a tile about 3500 to fill and to finish, a cluster 2500 more.
struct Shape { int splits, bn; };
double launch_cost(int64_t rows, int64_t n, int num_halves, int bn, int splits, int sms) {
  const int64_t tiles = (rows + kRows - 1) / kRows * ((n + bn - 1) / bn), fit = clusters_at_once(splits, sms), rounds = (tiles + fit - 1) / fit;
  const double walk = (double)((num_halves + splits - 1) / splits) * 12 * (bn == 128 ? 66 : 42);
  return splits == 1 ? (double)rounds * (walk + 1000.0) + 2500.0 : (double)rounds * (walk + 6000.0);
}
Shape choose_shape(int64_t rows_full, int64_t rows, int64_t n, int num_kb, int num_halves, int sms) {
  Shape best{1, 64};
  double least = -1;
  for (int splits = 1; splits <= 8 && splits <= num_kb; splits *= 2)
    for (int bn = 64; bn <= 128; bn *= 2) {
      const double c = launch_cost(rows_full, n, num_halves, bn, splits, sms);
      if (least < 0 || c < least) { least = c; best.splits = splits; }
    }
  least = -1;
  for (int bn = 64; bn <= 128; bn *= 2) {
    const double c = launch_cost(rows, n, num_halves, bn, best.splits, sms);
    if (least < 0 || c < least) { least = c; best.bn = bn; }
  }
  return best;
}

}  // namespace

struct F32UmmaLaunch {
  CUtensorMap tmA, tmB, tmY, tmR;
  F32UmmaParams p;
  int grid, bn;
  size_t smem;
};

bool f32_umma_supported(const F32Umma& c) {
  if (c.N < 1 || c.H < 1 || c.W < 1 || c.P < 1 || c.Q < 1 || c.K < 1 || c.C < 4 || c.C % 4) return false;   // TMA: rows of whole 16-byte pieces
  if (c.R < 1 || c.S < 1 || c.R > 128 || c.S > 128 || c.R * c.S > 4096 || c.stride_h < 1 || c.stride_w < 1 || c.stride_h > 8 || c.stride_w > 8) return false;
  if (c.pad_t > 127 || c.pad_l > 127) return false;   // the corners of an im2col map have eight bits
  const int64_t lim = 127, dw = (int64_t)(c.Q - 1) * c.stride_w - c.pad_l - (c.W - 1), dh = (int64_t)(c.P - 1) * c.stride_h - c.pad_t - (c.H - 1);
  if (dw < -128 || dw > lim || dh < -128 || dh > lim) return false;
  // (blocks: while a row is computed again, other roles' waits go on; half a million values take about a third of their limit)
  return (int64_t)c.N * c.P * c.Q < (1ll << 31) - kRows && c.K < (1 << 30) && f32_umma_blocks(c) < (1 << 13) && c.rows_full < (1ll << 40);
}
int64_t f32_umma_blocks(const F32Umma& c) { return (int64_t)c.R * c.S * ((c.C + kDepth - 1) / kDepth); }

// From 280 shapes timed on this kernel and on the CUDA cores (convolutions of 1 to 16 images of 7 x 7 to 56 x 56 pixels, 4 to 1024 channels, 1x1
// to 5x5 windows; products of 1 to 8192 rows), in us.  What a launch costs before its first product, 8 to 10, is what the CUDA cores need for
// few results or a short reduction (421 x 256 x 256: 12.2 there and 12.9 here; 3197 x 2048 x 1000: 324 and 109); taps with
// few channels leave most of a stage's 32 columns empty (8 x 26 x 26 x 8 -> 512, 5x5: 56 and 64); narrow results most of a tile's.
bool f32_umma_pays(const F32Umma& c) {
  const int64_t depth = (int64_t)c.R * c.S * c.C, results = c.rows_full * c.K, halves = (int64_t)c.R * c.S * ((c.C + kHalf - 1) / kHalf);
  if (getenv("ODLA_B200_NO_F32_UMMA") || c.K < 16 || 3 * depth < kHalf * halves) return false;
  return depth > 256 ? results > 16384 : (depth >= 64 ? results > 131072 : depth >= 24 && results > (1 << 20));
}

F32UmmaLaunch* f32_umma_prepare(const F32Umma& c, const void* x, const void* planes, void* y, const Epilogue& ep, int* status, int sms) {
  if (!f32_umma_supported(c) || (uintptr_t)x % 16 || (uintptr_t)y % 16 || !load_driver_entry_points()) return nullptr;
  auto* L = new F32UmmaLaunch();
  F32UmmaParams& p = L->p;
  p.M = c.N * c.P * c.Q; p.N = c.K; p.C = c.C; p.H = c.H; p.W = c.W; p.R = c.R; p.S = c.S; p.P = c.P; p.Q = c.Q;
  p.stride_h = c.stride_h; p.stride_w = c.stride_w; p.pad_t = c.pad_t; p.pad_l = c.pad_l;
  p.im2col = !(!c.x_w_stride && c.R == 1 && c.S == 1 && c.stride_h == 1 && c.stride_w == 1 && c.pad_t == 0 && c.pad_l == 0 && c.P == c.H && c.Q == c.W);
  p.chunks = (c.C + kDepth - 1) / kDepth;
  p.tail_halves = c.C - (p.chunks - 1) * kDepth > kHalf ? 2 : 1;
  p.num_kb = (int)f32_umma_blocks(c);
  p.a_row = c.C;
  p.a_w = c.x_w_stride ? c.x_w_stride / 4 : c.C; p.a_h = c.x_w_stride ? c.x_h_stride / 4 : (int64_t)c.W * c.C; p.a_img = p.a_h * c.H;
  const Shape shape = choose_shape(std::max<int64_t>(c.rows_full, p.M), p.M, c.K, p.num_kb, c.R * c.S * (2 * (p.chunks - 1) + p.tail_halves), sms);
  p.splits = shape.splits;
  L->bn = shape.bn;
  p.m_tiles = (p.M + kRows - 1) / kRows;
  const int64_t tiles = (int64_t)p.m_tiles * ((c.K + L->bn - 1) / L->bn);
  if (tiles * p.splits >= (1ll << 30)) { delete L; return nullptr; }
  p.total_tiles = (int)tiles;
  p.stages = L->bn == 128 ? 2 : 3;
  L->grid = p.splits > 1 ? p.total_tiles * p.splits : std::min(p.total_tiles, sms);
  L->smem = L->bn == 128 ? smem_bytes<128>() : smem_bytes<64>();
  // What a value of A is off by is below 2^-133 (split_last), what a product may lose below the smallest fp32 2^-149 six times; against 2^-26
  // of a result.  (Measured with nothing computed again, 2048 x 576 x 256: errors are those of ordinary sizes down to results of 2^-104.)
  p.least = std::max(0x1p-100f, (float)((double)c.R * c.S * c.C * 0x1p-107) * std::max(c.largest_weight, 0x1p-13f));
  p.spin_limit = kSpinLimit;
  p.test_skip_stage = getenv("ODLA_B200_TEST_SKIP_STAGE") != nullptr;   // (the hooks of umma_conv_prepare)
  if (const char* e = getenv("ODLA_B200_TEST_SPIN_LIMIT")) { const long v = atol(e); if (v >= 64 && v <= (1l << 18)) p.spin_limit = (uint32_t)v; }
  p.A = (const float*)x; p.planes = (const uint16_t*)planes; p.y = y; p.status = status; p.ep = ep;
  CUresult r;
  if (p.im2col) {
    cuuint64_t dims[4] = {(cuuint64_t)c.C, (cuuint64_t)c.W, (cuuint64_t)c.H, (cuuint64_t)c.N};
    cuuint64_t strides[3] = {(cuuint64_t)p.a_w * 4, (cuuint64_t)p.a_h * 4, (cuuint64_t)p.a_img * 4};
    int lower[2] = {-c.pad_l, -c.pad_t};
    int upper[2] = {(c.Q - 1) * c.stride_w - c.pad_l - (c.W - 1), (c.P - 1) * c.stride_h - c.pad_t - (c.H - 1)};
    cuuint32_t estr[4] = {1, (cuuint32_t)c.stride_w, (cuuint32_t)c.stride_h, 1};
    r = g_encode_im2col(&L->tmA, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void*)x, dims, strides, lower, upper, kHalf, kRows, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    int drv = 0;
    cudaDriverGetVersion(&drv);   // (the same work-around as in umma_conv_prepare)
    if (r == CUDA_SUCCESS && drv <= 13010 && c.N * p.a_img * 4 < 131072) ((uint64_t*)&L->tmA)[1] &= ~(1ull << 21);
  } else {
    cuuint64_t dims[2] = {(cuuint64_t)c.C, (cuuint64_t)p.M};
    cuuint64_t strides[1] = {(cuuint64_t)c.C * 4};
    cuuint32_t box[2] = {kHalf, kRows}, estr[2] = {1, 1};
    r = g_encode_tiled(&L->tmA, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)x, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (r == CUDA_SUCCESS) {
    cuuint64_t dims[3] = {kDepth, (cuuint64_t)c.K, (cuuint64_t)p.num_kb * 3};
    cuuint64_t strides[2] = {kDepth * 2, (cuuint64_t)c.K * kDepth * 2};
    cuuint32_t box[3] = {kDepth, (cuuint32_t)L->bn, 3}, estr[3] = {1, 1, 1};
    r = g_encode_tiled(&L->tmB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)planes, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  p.plain = c.K % 4 == 0 && !ep.mul && !ep.add_full && ep.out_dt == DT_F32 && ep.alpha == 1.f && !(ep.add1 && ep.add2) &&
            (ep.act == ACT_NONE || (ep.act == ACT_RELU && !ep.act_first)) && (!ep.res || (ep.res_dt == DT_F32 && (uintptr_t)ep.res % 16 == 0));
  p.boxed = p.plain && p.splits == 1;
  L->tmY = L->tmR = L->tmA;
  if (r == CUDA_SUCCESS && p.boxed) {
    cuuint64_t dims[2] = {(cuuint64_t)c.K, (cuuint64_t)p.M};
    cuuint64_t strides[1] = {(cuuint64_t)c.K * 4};
    cuuint32_t box[2] = {32, kRows}, estr[2] = {1, 1};
    auto encode = [&](CUtensorMap* m, const void* at, CUtensorMapL2promotion l2) {
      return g_encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)at, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, l2,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    r = encode(&L->tmY, y, CU_TENSOR_MAP_L2_PROMOTION_NONE);
    if (r == CUDA_SUCCESS && ep.res) r = encode(&L->tmR, ep.res, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
  }
  if (r != CUDA_SUCCESS || !(L->bn == 128 ? allow_smem<128>() : allow_smem<64>())) {
    if (!c.x_w_stride) fprintf(stderr, "[odla_b200] fp32 tensor-core launch cannot be prepared: %d\n", (int)r);  // overlapping strides are an optional fast path
    delete L;
    return nullptr;
  }
  return L;
}

int f32_umma_run(F32UmmaLaunch* L, cudaStream_t stream) {
  if (!L) return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)L->grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = L->smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  static const bool pdl = !getenv("ODLA_B200_NO_PDL");
  int na = 0;
  if (pdl) { attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[na].val.programmaticStreamSerializationAllowed = 1; ++na; }
  if (L->p.splits > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = (unsigned)L->p.splits; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  const cudaError_t e = L->bn == 128 ? cudaLaunchKernelEx(&cfg, f32_umma_kernel<128>, L->tmA, L->tmB, L->tmY, L->tmR, L->p)
                                   : cudaLaunchKernelEx(&cfg, f32_umma_kernel<64>, L->tmA, L->tmB, L->tmY, L->tmR, L->p);
  if (e != cudaSuccess) { fprintf(stderr, "[odla_b200] fp32 tensor-core launch failed: %s\n", cudaGetErrorString(e)); cudaGetLastError(); return -2; }
  return 0;
}
void f32_umma_destroy(F32UmmaLaunch* L) { delete L; }

}  // namespace b200
