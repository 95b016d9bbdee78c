// fp32 convolution (NHWC, one group) and batched GEMM on the CUDA cores, for what kernels_f32_umma.cu does not take: products of two
// run-time tensors, few results, short reductions, channels that are no multiple of four.  The bound is the FMA pipe: 128 fp32 FMA per clock and
// SM, 74 TFLOP/s at 1965 MHz.
//
//   C[b][M, N] = A[b][M, K] * B[b][N, K]^T      convolution: M = N*P*Q pixels, K = R*S*C gathered on the fly
//
// One CTA of two warps owns a 64 x 64 tile, a thread 8 x 8 results.  Both operands sit in shared memory K-major (rows of 32
// floats = 128 bytes), so that one 16-byte read brings four consecutive k of one row and the products go through the
// packed fma.rn.f32x2: each accumulator is a pair (even k, odd k) that is added up at the end -- no register moves to
// build operand pairs, 16 shared-memory reads per 128 packed FMAs.  Rows are swizzled like TMA's 128-byte mode (piece j of
// row r at j ^ (r & 7)), which makes the eight rows a warp reads at a time land in different banks.  Operands arrive by
// cp.async three stages deep: 16-byte pieces where four neighbouring k are contiguous and aligned, 4-byte elements otherwise
// (a 3-channel image, an odd reduction length, a transposed operand); out-of-range pieces are zero-filled by the copy.
//
// Measured: 37 TFLOP/s on a 3x3 convolution of 128 channels at 56 x 56 x 16 (the one-thread-per-output kernel before: 2.1).
// What is left: a packed FMA with three different register pairs takes 3.6 cycles instead of 2 (register reads; a loop
// of nothing else measures the same), scalar FMAs on the same tile reach the same rate from the instruction cache's side.
//
// Four CTAs share an SM (eight warps, 256 registers a thread).  When the tiles alone do not fill the chip the reduction is split
// over the CTAs of a cluster: each leaves its partial tile in its own shared memory and then adds up and stores a share
// of the rows, reading its peers' partials in rank order, so that the result does not depend on timing.
#include <cstdio>
#include <cstdlib>

#include <algorithm>

#include "epilogue.cuh"

namespace b200 {
namespace {

constexpr int kTile = 64, kThreads = 64, kStages = 3, kBK = 32;
constexpr int kOperandBytes = kTile * kBK * 4;                  // 8 KB per operand and stage
constexpr int kPitch = kTile + 4;                               // floats per row of the result tile: rows land 4 banks apart
constexpr int kSmem = kStages * 2 * kOperandBytes + kTile * 16;  // operand stages (the result tile reuses them) and the row table
static_assert(kTile * kPitch * 4 <= kStages * 2 * kOperandBytes, "the result tile fits the operand stages");

enum { LOAD_CONV_VEC, LOAD_CONV_SCALAR, LOAD_GEMM_VEC, LOAD_GEMM_SCALAR };

struct F32Params {
  int M, N, K, num_kb, m_tiles, n_tiles, splits, batches;
  int64_t a_row, a_col, a_batch, b_row, b_col, b_batch;
  int H, W, C, R, S, P, Q, stride_h, stride_w, pad_t, pad_l;
  const float *A, *B;
  void* y;
  Epilogue ep;
};
struct RowInfo { long long base; int h0, w0; };   // first input element of a pixel's window and where that window starts

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void lds_pair(uint32_t addr, unsigned long long& x, unsigned long long& y) {
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(addr));
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint32_t piece_at(uint32_t tile, int row, int piece) { return tile + (uint32_t)(row * 128 + ((piece ^ (row & 7)) << 4)); }

// One stage of A: k-block kb of the tile's 64 rows.
template <int LA>
__device__ __forceinline__ void load_a(const F32Params& p, uint32_t dst, const float* A, const RowInfo* rows, int m0, int kb) {
  const int t = threadIdx.x;
  if (LA == LOAD_CONV_VEC) {
    const int piece = t & 7, k = kb * kBK + piece * 4;
    const int tap = k / p.C, c = k - tap * p.C, r = tap / p.S, s = tap - r * p.S;
    const int64_t off = ((int64_t)r * p.W + s) * p.C + c;
    const bool k_ok = k < p.K;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = (t >> 3) + 8 * i;
      const RowInfo ri = rows[row];
      const bool ok = k_ok && (unsigned)(ri.h0 + r) < (unsigned)p.H && (unsigned)(ri.w0 + s) < (unsigned)p.W;
      copy16(piece_at(dst, row, piece), ok ? A + ri.base + off : A, ok);
    }
  } else if (LA == LOAD_CONV_SCALAR) {
    const int kl = t & 31, k = kb * kBK + kl;
    const int tap = k / p.C, c = k - tap * p.C, r = tap / p.S, s = tap - r * p.S;
    const int64_t off = ((int64_t)r * p.W + s) * p.C + c;
    const bool k_ok = k < p.K;
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
      const int row = (t >> 5) + 2 * i;
      const RowInfo ri = rows[row];
      const bool ok = k_ok && (unsigned)(ri.h0 + r) < (unsigned)p.H && (unsigned)(ri.w0 + s) < (unsigned)p.W;
      copy4(piece_at(dst, row, kl >> 2) + (kl & 3) * 4, ok ? A + ri.base + off : A, ok);
    }
  } else if (LA == LOAD_GEMM_VEC) {
    const int piece = t & 7, k = kb * kBK + piece * 4;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = (t >> 3) + 8 * i;
      const bool ok = k < p.K && m0 + row < p.M;
      copy16(piece_at(dst, row, piece), ok ? A + (int64_t)(m0 + row) * p.a_row + k : A, ok);
    }
  } else {
    const bool along_k = p.a_col == 1;   // neighbouring lanes read neighbouring addresses whichever axis is contiguous
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
      const int row = along_k ? (t >> 5) + 2 * i : t, kl = along_k ? t & 31 : i, k = kb * kBK + kl;
      const bool ok = k < p.K && m0 + row < p.M;
      copy4(piece_at(dst, row, kl >> 2) + (kl & 3) * 4, ok ? A + (int64_t)(m0 + row) * p.a_row + (int64_t)k * p.a_col : A, ok);
    }
  }
}
template <bool VEC>
__device__ __forceinline__ void load_b(const F32Params& p, uint32_t dst, const float* B, int n0, int kb) {
  const int t = threadIdx.x;
  if (VEC) {
    const int piece = t & 7, k = kb * kBK + piece * 4;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = (t >> 3) + 8 * i;
      const bool ok = k < p.K && n0 + row < p.N;
      copy16(piece_at(dst, row, piece), ok ? B + (int64_t)(n0 + row) * p.b_col + k : B, ok);
    }
  } else {
    const bool along_k = p.b_row == 1;
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
      const int row = along_k ? (t >> 5) + 2 * i : t, kl = along_k ? t & 31 : i, k = kb * kBK + kl;
      const bool ok = k < p.K && n0 + row < p.N;
      copy4(piece_at(dst, row, kl >> 2) + (kl & 3) * 4, ok ? B + (int64_t)(n0 + row) * p.b_col + (int64_t)k * p.b_row : B, ok);
    }
  }
}

// Four neighbouring results of one row, fp32 in and out without multiplier or full-matrix addend.  Every step is rounded by itself,
// as in epilogue_value.
__device__ __forceinline__ void finish4(const F32Params& p, float4 v, int64_t row, int col) {
  const Epilogue& ep = p.ep;
  float t[4] = {v.x, v.y, v.z, v.w};
  auto add = [&](const float4& a) { t[0] = __fadd_rn(t[0], a.x); t[1] = __fadd_rn(t[1], a.y); t[2] = __fadd_rn(t[2], a.z); t[3] = __fadd_rn(t[3], a.w); };
  if (ep.alpha != 1.f) {
#pragma unroll
    for (int j = 0; j < 4; ++j) t[j] = __fmul_rn(t[j], ep.alpha);
  }
  if (ep.add1) add(__ldg((const float4*)(ep.add1 + col)));
  if (ep.add2) add(__ldg((const float4*)(ep.add2 + col)));
  if (ep.act_first) apply_act_all<4>(ep.act, t, ep.act_a, ep.act_b);
  if (ep.res) add(*(const float4*)((const float*)ep.res + row * p.N + col));
  if (!ep.act_first) apply_act_all<4>(ep.act, t, ep.act_a, ep.act_b);
  *(float4*)((float*)p.y + row * p.N + col) = make_float4(t[0], t[1], t[2], t[3]);
}

template <int LA, bool BVEC>
__global__ void __launch_bounds__(kThreads, 4) f32_tile_kernel(const F32Params p) {
  extern __shared__ __align__(128) uint8_t smem[];
  RowInfo* rows = (RowInfo*)(smem + kStages * 2 * kOperandBytes);
  const int t = threadIdx.x, lane = t & 31, ty = lane >> 2, tx = (lane & 3) + 4 * (t >> 5);
  const int per_batch = p.m_tiles * p.n_tiles, batch = (int)blockIdx.x / per_batch, tile = (int)blockIdx.x - batch * per_batch;
  const int m0 = (tile % p.m_tiles) * kTile, n0 = (tile / p.m_tiles) * kTile;
  const int rank = (int)blockIdx.z;
  const int kb_lo = (int)((int64_t)p.num_kb * rank / p.splits), kb_hi = (int)((int64_t)p.num_kb * (rank + 1) / p.splits);
  const float *A = p.A + batch * p.a_batch, *B = p.B + batch * p.b_batch;
  if (LA == LOAD_CONV_VEC || LA == LOAD_CONV_SCALAR) {
    RowInfo ri;
    const int m = m0 + t, pq = p.P * p.Q;
    const int img = m / pq, rem = m - img * pq, op = rem / p.Q, oq = rem - op * p.Q;
    ri.h0 = m < p.M ? op * p.stride_h - p.pad_t : -(1 << 28);   // rows past the last pixel fail every bounds test
    ri.w0 = oq * p.stride_w - p.pad_l;
    ri.base = (((long long)img * p.H + ri.h0) * p.W + ri.w0) * p.C;
    rows[t] = ri;
    __syncthreads();
  }
  const uint32_t sbase = smem_u32(smem);
  asm volatile("griddepcontrol.wait;" ::: "memory");   // (a no-op unless launched as a programmatic dependent)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  unsigned long long acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  auto fetch = [&](int kb, int stage) {
    if (kb < kb_hi) {
      const uint32_t a = sbase + (uint32_t)stage * (2 * kOperandBytes);
      load_a<LA>(p, a, A, rows, m0, kb);
      load_b<BVEC>(p, a + kOperandBytes, B, n0, kb);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) fetch(kb_lo + s, s);
  int stage = 0;
  for (int kb = kb_lo; kb < kb_hi; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();   // this stage has landed for every thread, and every thread is done with the stage refilled below
    fetch(kb + kStages - 1, stage == 0 ? kStages - 1 : stage - 1);
    const uint32_t a = sbase + (uint32_t)stage * (2 * kOperandBytes) + (uint32_t)(ty * 128 + (ty << 4));
    const uint32_t b = sbase + (uint32_t)stage * (2 * kOperandBytes) + kOperandBytes + (uint32_t)(tx * 128 + (tx << 4));
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t aq = a ^ (uint32_t)(q << 4), bq = b ^ (uint32_t)(q << 4);
      unsigned long long ax[8], ay[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) lds_pair(aq + (uint32_t)(i * 1024), ax[i], ay[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        unsigned long long bx, by;
        lds_pair(bq + (uint32_t)(j * 1024), bx, by);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma2(acc[i][j], ax[i], bx);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma2(acc[i][j], ay[i], by);
      }
    }
    if (++stage == kStages) stage = 0;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* out = (float*)smem;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 f = *(const float2*)&acc[i][j];
      out[(ty + 8 * i) * kPitch + tx + 8 * j] = f.x + f.y;
    }
  const Epilogue& ep = p.ep;
  const bool f32_io = !ep.mul && !ep.add_full && (!ep.res || ep.res_dt == DT_F32) && ep.out_dt == DT_F32;
  const int r_lo = kTile * rank / p.splits, r_hi = min(kTile * (rank + 1) / p.splits, p.M - m0);
  if (p.splits > 1) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  } else __syncthreads();
  if (f32_io && (p.N & 3) == 0) {
    for (int e = t; e < (r_hi - r_lo) * (kTile / 4); e += kThreads) {
      const int r = r_lo + e / (kTile / 4), c = (e % (kTile / 4)) * 4;
      if (n0 + c >= p.N) continue;
      const uint32_t at = sbase + (uint32_t)((r * kPitch + c) * 4);
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.splits == 1) v = *(const float4*)(out + r * kPitch + c);
      else
        for (int k = 0; k < p.splits; ++k) {
          uint32_t peer;
          float4 u;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(k));
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(u.x), "=f"(u.y), "=f"(u.z), "=f"(u.w) : "r"(peer) : "memory");
          v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
      finish4(p, v, (int64_t)batch * p.M + m0 + r, n0 + c);
    }
  } else {
    // One result at a time: a thread keeps its column, whose addends it reads once, and the threads that the columns leave over
    // take further rows; eight results are read before the first is finished, because the stores keep the compiler from
    // gathering the reads.
    constexpr int kAhead = 8;
    const int cols = min(kTile, p.N - n0);
    int width = 1;
    while (width < cols) width *= 2;
    const int c = t & (width - 1), col = n0 + c, step = kThreads / width;
    if (c < cols) {
      const float a1 = ep.add1 ? __ldg(ep.add1 + col) : 0.f, a2 = ep.add2 ? __ldg(ep.add2 + col) : 0.f;
      for (int r0 = r_lo + t / width; r0 < r_hi; r0 += kAhead * step) {
        float v[kAhead], res[kAhead];
        const int64_t row0 = (int64_t)batch * p.M + m0 + r0;
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const bool here = r0 + i * step < r_hi;
          v[i] = here && p.splits == 1 ? out[(r0 + i * step) * kPitch + c] : 0.f;
          res[i] = here && f32_io && ep.res ? ((const float*)ep.res)[(row0 + i * step) * p.N + col] : 0.f;
        }
        if (p.splits > 1)
          for (int k = 0; k < p.splits; ++k) {   // every result adds its parts in rank order
            uint32_t peer;
            float u[kAhead];
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(sbase + (uint32_t)((r0 * kPitch + c) * 4)), "r"(k));
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
              u[i] = 0.f;
              if (r0 + i * step < r_hi) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(u[i]) : "r"(peer + (uint32_t)(i * step * kPitch * 4)) : "memory");
            }
#pragma unroll
            for (int i = 0; i < kAhead; ++i) v[i] += u[i];
          }
        if (f32_io) {
#pragma unroll
          for (int i = 0; i < kAhead; ++i) {
            if (ep.alpha != 1.f) v[i] = __fmul_rn(v[i], ep.alpha);
            if (ep.add1) v[i] = __fadd_rn(v[i], a1);
            if (ep.add2) v[i] = __fadd_rn(v[i], a2);
          }
          if (ep.act_first) apply_act_all<kAhead>(ep.act, v, ep.act_a, ep.act_b);
          if (ep.res) {
#pragma unroll
            for (int i = 0; i < kAhead; ++i) v[i] = __fadd_rn(v[i], res[i]);
          }
          if (!ep.act_first) apply_act_all<kAhead>(ep.act, v, ep.act_a, ep.act_b);
        }
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const int64_t row = row0 + i * step;
          if (r0 + i * step >= r_hi) break;
          if (f32_io) ((float*)p.y)[row * p.N + col] = v[i];
          else store_from_float(p.y, ep.out_dt, row * p.N + col, epilogue_value(ep, v[i], row, col, p.N));
        }
      }
    }
  }
  if (p.splits > 1) {   // nobody leaves while a peer may still read its partial tile
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }
}

// Few results over a long reduction (a classifier behind a small batch): a 64 x 64 tile would leave most of its threads and
// nearly all SMs without work and walk the reduction serially, 2 us per k-block.  Here a warp owns 4 x 2 results, its lanes
// share the reduction (16-byte loads, everything from L2) and the sums meet in shuffles.  64 x 10 results over 784: 20 -> 4 us.
constexpr int kFewRows = 4, kFewCols = 2;
__global__ void __launch_bounds__(128) f32_few_results_kernel(const F32Params p) {
  const int lane = threadIdx.x & 31, col_groups = (p.N + kFewCols - 1) / kFewCols, row_groups = (p.M + kFewRows - 1) / kFewRows;
  const int64_t w = blockIdx.x * 4 + (threadIdx.x >> 5), per_batch = (int64_t)col_groups * row_groups;
  dependency_wait();
  const int64_t batch = w / per_batch, g = w - batch * per_batch;
  const int m0 = (int)(g / col_groups) * kFewRows, n0 = (int)(g % col_groups) * kFewCols;
  if (batch >= p.batches) return;
  const float *A = p.A + batch * p.a_batch, *B = p.B + batch * p.b_batch;
  float acc[kFewRows][kFewCols] = {};
#pragma unroll 4
  for (int k = lane * 4; k < p.K; k += 128) {
    float4 a[kFewRows], b[kFewCols];
#pragma unroll
    for (int i = 0; i < kFewRows; ++i) a[i] = *(const float4*)(A + (int64_t)min(m0 + i, p.M - 1) * p.a_row + k);
#pragma unroll
    for (int j = 0; j < kFewCols; ++j) b[j] = __ldg((const float4*)(B + (int64_t)min(n0 + j, p.N - 1) * p.b_col + k));
#pragma unroll
    for (int i = 0; i < kFewRows; ++i)
#pragma unroll
      for (int j = 0; j < kFewCols; ++j) {
        acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]); acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
        acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]); acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
      }
  }
  float mine = 0.f;   // lane i * kFewCols + j finishes result (i, j)
#pragma unroll
  for (int i = 0; i < kFewRows; ++i)
#pragma unroll
    for (int j = 0; j < kFewCols; ++j) {
      float v = acc[i][j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == i * kFewCols + j) mine = v;
    }
  const int m = m0 + lane / kFewCols, n = n0 + lane % kFewCols;
  if (lane < kFewRows * kFewCols && m < p.M && n < p.N) {
    const int64_t row = batch * p.M + m;
    store_from_float(p.y, p.ep.out_dt, row * p.N + n, epilogue_value(p.ep, mine, row, n, p.N));
  }
}

int device_sms() {
  static int cache[16] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return 148;
  if (!cache[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cache[dev] = n;
  }
  return cache[dev];
}
// How many CTAs share one tile's reduction: 1, 2, 4 or 8 (clusters of other sizes were 20 % slower, they pack badly).  The
// busiest SM works off its CTAs in pairs -- one CTA's two warps reach two of the four schedulers, so an odd CTA costs as
// much as two -- at 1.04 us per k-block and CTA; every round of four resident CTAs pays about 4 us for filling the stages and
// writing the tile, a cluster 2 us more for its barriers and remote reads (measured on ResNet-50's layers at batch 8).
// Of equal costs the most shares are taken, and with up to two tiles an SM the most within 15 % of the least: the count leaves out
// that more CTAs hide each other's latencies, and what costs the whole batch nothing saves a launch that computes a part of it.
// ResNet-50 of 5 images 2615 -> 1806 us (without the 15 %: 2079), in two sub-batches 2692 -> 1912; BERT of 2 x 128: 3328 -> 2461 and
// 3129 -> 2415.  With more tiles 15 % lose: 736 tiles of 32 k-blocks 164 -> 183 us.
// `tiles` are those of the whole recorded batch: the number of shares is the order of the sums, and a launch that computes a
// part of the batch (another GPU's or sub-batch's rows) has to take the same one.
struct Splits { int n; double us; };
Splits pick_splits(int64_t tiles, int num_kb) {
  const int sms = device_sms();
  auto cost = [&](int n) {
    const int64_t per_sm = (tiles * n + sms - 1) / sms;
    return (double)((per_sm + 1) / 2 * 2) * ((num_kb + n - 1) / n) * 1.04 + (double)((per_sm + 3) / 4) * 4.0 + (n > 1 ? 2.0 : 0.0);
  };
  double least = cost(1);
  for (int n = 2; n <= 8 && n <= num_kb; n *= 2) least = std::min(least, cost(n));
  int most = 1;
  for (int n = 2; n <= 8 && n <= num_kb; n *= 2)
    if (cost(n) <= (tiles <= 2 * sms ? 1.15 : 1.0) * least) most = n;
  return {most, least};
}
// Whether a short reduction over few or narrow results is better off on the one-thread-per-output kernel, which has nothing to
// set up.  In us, fitted to 630 shapes (1 to 256 columns, 4 to 2048 values, 16 to 131072 rows; convolutions of 1 to 64 channels
// with 1x1 to 7x7 windows of 8 x 8 to 16 x 56 x 56 pixels), each launch bracketed: the tiles as pick_splits counts them and 5, 4-byte loads 1.35
// times; one thread per output 85 ns a value and 250 ns a tap until the chip is full, then a throughput per result and value.
// The fit is within a quarter on either side for most, so the tiles keep whatever is close.  131072 x 2 results of 10 values: 33 us on tiles, 9 on
// threads; 3x3 of 16 x 56 x 56 x 5 -> 1: 30 and 10; 16384 x 64 results of 16 values: 14 and 18.  Sums of up to 256 values in one chain only:
// beyond, the tiles are both faster and more exact.
bool direct_pays(int64_t M, int64_t N, int64_t K, int taps, bool wide_loads) {
  if (K > 256) return false;
  const double tiles = 5.0 + pick_splits((M + kTile - 1) / kTile * ((N + kTile - 1) / kTile), (int)((K + kBK - 1) / kBK)).us * (wide_loads ? 1.0 : 1.35);
  const double results = (double)M * N, chain = 1.0 + 0.085 * K + (taps > 1 ? 0.25 * taps : 0.0);
  const double rate = taps ? results * (12e-6 + (taps > 1 ? 1.7e-6 * taps : 0.0) + 3.4e-7 * K) : results * (8e-6 + 3.4e-7 * K) + 1.5e-6 * M * K;
  return 6.0 + std::max(chain, rate) < 0.9 * tiles;
}
// Up to this many results (of the whole recorded batch, see pick_splits) the warps of one launch fit the chip at once and the
// operands are re-read from L2 only.
constexpr int64_t kFewResults = 16384;
template <int LA, bool BVEC>
int launch_tiles(const F32Params& p, int64_t blocks, cudaStream_t s) {
  static bool set[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !set[dev]) {
    if (cudaFuncSetAttribute(f32_tile_kernel<LA, BVEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) { cudaGetLastError(); return -2; }
    if (dev >= 0 && dev < 16) set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks, 1, (unsigned)p.splits);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  static const bool pdl = !getenv("ODLA_B200_NO_PDL");
  int na = 0;
  if (pdl) { attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[na].val.programmaticStreamSerializationAllowed = 1; ++na; }
  if (p.splits > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = (unsigned)p.splits;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, f32_tile_kernel<LA, BVEC>, p);
  if (e != cudaSuccess) { fprintf(stderr, "[odla_b200] fp32 tile kernel launch failed: %s\n", cudaGetErrorString(e)); cudaGetLastError(); return -2; }
  return 0;
}
int run(F32Params p, int la, bool bvec, int64_t batch, int64_t batch_full, int64_t rows_full, cudaStream_t s) {
  p.num_kb = (p.K + kBK - 1) / kBK;
  p.m_tiles = (p.M + kTile - 1) / kTile;
  p.n_tiles = (p.N + kTile - 1) / kTile;
  const int64_t tiles = batch * p.m_tiles * p.n_tiles;
  if (tiles <= 0) return 0;
  p.splits = pick_splits(batch_full * ((rows_full + kTile - 1) / kTile) * p.n_tiles, p.num_kb).n;
  if (la == LOAD_CONV_VEC) return launch_tiles<LOAD_CONV_VEC, true>(p, tiles, s);
  if (la == LOAD_CONV_SCALAR) return launch_tiles<LOAD_CONV_SCALAR, true>(p, tiles, s);
  if (la == LOAD_GEMM_VEC) return bvec ? launch_tiles<LOAD_GEMM_VEC, true>(p, tiles, s) : launch_tiles<LOAD_GEMM_VEC, false>(p, tiles, s);
  return bvec ? launch_tiles<LOAD_GEMM_SCALAR, true>(p, tiles, s) : launch_tiles<LOAD_GEMM_SCALAR, false>(p, tiles, s);
}
// What the kernels' 32-bit indices can address: rows and columns of the last tile included, and one block per tile.
bool indexable(int64_t batch, int64_t M, int64_t N, int64_t K) {
  const int64_t most = (1ll << 31) - kTile;
  return M < most && N < most && K < (1ll << 30) && batch < (1ll << 31) && (double)batch * ((M + kTile - 1) / kTile) * ((N + kTile - 1) / kTile) < 2147483648.0;
}
}  // namespace

bool conv_f32_supported(const ConvGeom& g) {
  return g.groups == 1 && g.xs_c == 1 && g.P > 0 && g.Q > 0 && indexable(1, (int64_t)g.N * g.P * g.Q, g.K, (int64_t)g.R * g.S * g.C);
}
bool conv_f32_pays(const ConvGeom& g, int64_t images_full) { return !direct_pays(images_full * g.P * g.Q, g.K, (int64_t)g.R * g.S * g.C, g.R * g.S, g.C % 4 == 0); }
int conv_f32(const ConvGeom& g, int64_t images_full, const void* x, const void* w, int64_t w_pitch, void* y, const Epilogue& ep, cudaStream_t s) {
  F32Params p{};
  p.M = g.N * g.P * g.Q; p.N = g.K; p.K = g.R * g.S * g.C;
  p.H = g.H; p.W = g.W; p.C = g.C; p.R = g.R; p.S = g.S; p.P = g.P; p.Q = g.Q;
  p.stride_h = g.stride_h; p.stride_w = g.stride_w; p.pad_t = g.pad_t; p.pad_l = g.pad_l;
  p.A = (const float*)x; p.B = (const float*)w; p.y = y; p.ep = ep;
  p.b_row = 1; p.b_col = w_pitch;
  const bool vec = g.C % 4 == 0 && (uintptr_t)x % 16 == 0;
  return run(p, vec ? LOAD_CONV_VEC : LOAD_CONV_SCALAR, true, 1, 1, images_full * g.P * g.Q, s);
}
bool gemm_f32_supported(const GemmGeom& g) { return g.K > 0 && indexable(g.batch, g.M, g.N, g.K); }
bool gemm_f32_pays(const GemmGeom& g, int64_t batch_full, int64_t rows_full, bool b_kmajor) {
  const bool wide = g.a_col == 1 && b_kmajor && g.K % 4 == 0;
  if (batch_full > 1 || (wide && rows_full * g.N <= kFewResults)) return true;
  return !direct_pays(rows_full, g.N, g.K, 0, wide);
}
int gemm_f32(const GemmGeom& g, int64_t batch_full, int64_t rows_full, const void* A, const void* B, void* C, const Epilogue& ep, cudaStream_t s) {
  if (g.batch <= 0 || g.M <= 0 || g.N <= 0) return 0;
  F32Params p{};
  p.M = (int)g.M; p.N = (int)g.N; p.K = (int)g.K;
  p.a_row = g.a_row; p.a_col = g.a_col; p.a_batch = g.a_batch;
  p.b_row = g.b_row; p.b_col = g.b_col; p.b_batch = g.b_batch;
  p.A = (const float*)A; p.B = (const float*)B; p.y = C; p.ep = ep;
  const bool avec = g.a_col == 1 && g.K % 4 == 0 && g.a_row % 4 == 0 && g.a_batch % 4 == 0 && (uintptr_t)A % 16 == 0;
  // (pieces past K are zero on the A side, so a B row padded to a multiple of four floats may hold anything there)
  const bool bvec = g.b_row == 1 && g.b_col % 4 == 0 && (g.K % 4 == 0 || g.b_batch == 0) && g.b_batch % 4 == 0 && (uintptr_t)B % 16 == 0;
  if (avec && bvec && g.K % 4 == 0 && batch_full * rows_full * g.N <= kFewResults) {
    p.batches = (int)g.batch;
    const int64_t warps = g.batch * ((g.M + kFewRows - 1) / kFewRows) * ((g.N + kFewCols - 1) / kFewCols);
    b200::launch(f32_few_results_kernel, (unsigned)((warps + 3) / 4), 128, 0, s, p);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
  }
  return run(p, avec ? LOAD_GEMM_VEC : LOAD_GEMM_SCALAR, bvec, g.batch, batch_full, rows_full, s);
}

}  // namespace b200
