// Depth-only attention (parallel_fda, fda_v12.py:1346) as HBM-bandwidth kernels.
//
// Each query position attends only to the L depth K/V rows of its own position, so the
// operator moves 2*L*D elements per position for 4*G*L*D flops: about G flops per byte.  The
// attention-tile pipeline (128-row tiles) would multiply every query against the depth rows of 127
// other positions; here one warp owns one (batch, position, head) - a unit - and writes o / lse
// (forward) or dq, d_depth_k, d_depth_v (backward; rows are owner-exclusive, no atomics).
// Numerics as in the other kernels: scores scaled by scale*log2(e), exp2, lse = m + log2(l),
// delta from the stored o, dq and dk scaled by `scale` at the end.
//
// A unit's K/V rows are a few KB (11 rows of 128 bytes in a vision transformer), so two things
// bound such a kernel before HBM does: the instructions of a unit, and the time between a unit's
// loads and its last store.
//  * Instructions: the up to 8 query rows of a position are columns of m16n8k16 matrix instructions.
//    Per 16 depth rows that replaces 16 fp32 FMAs for every 16 bytes of K or V and query row, and
//    the reductions over the lanes of a row.
//  * Latency: every warp has two shared-memory stages of 16 K rows + 16 V rows (and the query rows of
//    its units), so that the loads of the next step, usually another unit's, are under way while
//    this one is computed.  TMA fills them: one lane, three to seven instructions a step and hardly
//    any address arithmetic (filled by 16-byte cp.async, a unit of 11 rows of D = 64 took 740
//    instructions, as many as on fp32 FMAs).  The backward's gradient rows take the place of the K
//    and V rows of their stage and leave by TMA too.
// Against the fp32-FMA kernels these replace: B = 256, T = 197, H = 6, D = 64, L = 11: forward 0.356 ->
// 0.166 ms, backward 0.479 -> 0.312 ms (6.0 of the measured 6.5 TB/s copy bandwidth); D = 128, L = 32, G = 1 (53 GB):
// 8.53 -> 7.93 ms; B = 2, T = 4093, H = 4, G = 4, D = 128, L = 24: 0.241 -> 0.077 ms and, against the
// attention-tile mma.sync kernels, 0.520 -> 0.150 ms.
//
// Lane layout: g = lane >> 2, t = lane & 3.  A chunk is 16 bytes = 8 channels of a row.
//  * K (and q, dO; V for dO V^T): lane (g, t) takes chunks t, t + 4, .. of row g.  Word w of chunk
//    t + 4 j is the operand of k-step (j, w >> 1): the channels a k-step contracts are permuted the
//    same way in both operands, which a sum does not see.
//  * V (for P V; K for dS K): lane (g, t) takes chunks g, g + 8, .. of four rows; byte permutations of
//    two of them make the operand of a channel with the depth rows as the contracted index.
//  * An 8 x 8 transpose (movmatrix) of the words of the first layout gives the right operand with
//    the query rows as the contracted index, for channels 32 j + 8 t + 2 w, + 1 of the result: a lane's
//    results of the four words are one 16-byte chunk.
// P and dS enter as the sum of 16-bit numbers, so that what they have beyond 16 bits is not lost: three
// (split3), which hold all 24 bits of the fp32 value, or in the backward at G > 4 two (split2, 2^-18
// relative for bf16); in fp16, whose range is smaller, after a power of two has been taken out
// (Scaled).  With up to four query rows the parts take the other four columns (rows, where the queries
// are the contracted index) of the same instructions: query q has columns 2 q, 2 q + 1, whose scores
// come out twice, and the results of the two are added in the end.  Scores are summed in fp32 outside
// the matrix unit, which cuts its running sum at every step.
// Against 64 bits (q of 1/4, 1 and 4, dO of 1e-5..64, L = 1..64, G = 1..8, both head dims) the errors of o, dq, dk
// and dv are then those of the fp32-FMA kernels to 1e-5 of themselves, and values that are not the rounded
// exact one as few (o in bf16 1.0e-4, 1.2e-4 with FMAs); lse errs by 4.5e-8 (bf16) and 5.0e-8 (fp16), 5.0e-8
// and 4.9e-8 with FMAs.  (Two parts for all and sums in the matrix unit: 1.4e-3 of o; in fp16 gradients of dO =
// 1e-5 up to eight times the error, and NaN where scale dS passed 65504.)
#pragma once
#include "common.cuh"
#include "simt_mma_kernels.cuh"
#include "tc_bwd_kernels.cuh"

namespace moda {
namespace fda {

constexpr int kWarps = 4;             // warps of a block: they share nothing but the launch
constexpr int kRows = 16;             // depth rows of a stage

template <typename T> __device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const float2 a = Pack<T>::unpack(u.x), b = Pack<T>::unpack(u.y), c = Pack<T>::unpack(u.z), d = Pack<T>::unpack(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
// f += the eight stored 16-bit values of u
template <typename T> __device__ __forceinline__ void add8(float (&f)[8], const uint4& u) {
  float g[8];
  unpack8<T>(u, g);
#pragma unroll
  for (int e = 0; e < 8; ++e) f[e] += g[e];
}
template <typename T> __device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(Pack<T>::pack(f[0], f[1]), Pack<T>::pack(f[2], f[3]), Pack<T>::pack(f[4], f[5]), Pack<T>::pack(f[6], f[7]));
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
// (a, b) cut to 16 bits each.
template <typename T> __device__ __forceinline__ uint32_t cut_pair(float a, float b);
template <> __device__ __forceinline__ uint32_t cut_pair<__nv_bfloat16>(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632u);
}
template <> __device__ __forceinline__ uint32_t cut_pair<__half>(float a, float b) {
  uint32_t w;
  asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(b), "f"(a));
  return w;
}
// (a, b) as the sum of three 16-bit pairs: the value cut to 8 (bf16) or 11 (fp16) bits, what that left over cut
// again, and the rest.  2^-30 of the value keeps the later parts from being zero, which have the sign of
// the first one, so that P V is infinite, and not NaN, where a row of V is.
template <typename T> __device__ __forceinline__ void split3(float a, float b, uint32_t (&w)[3]) {
  constexpr float kKeep = 0x1p-30f;
  w[0] = cut_pair<T>(a, b);
  const float2 x = Pack<T>::unpack(w[0]);
  const float a1 = fmaf(a, kKeep, a - x.x), b1 = fmaf(b, kKeep, b - x.y);
  w[1] = cut_pair<T>(a1, b1);
  const float2 y = Pack<T>::unpack(w[1]);
  w[2] = cut_pair<T>(fmaf(a, kKeep, a1 - y.x), fmaf(b, kKeep, b1 - y.y));
}
// (a, b) rounded to 16 bits, and what the rounding left over.
template <typename T> __device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = Pack<T>::pack(a, b);
  const float2 h = Pack<T>::unpack(hi);
  lo = Pack<T>::pack(a - h.x, b - h.y);
}
// At most four query rows, contracted index = depth rows: the operand words of a pair of them.  The first column of
// a query holds parts 0 and 2, its second part 1 and nothing more (2^-30, as above).
template <typename T> __device__ __forceinline__ void split3_columns(float a, float b, bool second, uint32_t& w0, uint32_t& w1) {
  uint32_t w[3];
  split3<T>(a, b, w);
  w0 = second ? w[1] : w[0];
  w1 = second ? cut_pair<T>(a * 0x1p-30f, b * 0x1p-30f) : w[2];
}
// The same, contracted index = queries: the words of one query's two indexes.
template <typename T> __device__ __forceinline__ float cut(float a) { return Pack<T>::unpack(cut_pair<T>(a, 0.f)).x; }
template <typename T> __device__ __forceinline__ void split3_rows(float a, uint32_t& w0, uint32_t& w1) {
  const float h = cut<T>(a), r = a - h, m = cut<T>(r);
  w0 = cut_pair<T>(h, m);
  w1 = cut_pair<T>(r - m, 0.f);
}
// What a fp16 operand holds of fp32 values: those of a warp's step times the power of two that takes their
// largest magnitude to [2^14, 2^15), so that none overflows and the smallest step left is 2^-38 of the
// largest (times 65504 that is less than the smallest fp16 result).  bf16 has the range of fp32.
template <typename T> struct Scaled {
  float up = 1.f, down = 1.f;
  static constexpr bool kUsed = std::is_same<T, __half>::value;
  __device__ __forceinline__ Scaled(float a, float b, float c, float d) {
    if constexpr (kUsed) {
      const float m = fmaxf(fmaxf(fabsf(a), fabsf(b)), fmaxf(fabsf(c), fabsf(d)));
      const uint32_t e = min(240u, 268u - (__reduce_max_sync(0xffffffffu, __float_as_uint(m)) >> 23));
      up = __uint_as_float(e << 23);
      down = __uint_as_float((254u - e) << 23);
    }
  }
};
constexpr float kUpP = 0x1p15f, kDownP = 0x1p-15f;     // the same for probabilities, which are at most 1
template <typename T> __device__ __forceinline__ constexpr float up_p() { return Scaled<T>::kUsed ? kUpP : 1.f; }
template <typename T> __device__ __forceinline__ constexpr float down_p() { return Scaled<T>::kUsed ? kDownP : 1.f; }
__device__ __forceinline__ float quad_sum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  return x + __shfl_xor_sync(0xffffffffu, x, 2);
}

// Rows of a stage are permuted so that both ways of reading it are free of bank conflicts under the
// TMA unit's 128-byte swizzle (chunk c of row r sits at chunk c ^ (r & 7)): column 2 t + e of matrix
// operand nt is tile row 8 nt + row_of(t, e).  Two lanes of a K access then differ in bit 2 of the row,
// the four rows of a V access (same e) in bits 1 and 2.
__device__ __forceinline__ int row_of(int t, int e) {
  // t: 0 1 2 3 -> e = 0: 0 2 5 7, e = 1: 4 6 1 3
  return (2 * t + (t >> 1)) ^ (e << 2);
}
// 16-byte chunk c of row r of a tile of 64-channel boxes of `rows` rows each
template <int ROWS> __device__ __forceinline__ uint32_t chunk_at(int r, int c) { return (c >> 3) * (ROWS * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4); }
template <int ROWS> __device__ __forceinline__ uint4 tile_chunk(const unsigned char* tile, int r, int c) {
  return *reinterpret_cast<const uint4*>(tile + chunk_at<ROWS>(r, c));
}

// One step of a warp: a block of 16 depth rows of a unit, for query rows [g0, g0 + 8) of its position.
// Units are numbered h-fastest; a warp takes every (warps of the grid)-th one, and the step from one to
// the next is an addition with carries (a division costs more than the rest of the bookkeeping).
struct Step { int b, t, h, l0, g0; };
struct Stride {
  int b, t, h;
  __device__ __forceinline__ Stride(const Params& p, unsigned n) {
    h = (int)(n % (unsigned)p.H);
    n /= (unsigned)p.H;
    t = (int)(n % (unsigned)p.T_kv);
    b = (int)(n / (unsigned)p.T_kv);
  }
  __device__ __forceinline__ void advance(const Params& p, Step& s) const {
    s.l0 += kRows;
    if (s.l0 < p.L) return;
    s.l0 = 0;
    s.g0 += 8;
    if (s.g0 < p.G) return;
    s.g0 = 0;
    s.h += h;
    if (s.h >= p.H) { s.h -= p.H; ++s.t; }
    s.t += t;
    if (s.t >= p.T_kv) { s.t -= p.T_kv; ++s.b; }
    s.b += b;
  }
};

__device__ __forceinline__ Step first_step(const Params& p) {
  const Stride at(p, blockIdx.x * kWarps + (threadIdx.x >> 5));
  return Step{at.b, at.t, at.h, 0, 0};
}

// k, v: boxes of 16 depth rows x 64 channels; kt, vt: of the L % 16 rows of a unit's last block, so that
// nothing of the next position (or of a cache's unwritten layers) is read.  q, dout, o: the query
// rows of a position (8 of them at most), unswizzled.
struct Maps { CUtensorMap k, v, kt, vt, q, dout, o; };
struct OutMaps { CUtensorMap dk, dv, dkt, dvt; };     // the same boxes of the depth gradients

// Shared memory of a block: per warp two stages {K tile, V tile} (NT = 2) or {K, V, dK, dV} (NT = 4: gradients
// that are added to); per warp one group of the query rows of q (NQ = 1) or q, dout, o (NQ = 3); per
// warp two mbarriers; the abort words.
template <int D> __host__ __device__ constexpr uint32_t tile_bytes() { return kRows * 2 * D; }
// Tiles of a backward stage.  Gradients to add to are in HBM like K and V, and loaded where they are
// added they stall the warp once a step; at D = 64 they are tiles of the ring.  At D = 128 that would
// leave one block an SM, and they are loaded row by row.  B = 64, T = 197, H = 6, D = 64: eleven calls of L = 1..11
// layers 1.33 -> 1.02 ms, fifteen of 1..15 2.04 -> 1.56 ms.
template <int D, bool kAdd> __host__ __device__ constexpr int bwd_tiles() { return kAdd && D == 64 ? 4 : 2; }
template <int D, int NQ, int NT = 2> __host__ __device__ constexpr uint32_t smem_bytes(int G) {
  return kWarps * (2 * NT * tile_bytes<D>() + NQ * (G < 8 ? G : 8) * 2 * D + 16) + 16;
}

// The ring of one warp.
template <int D, int NQ, int NT = 2>
struct Ring {
  static constexpr uint32_t kStage = NT * tile_bytes<D>();
  unsigned char *tiles, *queries;
  uint32_t bars;
  volatile int* abort_flag;
  int issued = 0, taken = 0;           // steps issued / taken so far
  bool failed;                         // the call has, before this block began
  __device__ __forceinline__ Ring(const Params& p, unsigned char* smem) {
    const int w = threadIdx.x >> 5;
    const uint32_t q_bytes = NQ * min(p.G, 8) * 2 * D;
    tiles = smem + w * 2 * kStage;
    queries = smem + kWarps * 2 * kStage + w * q_bytes;
    unsigned char* ctl = smem + kWarps * (2 * kStage + q_bytes);
    bars = smem_u32(ctl) + w * 16;
    abort_flag = reinterpret_cast<volatile int*>(ctl + kWarps * 16);     // abort, drain
    if (threadIdx.x == 0) { abort_flag[0] = 0; abort_flag[1] = tc::failure_seen(p) ? 1 : 0; }
    if ((threadIdx.x & 31) == 0) {
      tc::mbar_init(bars, 1);
      tc::mbar_init(bars + 8, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    failed = abort_flag[1] != 0;
  }
  // Loads of step s; a unit's first step brings the query rows.
  __device__ __forceinline__ void issue(const Params& p, const Maps& maps, const OutMaps* grads, const Step& s) {
    if (tc::elect_one()) {
      const int n = min(p.L - s.l0, kRows), row = s.t * p.Ls + s.l0;
      const uint32_t bar = bars + 8 * (issued & 1), dst = smem_u32(tiles) + (issued & 1) * kStage;
      const uint32_t q_rows = min(p.G, 8) * 2 * D;
      tc::mbar_expect_tx(bar, n * NT * 2 * D + (s.l0 == 0 ? NQ * q_rows : 0));
      tc::tma_load_tile<D>(dst, n == kRows ? &maps.k : &maps.kt, bar, kRows * 128, s.h, row, s.b);
      tc::tma_load_tile<D>(dst + tile_bytes<D>(), n == kRows ? &maps.v : &maps.vt, bar, kRows * 128, s.h, row, s.b);
      if constexpr (NT == 4) {
        tc::tma_load_tile<D>(dst + 2 * tile_bytes<D>(), n == kRows ? &grads->dk : &grads->dkt, bar, kRows * 128, s.h, row, s.b);
        tc::tma_load_tile<D>(dst + 3 * tile_bytes<D>(), n == kRows ? &grads->dv : &grads->dvt, bar, kRows * 128, s.h, row, s.b);
      }
      if (s.l0 == 0) {
        const int r = s.t * p.G + s.g0;
        tc::tma_load_4d(smem_u32(queries), &maps.q, bar, 0, s.h, r, s.b);
        if constexpr (NQ == 3) {
          tc::tma_load_4d(smem_u32(queries) + q_rows, &maps.dout, bar, 0, s.h, r, s.b);
          tc::tma_load_4d(smem_u32(queries) + 2 * q_rows, &maps.o, bar, 0, s.h, r, s.b);
        }
      }
    }
    __syncwarp();
    ++issued;
  }
  // Waits for the next step's rows; false: the wait expired (bounded, as everywhere).
  __device__ __forceinline__ bool wait() {
    const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(bars + 8 * (taken & 1), (taken >> 1) & 1, abort_flag, 30));
    ++taken;
    return ok;
  }
  // The stage of the current step, which now holds gradient rows, to memory; the lane that stores is the
  // one that waits (stored_read) before the stage is filled again.
  __device__ __forceinline__ void store(const Params& p, const OutMaps& maps, const Step& s) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (tc::elect_one()) {
      const bool full = p.L - s.l0 >= kRows;
      const uint32_t src = smem_u32(tiles) + ((taken - 1) & 1) * kStage;
      const int row = s.t * p.Ls + s.l0;
#pragma unroll
      for (int bx = 0; bx < D / 64; ++bx) {
        tc::tma_store_4d(full ? &maps.dk : &maps.dkt, src + bx * kRows * 128, 64 * bx, s.h, row, s.b);
        tc::tma_store_4d(full ? &maps.dv : &maps.dvt, src + tile_bytes<D>() + bx * kRows * 128, 64 * bx, s.h, row, s.b);
      }
      tc::bulk_commit();
    }
    __syncwarp();
  }
  __device__ __forceinline__ void stored_read() {
    if (tc::elect_one()) tc::bulk_wait_read_all();
    __syncwarp();
  }
  // After a failed wait: loads in flight land before the shared memory is given up.
  __device__ __forceinline__ void drain() {
    for (int i = taken - 1; i < issued; ++i) tc::mbar_wait(bars + 8 * (i & 1), (i >> 1) & 1, abort_flag + 1, 30);
  }
  __device__ __forceinline__ const unsigned char* stage() const { return tiles + ((taken - 1) & 1) * kStage; }
};
template <int D> __device__ __forceinline__ uint4 query_chunk(const unsigned char* rows, int r, int c) {
  return *reinterpret_cast<const uint4*>(rows + r * 2 * D + c * 16);
}

// acc[i] += (rows of `tile`)^T x: for 64 channels of a tile (box i) the 8 channels of chunk g as left
// operands, each made from the tile rows of operand columns 2 t, 2 t + 1 (+ 8), and the N parts of x
// as right operands, x = their sum times `down`.  Result [e][c]: channel 8 g + e of query 2 t + c.
// `left` rows of the tile exist (kAll: all, or the others are zeros).
template <typename T, bool kAll, bool kScaled, int N>
__device__ __forceinline__ void add_transposed(float (&acc)[8][2], const unsigned char* tile, int i, int g, int t4, int left,
                                               const uint32_t (&x0)[N], const uint32_t (&x1)[N], float down) {
  uint32_t w[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x) {                     // a row that does not exist is whatever the stage held before
    const int r = 8 * (x >> 1) + row_of(t4, x & 1);
    const uint4 v4 = kAll || r < left ? tile_chunk<kRows>(tile, r, g + 8 * i) : make_uint4(0, 0, 0, 0);
    w[x][0] = v4.x; w[x][1] = v4.y; w[x][2] = v4.z; w[x][3] = v4.w;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {                     // channels 2 e (rows g of the operand) and 2 e + 1 (rows g + 8)
    const uint32_t a[4] = {__byte_perm(w[0][e], w[1][e], 0x5410u), __byte_perm(w[0][e], w[1][e], 0x7632u),
                           __byte_perm(w[2][e], w[3][e], 0x5410u), __byte_perm(w[2][e], w[3][e], 0x7632u)};
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    if (!kScaled) { c[0] = acc[2 * e][0]; c[1] = acc[2 * e][1]; c[2] = acc[2 * e + 1][0]; c[3] = acc[2 * e + 1][1]; }
#pragma unroll
    for (int part = N - 1; part >= 0; --part) simt::Mma<T>::run(c, a, x0[part], x1[part]);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      float& r = acc[2 * e + (x >> 1)][x & 1];
      r = kScaled ? fmaf(c[x], down, r) : c[x];
    }
  }
}

// kOne: L <= 16, a unit is one step.  The rows of a stage that no unit fills are then zeroed once, the
// probabilities are normalised before P V, and nothing is carried from step to step.
template <int D, int NQ, int NT> __device__ __forceinline__ void zero_tiles(const Ring<D, NQ, NT>& ring) {
  for (uint32_t i = (threadIdx.x & 31) * 16; i < 2 * ring.kStage; i += 32 * 16) *reinterpret_cast<uint4*>(ring.tiles + i) = make_uint4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // before the TMA unit writes there
  __syncwarp();
}

// ------------------------------------------------------------------------- forward
// QR: query rows that a step has columns for, 4 (G <= 4) or 8.
template <typename T, int D, bool kOne, int QR>
__global__ void __launch_bounds__(kWarps * 32, D == 64 ? (kOne ? 6 : 5) : 3) fwd_kernel(const __grid_constant__ Params p, const __grid_constant__ Maps maps) {
  constexpr int J = D / 32, I = D / 64;
  extern __shared__ __align__(1024) unsigned char smem[];
  if (smem_u32(smem) & 1023u) {                     // the swizzle is a function of the shared-memory address
    if (threadIdx.x == 0) tc::record_failure(2 << 8);
    return;
  }
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int my_row = row_of(g >> 1, g & 1);         // tile row (+ 8 nt) of this lane's K operand
  const int my_q = QR == 4 ? g >> 1 : g;            // query of this lane's scores
  Ring<D, 1> ring(p, smem);
  if (ring.failed) return;
  if (kOne) zero_tiles(ring);
  const Stride stride(p, gridDim.x * kWarps);
  Step s = first_step(p);
  if (s.b < p.B) ring.issue(p, maps, nullptr, s);
  uint4 qa[J];
  float m = -INFINITY, lsum = 0.f;
  float acc[I][8][2];                               // [channel 8 (g + 8 i) + e][query 2 t + c]
  bool ok = true;
  while (s.b < p.B) {
    Step next = s;
    stride.advance(p, next);
    if (!(ok = ring.wait())) break;
    const int n_rows = p.G - s.g0;                  // query rows of the step (8 or more: 8)
    const bool first = kOne || s.l0 == 0;
    if (first) {
#pragma unroll
      for (int j = 0; j < J; ++j) qa[j] = my_q < n_rows ? query_chunk<D>(ring.queries, my_q, t4 + 4 * j) : make_uint4(0, 0, 0, 0);
    }
    __syncwarp();                                   // the other stage and the query rows have been read
    if (next.b < p.B) ring.issue(p, maps, nullptr, next);
    const unsigned char *kt = ring.stage(), *vt = kt + tile_bytes<D>();
    const int left = p.L - s.l0;                    // rows of the tile that exist (16 or more: all)

    float pv[4];                                    // scores of my_q; columns 2 t, 2 t + 1, 8 + 2 t, 8 + 2 t + 1
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const uint4 kw = tile_chunk<kRows>(kt, 8 * nt + my_row, t4 + 4 * j);
        const uint32_t a0[4] = {qa[j].x, 0u, qa[j].y, 0u}, a1[4] = {qa[j].z, 0u, qa[j].w, 0u};
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};           // [2], [3] stay 0
        simt::Mma<T>::run(s0, a0, kw.x, kw.y);
        simt::Mma<T>::run(s1, a1, kw.z, kw.w);
        pv[2 * nt] = j == 0 ? s0[0] + s1[0] : pv[2 * nt] + (s0[0] + s1[0]);
        pv[2 * nt + 1] = j == 0 ? s0[1] + s1[1] : pv[2 * nt + 1] + (s0[1] + s1[1]);
      }
    }
    float bm = -INFINITY;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      pv[x] = 8 * (x >> 1) + row_of(t4, x & 1) < left ? pv[x] * p.scale_log2 : -INFINITY;
      bm = fmaxf(bm, pv[x]);
    }
    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 2));
    const float m_old = m;
    m = first ? bm : fmaxf(m, bm);                  // finite: the first row of a block always exists
#pragma unroll
    for (int x = 0; x < 4; ++x) pv[x] = fast_exp2(pv[x] - m);      // 0 for rows that do not exist
    const float part = (pv[0] + pv[1]) + (pv[2] + pv[3]);
    float total = 0.f;
    if (kOne) {
      total = quad_sum(part);
      const float inv = up_p<T>() / total;
#pragma unroll
      for (int x = 0; x < 4; ++x) pv[x] *= inv;
    }
    if (first) {
      lsum = part;
#pragma unroll
      for (int i = 0; i < I; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[i][e][0] = acc[i][e][1] = 0.f;
    } else {
      const float alpha = fast_exp2(m_old - m);
      lsum = fmaf(lsum, alpha, part);
      const float a0 = __shfl_sync(0xffffffffu, alpha, 8 * t4), a1 = __shfl_sync(0xffffffffu, alpha, 8 * t4 + 4);   // queries 2 t, 2 t + 1
#pragma unroll
      for (int i = 0; i < I; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) { acc[i][e][0] *= a0; acc[i][e][1] *= a1; }
    }
    if (!kOne && Scaled<T>::kUsed) {
#pragma unroll
      for (int x = 0; x < 4; ++x) pv[x] *= kUpP;
    }
    constexpr int N = QR == 4 ? 2 : 3;
    uint32_t p0[N], p1[N];
    if constexpr (QR == 4) {
      split3_columns<T>(pv[0], pv[1], g & 1, p0[0], p0[1]);
      split3_columns<T>(pv[2], pv[3], g & 1, p1[0], p1[1]);
    } else {
      split3<T>(pv[0], pv[1], p0);
      split3<T>(pv[2], pv[3], p1);
    }
#pragma unroll
    for (int i = 0; i < I; ++i) add_transposed<T, kOne, false>(acc[i], vt, i, g, t4, left, p0, p1, 1.f);

    if (kOne || left <= kRows) {
      const int r = s.t * p.G + s.g0;
      float inv[2] = {1.f, 1.f};
      if (!kOne) {
        total = quad_sum(lsum);
        const float v = down_p<T>() / total;
        inv[0] = __shfl_sync(0xffffffffu, v, 8 * t4);
        inv[1] = __shfl_sync(0xffffffffu, v, 8 * t4 + 4);
      }
      constexpr int NC = QR == 4 ? 1 : 2;           // query rows that a lane ends with
      T* op = reinterpret_cast<T*>(p.o.ptr) + p.o.off(s.b, r + NC * t4, s.h) + 8 * g;
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (NC * t4 + c < n_rows)
#pragma unroll
          for (int i = 0; i < I; ++i) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = (QR == 4 ? acc[i][e][0] + acc[i][e][1] : acc[i][e][c]) * (kOne ? down_p<T>() : inv[c]);
            *reinterpret_cast<uint4*>(op + c * p.o.st + 64 * i) = pack8<T>(f);
          }
      if (t4 == 0 && my_q < n_rows && (QR == 8 || (g & 1) == 0)) p.lse[((int64_t)s.b * p.T_q + r + my_q) * p.H + s.h] = m + log2f(total);
    }
    s = next;
  }
  if (!ok) {
    ring.drain();
    tc::publish_failure(p, ring.abort_flag);
  }
}

// ------------------------------------------------------------------------- backward
// G <= 8: the query rows of a position are one group.  Scores are computed transposed (K as the left
// operand: 16 depth rows at once), so that P^T and dS^T are left operands of dV = P^T dO and
// dK = dS^T Q as they come.
template <typename T, int D, bool kOne, bool kAdd, int QR>
__global__ void __launch_bounds__(kWarps * 32, D == 64 ? (kAdd ? 3 : 4) : 3) bwd_kernel(const __grid_constant__ Params p, const __grid_constant__ Maps maps, const __grid_constant__ OutMaps omaps) {
  constexpr int J = D / 32, I = D / 64;
  extern __shared__ __align__(1024) unsigned char smem[];
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0) tc::record_failure(2 << 8);
    return;
  }
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int my_row = row_of(g >> 1, g & 1);         // tile row (+ 8) of this lane's operands and results
  constexpr int NC = QR == 4 ? 1 : 2;               // queries of a lane's two columns
  const int my_q = QR == 4 ? g >> 1 : g, q0 = NC * t4;       // query of this lane's rows; first query of its columns
  const bool row_ok = my_q < p.G;
  constexpr int NT = bwd_tiles<D, kAdd>();
  Ring<D, 3, NT> ring(p, smem);
  if (ring.failed) return;
  if (kOne) zero_tiles(ring);
  const Stride stride(p, gridDim.x * kWarps);
  Step s = first_step(p);
  uint4 qa[J], da[J];
  float delta[2] = {0.f, 0.f}, lse[2] = {0.f, 0.f};          // of queries q0 (NC = 2: and q0 + 1)
  float lse_next[2] = {INFINITY, INFINITY};                  // P of a query that does not exist: exp2(-inf) = 0
  float dq[I][8][2];                                         // [channel 8 (g + 8 i) + e][query 2 t + c]
  bool ok = true;
  auto issue = [&](const Step& x) {
    ring.issue(p, maps, &omaps, x);
    if (kOne || x.l0 == 0) {
      const float* l = p.lse + ((int64_t)x.b * p.T_q + x.t * p.G + q0) * p.H + x.h;
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (q0 + c < p.G) lse_next[c] = l[c * p.H];
    }
  };
  if (s.b < p.B) issue(s);
  while (s.b < p.B) {
    Step next = s;
    stride.advance(p, next);
    if (!(ok = ring.wait())) break;
    if (kOne || s.l0 == 0) {
      lse[0] = lse_next[0];
      lse[1] = lse_next[1];
      float dl = 0.f;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const uint4 zero = make_uint4(0, 0, 0, 0);
        qa[j] = row_ok ? query_chunk<D>(ring.queries, my_q, t4 + 4 * j) : zero;
        da[j] = row_ok ? query_chunk<D>(ring.queries + p.G * 2 * D, my_q, t4 + 4 * j) : zero;
        const uint4 oa = row_ok ? query_chunk<D>(ring.queries + 2 * p.G * 2 * D, my_q, t4 + 4 * j) : zero;
        float of[8], df[8];
        unpack8<T>(oa, of);
        unpack8<T>(da[j], df);
#pragma unroll
        for (int e = 0; e < 8; ++e) dl = fmaf(of[e], df[e], dl);
      }
      dl = quad_sum(dl);
      delta[0] = __shfl_sync(0xffffffffu, dl, 8 * t4);
      if (NC == 2) delta[1] = __shfl_sync(0xffffffffu, dl, 8 * t4 + 4);
#pragma unroll
      for (int i = 0; i < I; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) dq[i][e][0] = dq[i][e][1] = 0.f;
    }
    ring.stored_read();                             // the other stage and the query rows have been read
    if (next.b < p.B) issue(next);
    const unsigned char *kt = ring.stage(), *vt = kt + tile_bytes<D>();
    const int left = p.L - s.l0;                    // rows of the tile that exist (16 or more: all)

    // S^T and dP^T: [2 nt + c] = (tile row my_row + 8 nt, query q0 + c)
    float sc[4], dp[4];
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const uint4 k0 = tile_chunk<kRows>(kt, my_row, t4 + 4 * j), k1 = tile_chunk<kRows>(kt, 8 + my_row, t4 + 4 * j);
      const uint32_t ka[4] = {k0.x, k1.x, k0.y, k1.y}, kb[4] = {k0.z, k1.z, k0.w, k1.w};
      float s0[4] = {0.f, 0.f, 0.f, 0.f}, d0[4] = {0.f, 0.f, 0.f, 0.f};
      simt::Mma<T>::run(s0, ka, qa[j].x, qa[j].y);
      simt::Mma<T>::run(s0, kb, qa[j].z, qa[j].w);
      const uint4 v0 = tile_chunk<kRows>(vt, my_row, t4 + 4 * j), v1 = tile_chunk<kRows>(vt, 8 + my_row, t4 + 4 * j);
      const uint32_t va[4] = {v0.x, v1.x, v0.y, v1.y}, vb[4] = {v0.z, v1.z, v0.w, v1.w};
      simt::Mma<T>::run(d0, va, da[j].x, da[j].y);
      simt::Mma<T>::run(d0, vb, da[j].z, da[j].w);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        sc[x] = j == 0 ? s0[x] : sc[x] + s0[x];
        dp[x] = j == 0 ? d0[x] : dp[x] + d0[x];
      }
    }
    // left operands P^T and scale dS^T: rows my_row, my_row + 8; contracted index = queries, twice
    float pw[2][NC], ds[2][NC];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const bool live = my_row + 8 * nt < left;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        pw[nt][c] = live ? fast_exp2(fmaf(sc[2 * nt + c], p.scale_log2, -lse[c])) : 0.f;
        ds[nt][c] = live ? pw[nt][c] * (dp[2 * nt + c] - delta[c]) * p.scale : 0.f;
      }
    }
    const Scaled<T> ps(pw[0][0], pw[1][0], pw[0][NC - 1], pw[1][NC - 1]), dss(ds[0][0], ds[1][0], ds[0][NC - 1], ds[1][NC - 1]);
    uint32_t pt[4], dt[4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      if constexpr (QR == 4) {
        split3_rows<T>(pw[nt][0] * ps.up, pt[nt], pt[nt + 2]);
        split3_rows<T>(ds[nt][0] * dss.up, dt[nt], dt[nt + 2]);
      } else {
        split2<T>(pw[nt][0] * ps.up, pw[nt][1] * ps.up, pt[nt], pt[nt + 2]);
        split2<T>(ds[nt][0] * dss.up, ds[nt][1] * dss.up, dt[nt], dt[nt + 2]);
      }
    }
    {   // dQ^T += K^T (scale dS)^T
      const uint32_t d0[2] = {transpose8x8(dt[0]), transpose8x8(dt[2])}, d1[2] = {transpose8x8(dt[1]), transpose8x8(dt[3])};
#pragma unroll
      for (int i = 0; i < I; ++i) add_transposed<T, kOne, Scaled<T>::kUsed>(dq[i], kt, i, g, t4, left, d0, d1, dss.down);
    }
    // The gradient rows take the place of the K and V rows and leave as a tile: stored from registers, a
    // lane's 16 bytes beside three others', every instruction would write half lines.
    __syncwarp();                                   // the K and V rows have been read by every lane
    unsigned char* out = ring.tiles + (kt - ring.tiles);
    T* dkb = reinterpret_cast<T*>(p.dkd.ptr) + p.dkd.off(s.b, (int64_t)s.t * p.Ls + s.l0 + my_row, s.h) + 8 * t4;
    T* dvb = reinterpret_cast<T*>(p.dvd.ptr) + p.dvd.off(s.b, (int64_t)s.t * p.Ls + s.l0 + my_row, s.h) + 8 * t4;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const uint32_t qw[4] = {qa[j].x, qa[j].y, qa[j].z, qa[j].w}, dw[4] = {da[j].x, da[j].y, da[j].z, da[j].w};
      float gk[2][8], gv[2][8];                     // tile rows my_row, my_row + 8; chunk t + 4 j
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        float ck[4] = {0.f, 0.f, 0.f, 0.f}, cv[4] = {0.f, 0.f, 0.f, 0.f};
        const uint32_t qb = transpose8x8(qw[w]), db = transpose8x8(dw[w]);
        simt::Mma<T>::run(ck, dt, qb, qb);
        simt::Mma<T>::run(cv, pt, db, db);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          gk[x >> 1][2 * w + (x & 1)] = ck[x] * dss.down;
          gv[x >> 1][2 * w + (x & 1)] = cv[x] * ps.down;
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
        if (my_row + 8 * nt < left) {
          if (kAdd) {   // gradient cache shared by several layers: add to what earlier calls left
            if constexpr (NT == 4) {
              add8<T>(gk[nt], tile_chunk<kRows>(kt + 2 * tile_bytes<D>(), my_row + 8 * nt, t4 + 4 * j));
              add8<T>(gv[nt], tile_chunk<kRows>(kt + 3 * tile_bytes<D>(), my_row + 8 * nt, t4 + 4 * j));
            } else {
              add8<T>(gk[nt], *reinterpret_cast<const uint4*>(dkb + 8 * nt * p.dkd.st + 32 * j));
              add8<T>(gv[nt], *reinterpret_cast<const uint4*>(dvb + 8 * nt * p.dvd.st + 32 * j));
            }
          }
          *reinterpret_cast<uint4*>(out + chunk_at<kRows>(my_row + 8 * nt, t4 + 4 * j)) = pack8<T>(gk[nt]);
          *reinterpret_cast<uint4*>(out + tile_bytes<D>() + chunk_at<kRows>(my_row + 8 * nt, t4 + 4 * j)) = pack8<T>(gv[nt]);
        }
    }
    ring.store(p, omaps, s);

    if (kOne || left <= kRows) {
      T* qp = reinterpret_cast<T*>(p.dq.ptr) + p.dq.off(s.b, s.t * p.G + q0, s.h) + 8 * g;
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (q0 + c < p.G)
#pragma unroll
          for (int i = 0; i < I; ++i) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = QR == 4 ? dq[i][e][0] + dq[i][e][1] : dq[i][e][c];
            *reinterpret_cast<uint4*>(qp + c * p.dq.st + 64 * i) = pack8<T>(f);
          }
    }
    s = next;
  }
  if (!ok) {
    ring.drain();
    tc::publish_failure(p, ring.abort_flag);
  }
  ring.stored_read();                               // before the shared memory goes
}

// ------------------------------------------------------------------------- host side
inline bool make_maps(Maps* m, OutMaps* om, const Params& p, int dtype, int D, bool is_bwd) {
  memset(m, 0, sizeof(*m));
  memset(om, 0, sizeof(*om));
  const int64_t rows = (int64_t)p.T_kv * p.Ls;
  const int tail = p.L % kRows, g8 = p.G < 8 ? p.G : 8;
  if (p.L >= kRows && !(tc::make_map_rows(&m->k, p.kd, dtype, p.B, rows, p.H, D, kRows) && tc::make_map_rows(&m->v, p.vd, dtype, p.B, rows, p.H, D, kRows)))
    return false;
  if (tail != 0 && !(tc::make_map_rows(&m->kt, p.kd, dtype, p.B, rows, p.H, D, tail) && tc::make_map_rows(&m->vt, p.vd, dtype, p.B, rows, p.H, D, tail)))
    return false;
  if (!tc::make_map_rows(&m->q, p.q, dtype, p.B, p.T_q, p.H, D, g8, false)) return false;
  if (is_bwd && p.L >= kRows && !(tc::make_map_rows(&om->dk, p.dkd, dtype, p.B, rows, p.H, D, kRows) && tc::make_map_rows(&om->dv, p.dvd, dtype, p.B, rows, p.H, D, kRows)))
    return false;
  if (is_bwd && tail != 0 && !(tc::make_map_rows(&om->dkt, p.dkd, dtype, p.B, rows, p.H, D, tail) && tc::make_map_rows(&om->dvt, p.dvd, dtype, p.B, rows, p.H, D, tail)))
    return false;
  return !is_bwd || (tc::make_map_rows(&m->dout, p.dout, dtype, p.B, p.T_q, p.H, D, g8, false) &&
                     tc::make_map_rows(&m->o, p.o, dtype, p.B, p.T_q, p.H, D, g8, false));
}

// The backward keeps all query rows of a position in one group.
inline bool bwd_supported(int G) { return G <= 8; }

}  // namespace fda
}  // namespace moda
