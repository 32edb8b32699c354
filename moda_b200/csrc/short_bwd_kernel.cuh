// Backward of the sequence keys for short sequences (D = 64, at most 256 keys): one CTA owns a (batch,
// KV head), all of its keys and all of its query rows, so that the scores are computed once (five
// matmuls instead of the seven of dq_kernel + dkv_kernel), every operand is read once and dq needs no
// sum over CTAs.
//
// What bounds the tile kernels there is not their matmuls: a CTA of dq_kernel or dkv_kernel has four
// steps at T = 197 and spends most of its life in set-up, first loads and stores, alone on its SM.
// Here a warp owns 16 keys (warp-level m16n8k16 matrix instructions, dK and dV in registers) and the
// CTA walks the query rows in blocks of 32 with one barrier a block:
//
//   S^T = K Q^T, dP^T = V dO^T  ->  P^T, dS^T (registers)  ->  dV += P^T dO, dK += dS^T Q;  dS^T also to shared memory
//   barrier
//   dQ = dS K of the block, divided over the warps (16 rows x 16 channels each)
//
// dS^T is double-buffered, so a warp that has no share of dQ goes on to the next block.  The tiles of
// block i + 2 (cp.async) and the row sums delta = o . dO of block i + 1 are made during block i, which
// takes the statistics launch and its pass over o and dO away.
// What bounds it now is the chain from block to block of its one CTA an SM (13 warps at T = 197: issue slots 31 %
// busy, tensor pipe 24 %, most stalls at the block's barrier and on dependent instructions), which is why it
// has no advantage beyond a few hundred keys, nor on the GPU alone with few heads (use_short_bwd).  1536 heads (B = 256, H = 6),
// T = 197: statistics + dq + dk/dv 404 us -> 351 us; 384 heads: 122 -> 97 us a layer.
#pragma once
#include "simt_mma_kernels.cuh"

namespace moda {
namespace shortseq {

constexpr int kD = 64, kBQ = 32;                 // head dim; query rows of a block
constexpr int kMaxKeys = 256;
constexpr int kLdS = kBQ + 8;                    // row stride of the dS^T tile (80 bytes: no bank conflicts)
constexpr int kLd = kD + 8;                      // row stride of every other tile (simt::Tile)

// K, V; three blocks of {Q, dO}; two of O; two dS^T tiles; two of {lse, delta}.
__host__ __device__ constexpr size_t smem_bytes(int warps) {
  const size_t keys = 16 * (size_t)warps;
  return 2 * keys * kLd * 2 + (3 * 2 + 2) * (size_t)kBQ * kLd * 2 + 2 * keys * kLdS * 2 + 2 * 2 * kBQ * 4;
}

// A warp has 128 registers (four warps a sub-partition from 13 on): 64 of dK and dV, 16 of its K rows as
// left operands; the V operands are read again for every 16 query rows.
template <typename T>
__global__ void __launch_bounds__(kMaxKeys * 2, 1) bwd_kernel(const __grid_constant__ Params p) {
  using TL = simt::Tile<T, kD>;
  using Mma = simt::Mma<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int warps = nt >> 5, keys = warps * 16;
  T* sK = reinterpret_cast<T*>(smem_raw);
  T* sV = sK + keys * kLd;
  T* sQ = sV + keys * kLd;                       // slot s: sQ + s * kBQ * kLd
  T* sDO = sQ + 3 * kBQ * kLd;
  T* sO = sDO + 3 * kBQ * kLd;
  T* sS = sO + 2 * kBQ * kLd;                    // [2][keys][kLdS]
  float* sStat = reinterpret_cast<float*>(sS + 2 * keys * kLdS);   // [2][lse, delta][kBQ]
  const int h = blockIdx.x % p.H, b = blockIdx.x / p.H;
  const int n_blocks = (p.T_q + kBQ - 1) / kBQ;
  const bool causal = p.mode != kNonCausal;

  const T* gq = reinterpret_cast<const T*>(p.q.ptr) + p.q.off(b, 0, h);
  const T* gdo = reinterpret_cast<const T*>(p.dout.ptr) + p.dout.off(b, 0, h);
  const T* go = reinterpret_cast<const T*>(p.o.ptr) + p.o.off(b, 0, h);

  // rows [row0, row0 + rows) of a tensor, zeros past n_rows
  auto load = [&](T* s, const T* gsrc, int64_t st, int row0, int rows, int n_rows) {
    for (int i = tid; i < rows * (kD / 8); i += nt) {
      const int r = i / (kD / 8), c = i % (kD / 8);
      T* dst = s + r * kLd + c * 8;
      if (row0 + r < n_rows) simt::cp_async16(smem_u32(dst), gsrc + (int64_t)(row0 + r) * st + c * 8);
      else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
    }
  };
  auto load_block = [&](int i) {
    const int slot = i % 3;
    load(sQ + slot * kBQ * kLd, gq, p.q.st, i * kBQ, kBQ, p.T_q);
    load(sDO + slot * kBQ * kLd, gdo, p.dout.st, i * kBQ, kBQ, p.T_q);
    load(sO + (i & 1) * kBQ * kLd, go, p.o.st, i * kBQ, kBQ, p.T_q);
  };
  // delta and lse of block i: four lanes a row, 16 channels each
  auto statistics = [&](int i) {
    for (int x = tid; x < kBQ * 4; x += nt) {            // whole warps: the four lanes of a row are in one
      const int r = x >> 2, row = i * kBQ + r;
      const T* po = sO + (i & 1) * kBQ * kLd + r * kLd + (x & 3) * 16;
      const T* pd = sDO + (i % 3) * kBQ * kLd + r * kLd + (x & 3) * 16;
      float s = 0.f;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint4 a = *reinterpret_cast<const uint4*>(po + 8 * c), d = *reinterpret_cast<const uint4*>(pd + 8 * c);
        const uint32_t av[4] = {a.x, a.y, a.z, a.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 u = Pack<T>::unpack(av[e]), w = Pack<T>::unpack(dv[e]);
          s = fmaf(u.x, w.x, fmaf(u.y, w.y, s));
        }
      }
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if ((x & 3) == 0) {
        float* st = sStat + (i & 1) * 2 * kBQ;
        st[r] = row < p.T_q ? p.lse[((int64_t)b * p.T_q + row) * p.H + h] : 0.f;
        st[kBQ + r] = s;
      }
    }
  };

  load(sK, reinterpret_cast<const T*>(p.k.ptr) + p.k.off(b, 0, h), p.k.st, 0, keys, p.T_kv);
  load(sV, reinterpret_cast<const T*>(p.v.ptr) + p.v.off(b, 0, h), p.v.st, 0, keys, p.T_kv);
  load_block(0);
  if (n_blocks > 1) load_block(1);
  simt::cp_async_commit();
  simt::cp_async_wait<0>();
  __syncthreads();
  statistics(0);
  __syncthreads();

  uint32_t kf[4][4];                             // K rows of this warp as left operands
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) TL::ldA(kf[kk], sK, warp * 16, kk * 16, lane);
  float dk[8][4], dv[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) { dk[i][0] = dk[i][1] = dk[i][2] = dk[i][3] = dv[i][0] = dv[i][1] = dv[i][2] = dv[i][3] = 0.f; }
  // first query row that sees key g (key g + 8) of the warp; T_q: none does
  const int keyA = warp * 16 + g, keyB = keyA + 8;
  const int loA = keyA < p.T_kv ? (causal ? keyA * p.G : 0) : p.T_q, loB = keyB < p.T_kv ? (causal ? keyB * p.G : 0) : p.T_q;
  const int lo_all = causal ? (warp * 16 + 15) * p.G : 0;          // from here on every key of the warp is seen
  const bool whole = warp * 16 + 16 <= p.T_kv;
  const float c = p.scale_log2;

  for (int i = 0; i < n_blocks; ++i) {
    if (i + 2 < n_blocks) load_block(i + 2);
    simt::cp_async_commit();
    const int q0 = i * kBQ, r_last = min(q0 + kBQ, p.T_q) - 1;
    // groups of 16 keys that a row of the block sees; the warps of the others have nothing to do
    const int n_groups = causal ? min(warps, r_last / p.G / 16 + 1) : warps;
    const T *cQ = sQ + (i % 3) * kBQ * kLd, *cDO = sDO + (i % 3) * kBQ * kLd;
    T* cS = sS + (i & 1) * keys * kLdS;
    if (warp < n_groups) {
      const float* st = sStat + (i & 1) * 2 * kBQ;
      const bool masked = !whole || q0 < lo_all || q0 + kBQ > p.T_q;
      const int n_half = (min(kBQ, p.T_q - q0) + 15) / 16;
#pragma unroll 1
      for (int j = 0; j < n_half; ++j) {
        float s[2][4], dp[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) { s[n][0] = s[n][1] = s[n][2] = s[n][3] = dp[n][0] = dp[n][1] = dp[n][2] = dp[n][3] = 0.f; }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          uint32_t bq[4], bd[4], va[4];
          TL::ldB_nk(bq, cQ, j * 16, kk * 16, lane);
          TL::ldB_nk(bd, cDO, j * 16, kk * 16, lane);
          TL::ldA(va, sV, warp * 16, kk * 16, lane);
          Mma::run(s[0], kf[kk], bq[0], bq[1]);
          Mma::run(s[1], kf[kk], bq[2], bq[3]);
          Mma::run(dp[0], va, bd[0], bd[1]);
          Mma::run(dp[1], va, bd[2], bd[3]);
        }
        uint32_t pa[4], da[4];                   // P^T and dS^T as left operands
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const int col = j * 16 + n * 8 + t4 * 2, r = q0 + col;
          const float2 l = *reinterpret_cast<const float2*>(st + col), d = *reinterpret_cast<const float2*>(st + kBQ + col);
          float pr[4] = {fast_exp2(fmaf(s[n][0], c, -l.x)), fast_exp2(fmaf(s[n][1], c, -l.y)),
                         fast_exp2(fmaf(s[n][2], c, -l.x)), fast_exp2(fmaf(s[n][3], c, -l.y))};
          if (masked) {
            if (r < loA || r >= p.T_q) pr[0] = 0.f;
            if (r + 1 < loA || r + 1 >= p.T_q) pr[1] = 0.f;
            if (r < loB || r >= p.T_q) pr[2] = 0.f;
            if (r + 1 < loB || r + 1 >= p.T_q) pr[3] = 0.f;
          }
          pa[2 * n] = Pack<T>::pack(pr[0], pr[1]);
          pa[2 * n + 1] = Pack<T>::pack(pr[2], pr[3]);
          da[2 * n] = Pack<T>::pack(pr[0] * (dp[n][0] - d.x), pr[1] * (dp[n][1] - d.y));
          da[2 * n + 1] = Pack<T>::pack(pr[2] * (dp[n][2] - d.x), pr[3] * (dp[n][3] - d.y));
          *reinterpret_cast<uint32_t*>(cS + keyA * kLdS + col) = da[2 * n];
          *reinterpret_cast<uint32_t*>(cS + keyB * kLdS + col) = da[2 * n + 1];
        }
#pragma unroll
        for (int d2 = 0; d2 < 4; ++d2) {
          uint32_t bb[4];
          TL::ldB_kn(bb, cDO, j * 16, d2 * 16, lane);
          Mma::run(dv[2 * d2], pa, bb[0], bb[1]);
          Mma::run(dv[2 * d2 + 1], pa, bb[2], bb[3]);
          TL::ldB_kn(bb, cQ, j * 16, d2 * 16, lane);
          Mma::run(dk[2 * d2], da, bb[0], bb[1]);
          Mma::run(dk[2 * d2 + 1], da, bb[2], bb[3]);
        }
      }
    }
    if (i + 1 < n_blocks) statistics(i + 1);
    simt::cp_async_wait<0>();
    __syncthreads();
    // dQ of the block: unit u = 16 rows x 16 channels; the last warps first (under a causal mask they are idle)
    for (int u = warps - 1 - warp; u < 2 * 4; u += warps) {
      const int m0 = (u & 1) * 16, d0 = (u >> 1) * 16;
      if (q0 + m0 >= p.T_q) continue;
      float acc[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n) { acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f; }
#pragma unroll 4
      for (int kg = 0; kg < n_groups; ++kg) {
        uint32_t a[4], bb[4];
        simt::ldsm_x4_t(a, smem_u32(cS + (kg * 16 + (lane & 7) + (lane >> 4) * 8) * kLdS + m0 + ((lane >> 3) & 1) * 8));
        TL::ldB_kn(bb, sK, kg * 16, d0, lane);
        Mma::run(acc[0], a, bb[0], bb[1]);
        Mma::run(acc[1], a, bb[2], bb[3]);
      }
      T* gdq = reinterpret_cast<T*>(p.dq.ptr) + p.dq.off(b, 0, h);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = q0 + m0 + g + 8 * e;
        if (row < p.T_q) {
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            uint32_t* dst = reinterpret_cast<uint32_t*>(gdq + (int64_t)row * p.dq.st + d0 + n * 8 + t4 * 2);
            float x = acc[n][2 * e] * p.scale, y = acc[n][2 * e + 1] * p.scale;
            if (p.merge_depth) { const float2 prev = Pack<T>::unpack(*dst); x += prev.x; y += prev.y; }
            *dst = Pack<T>::pack(x, y);
          }
        }
      }
    }
  }
  // dK and dV rows leave through the tiles of K and V, 16 bytes a lane
  __syncthreads();                               // the last dQ has read K
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const int o = n * 8 + t4 * 2;
    *reinterpret_cast<uint32_t*>(sK + keyA * kLd + o) = Pack<T>::pack(dk[n][0] * p.scale, dk[n][1] * p.scale);
    *reinterpret_cast<uint32_t*>(sK + keyB * kLd + o) = Pack<T>::pack(dk[n][2] * p.scale, dk[n][3] * p.scale);
    *reinterpret_cast<uint32_t*>(sV + keyA * kLd + o) = Pack<T>::pack(dv[n][0], dv[n][1]);
    *reinterpret_cast<uint32_t*>(sV + keyB * kLd + o) = Pack<T>::pack(dv[n][2], dv[n][3]);
  }
  __syncwarp();
  T* gdk = reinterpret_cast<T*>(p.dk.ptr) + p.dk.off(b, 0, h);
  T* gdv = reinterpret_cast<T*>(p.dv.ptr) + p.dv.off(b, 0, h);
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const int row = warp * 16 + x * 4 + (lane >> 3), ch = (lane & 7) * 8;
    if (row < p.T_kv) {
      *reinterpret_cast<uint4*>(gdk + (int64_t)row * p.dk.st + ch) = *reinterpret_cast<const uint4*>(sK + row * kLd + ch);
      *reinterpret_cast<uint4*>(gdv + (int64_t)row * p.dv.st + ch) = *reinterpret_cast<const uint4*>(sV + row * kLd + ch);
    }
  }
}

}  // namespace shortseq
}  // namespace moda
