// Host side of the tcgen05 backward: workspace layout, tensor maps and the launch sequences.
//
// Two sequences exist.  The default TWO-KERNEL one is the reference's structure: a query-parallel
// dq kernel and a key-parallel dk/dv kernel that both recompute the scores (seven executed matmuls).
// The FUSED one (D = 128, selected with MODA_PATH_TCGEN05_FUSED_BWD) runs
//     bounds (kvmax, pre, scale)  ->  bwd_fused_kernel over the sequence key tiles (dK, dV and the
//     sequence keys' share of dQ in a fixed-point accumulator)  ->  dq_kernel over the depth keys only,
//     which adds the two shares and writes dq  ->  depth gradients
// and executes the five matmuls of the backward once each; measured, it is no faster (see
// tc_bwd_fused_kernel.cuh), which is why it is not the default.
#pragma once
#include <algorithm>
#include <functional>

#include "tc_bwd_fused_kernel.cuh"

namespace moda {
namespace tc {

inline int padded_rows(int T_q) { return (T_q + 63) / 64 * 64 + 64; }

inline bool bwd_supported(const moda_problem* pr) {
  return (pr->D == 128 || pr->D == 64) && pr->mode != MODA_DEPTH_ONLY && pr->scale > 0.f && depth_layout_supported(pr);
}
inline bool bwd_is_fused(const moda_problem* pr) {
  return bwd_supported(pr) && pr->D == 128 && pr->path == MODA_PATH_TCGEN05_FUSED_BWD;
}

inline size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

// Workspace after the per-row delta of the generic path: delta_t, lse_t [B, H, T_qp] fp32 and, for
// the fused sequence, norm_t [B, H, T_qp] fp32, scale_blk [B, H, T_qp / 64] float4, kvmax [B, H, 2]
// and the dQ accumulator [B, H, T_qp, 128] int32.
struct BwdWorkspace {
  size_t stat = 0, scale = 0, kvmax = 0, acc = 0, total = 0;
  explicit BwdWorkspace(const moda_problem* pr) {
    if (!bwd_supported(pr)) return;
    const size_t rows = (size_t)pr->B * pr->H * padded_rows(pr->T_kv * pr->G);
    stat = align256(rows * sizeof(float));
    total = 2 * stat;
    if (bwd_is_fused(pr)) {
      scale = align256(rows / 64 * sizeof(float4));
      kvmax = align256((size_t)pr->B * pr->H * 2 * sizeof(int));
      acc = align256(rows * 128 * sizeof(int));
      total += stat + scale + kvmax + acc;
    }
  }
};
inline size_t bwd_extra_workspace_bytes(const moda_problem* pr) { return BwdWorkspace(pr).total; }

struct BwdMaps { DqMaps dq; DkvMaps dkv; DgOutMaps out; };
struct BwdBuffers { float *delta_t, *lse_t, *norm_t; float4* scale_blk; int* kvmax; int* dq_acc; size_t acc_bytes, kvmax_bytes; };

// CTAs that share a key tile of the dk/dv kernel.  A tile's query steps are a serial chain on one SM and
// under a causal mask the first tile has twice the average: with few tiles the launch lasts as long as
// that one.  But dk/dv's CTAs also run beside dq's, and shares that find no free SM at once cost more than they save.
// So the two grids are dealt out to the SMs as the GPU does it, heaviest CTA first, and the split whose last
// CTA ends first is taken if it wins a twentieth (beside the depth-gradient grid, which the deal leaves out:
// three).  In steps of 64 query rows x 128 keys a CTA takes its steps (dq's, of 64 keys, 0.7 each) and a fixed
// part: 15 for dq, 20 for dk/dv (set-up, first loads, stores), 3 more in a cluster (the sums' way through it);
// clusters of two and four find room on 95 and 87 % of the SMs.  344 shapes (2..320 tiles, D = 64 and 128, both types,
// three modes) with one, two and four CTAs a tile timed each: the choice is 0.7 % off the best on average, and
// slower than one CTA by more than 4 % (5 %) at one; dk/dv looked at as if it had the GPU to itself is 5 % off, and
// slower, by up to 39 %, at 61.
// D = 128, causal, us with one, two, four: T = 1024, G = 1: H = 4 30, 25, 35, H = 12 36, 42, 72; T = 4096, G = 2, H = 2 115, 70, 88.
struct SplitShape { int n_sm, T_kv, G, heads, causal, beside_dq, beside_depth; };
inline bool operator==(const SplitShape& a, const SplitShape& b) {
  return a.n_sm == b.n_sm && a.T_kv == b.T_kv && a.G == b.G && a.heads == b.heads && a.causal == b.causal && a.beside_dq == b.beside_dq &&
         a.beside_depth == b.beside_depth;
}
constexpr int kSplitSms = 512;
inline double last_cta_end(const SplitShape& s, int parts) {
  constexpr double kDqStep = 0.7, kDqFixed = 15, kFixed = 20, kCluster = 3;
  double free_at[kSplitSms] = {0.};                         // a heap, the SM that is free first on top
  const int n_sm = parts == 1 ? s.n_sm : parts == 2 ? s.n_sm * 95 / 100 : s.n_sm * 87 / 100;
  double end = 0;
  auto deal = [&](int tiles, double steps, double fixed, int n) {
    for (int i = 0; i < tiles; ++i) {
      const double cost = fixed + steps * (s.causal ? 1. - (double)i / tiles : 1.);
      for (int h = 0; h < s.heads; ++h) {
        for (int k = 0; k < n; ++k) std::pop_heap(free_at, free_at + n_sm - k, std::greater<double>());
        const double t = free_at[n_sm - n] + cost;          // from when the last of the n SMs is free
        for (int k = n - 1; k >= 0; --k) {
          free_at[n_sm - 1 - k] = t;
          std::push_heap(free_at, free_at + n_sm - k, std::greater<double>());
        }
        end = std::max(end, t);
      }
    }
  };
  const int64_t T_q = (int64_t)s.T_kv * s.G, q_tiles = (T_q + kBM - 1) / kBM, q_steps = (T_q + kStep - 1) / kStep;
  // dq with more than two CTAs an SM ends on all SMs at about the same time
  if (s.beside_dq && q_tiles * s.heads <= 2 * s.n_sm) deal((int)q_tiles, kDqStep * ((s.T_kv + kStep - 1) / kStep), kDqFixed, 1);
  deal((s.T_kv + kBN - 1) / kBN, (double)q_steps / parts, kFixed + (parts > 1 ? kCluster : 0), parts);
  return end;
}
inline int dkv_parts(const Params& p, int n_sm, bool beside_dq, bool beside_depth) {
  const int64_t tiles = (int64_t)((p.T_kv + kBN - 1) / kBN) * p.H * p.B, steps = (p.T_q + kStep - 1) / kStep;
  if (tiles > 2 * n_sm || steps < 4 || n_sm < 8 || n_sm > kSplitSms) return 1;
  const SplitShape shape{n_sm, p.T_kv, p.G, p.H * p.B, p.mode != kNonCausal, beside_dq, beside_depth};
  // The deal takes some 30 us of host time, and its answer depends on the shape alone: a thread keeps a few.
  static thread_local struct { SplitShape shape; int parts; } known[16];       // parts 0: empty
  auto& slot = known[((uint32_t)p.T_kv * 31u + (uint32_t)p.G * 7u + (uint32_t)shape.heads) & 15u];
  if (slot.parts != 0 && slot.shape == shape) return slot.parts;
  double best = last_cta_end(shape, 1);
  int parts = 1;
  for (int n = 2; n <= 4 && steps >= 2 * n; n *= 2) {
    const double t = last_cta_end(shape, n);
    if (t < (beside_depth ? 0.85 : 0.95) * best) { best = t; parts = n; }
  }
  slot.shape = shape;
  slot.parts = parts;
  return parts;
}

// `overlap`: the launch may begin when every CTA of the one before it has reached grid_started()
// (tc_bwd_kernels.cuh says how the kernels keep their order); `parts` CTAs in x form a cluster.
template <typename... KernelArgs, typename... Args>
inline cudaError_t launch_next(void (*kern)(KernelArgs...), dim3 grid, int threads, size_t smem, int parts, bool overlap, cudaStream_t st,
                               const Args&... args) {
  cudaLaunchAttribute attr[2]{};
  int n = 0;
  if (overlap) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (parts > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = parts;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

template <typename T, int D>
inline cudaError_t launch_bwd(const Params& p, const BwdMaps& m, const BwdBuffers& w, int T_qp, bool dg, bool fused,
                              int n_sm, cudaStream_t st, int* launches) {
  cudaError_t e;
  float* delta_t = w.delta_t;
  float* lse_t = w.lse_t;
  const int n_seq = (p.T_kv + kBN - 1) / kBN;
  const int n_dep_tiles = (int)(((int64_t)p.T_kv * p.L + kBN - 1) / kBN);
  // The ends of a launch are a share of it that shrinks with the CTAs an SM works through.  Backward with overlap
  // against without (causal, all keys, chunk-visible, D = 64 and 128): 0.80-0.94 at one or two CTAs of dq an SM,
  // 0.94-0.98 at 3.5, 0.97-0.99 at 7, 0.98-1.01 at 14, 0.95-1.08 and no tendency at 28 and 42.
  // A caller may have the key gradients written over the keys: every key tile is read by the CTA that writes its
  // gradient and, before that, by dq, which must then have ended.
  auto over = [](const View& out, const View& a, const View& b) { return out.ptr != nullptr && (out.ptr == a.ptr || out.ptr == b.ptr); };
  const bool in_place = over(p.dk, p.k, p.v) || over(p.dv, p.k, p.v) || over(p.dkd, p.kd, p.vd) || over(p.dvd, p.kd, p.vd);
  const bool overlap = !fused && !in_place && (int64_t)((p.T_q + kBM - 1) / kBM) * p.H * p.B <= (int64_t)16 * n_sm;
  if (fused) {
    if constexpr (D == 128) {
      if ((e = cudaMemsetAsync(w.kvmax, 0, w.kvmax_bytes, st)) != cudaSuccess) return e;
      const int64_t groups = (int64_t)p.B * p.H * ((p.T_kv + 31) / 32);
      const int64_t cap = (int64_t)n_sm * 16;
      prof::Scope ps(prof::kBwdBoundsTc, st);
      kvmax_kernel<T><<<(int)(groups < cap ? groups : cap), 256, 0, st>>>(p, w.kvmax);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      *launches += 1;
    }
  }
  {
    const int64_t groups = (int64_t)p.B * p.H * (T_qp / 32);
    const int64_t cap = (int64_t)n_sm * 16;
    const int blocks = (int)(groups < cap ? groups : cap);
    prof::Scope ps(prof::kPreTc, st);
    pre_kernel<T, D><<<blocks, 256, 0, st>>>(p, delta_t, lse_t, fused ? w.norm_t : nullptr, T_qp);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  *launches += 1;
  const size_t dq_smem = dq_ring<D>() * 2 * (size_t)step_tile<D>() + 2 * (size_t)kScoreTile + kCtlBytes;
  const size_t dkv_smem = dkv_ring<D>() * (2 * (size_t)step_tile<D>() + 512) + 2 * (size_t)kDkvPairBytes + kCtlBytes;
  if (fused) {
    if constexpr (D == 128) {
      {
        const int64_t n_blk = (int64_t)p.B * p.H * (T_qp / 64);
        const int64_t want = (n_blk + 7) / 8, cap = (int64_t)n_sm * 8;
        prof::Scope ps(prof::kBwdBoundsTc, st);
        scale_kernel<<<(int)(want < cap ? want : cap), 256, 0, st>>>(delta_t, w.norm_t, w.kvmax, w.scale_blk, T_qp, n_blk);
      }
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      *launches += 1;
      if ((e = cudaMemsetAsync(w.dq_acc, 0, w.acc_bytes, st)) != cudaSuccess) return e;
      {
        auto kern = bwd_fused_kernel<T>;
        if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFuSmem)) != cudaSuccess) return e;
        dim3 grid(n_seq, p.H, p.B);
        prof::Scope ps(prof::kBwdFusedTc, st);
        kern<<<grid, kFusedBwdThreads, kFuSmem, st>>>(p, m.dkv, delta_t, lse_t, w.scale_blk, w.dq_acc, T_qp);
      }
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      *launches += 1;
      {   // depth keys' share of dQ, added to the accumulated sequence share; writes dq
        auto kern = dq_kernel<T, D>;
        if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dq_smem)) != cudaSuccess) return e;
        dim3 grid((p.T_q + kBM - 1) / kBM, p.H, p.B);
        prof::Scope ps(prof::kDqTc, st);
        kern<<<grid, kDqThreads, dq_smem, st>>>(p, m.dq, delta_t, lse_t, T_qp, w.dq_acc, w.scale_blk);
      }
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      *launches += 1;
      if (!dg && n_dep_tiles > 0) {   // depth key tiles the query-stationary kernel cannot own: key-parallel kernel on them alone
        auto kern = dkv_kernel<T, D, false>;
        if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dkv_smem)) != cudaSuccess) return e;
        dim3 grid(n_dep_tiles, p.H, p.B);
        prof::Scope ps(prof::kDkvTc, st);
        kern<<<grid, kDkvThreads, dkv_smem, st>>>(p, m.dkv, delta_t, lse_t, T_qp, 0);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        *launches += 1;
      }
    }
  } else {
    {
      auto kern = dq_kernel<T, D>;
      if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dq_smem)) != cudaSuccess) return e;
      dim3 grid((p.T_q + kBM - 1) / kBM, p.H, p.B);
      prof::Scope ps(prof::kDqTc, st);
      e = launch_next(kern, grid, kDqThreads, dq_smem, 1, overlap, st, p, m.dq, (const float*)delta_t, (const float*)lse_t, T_qp, (const int*)nullptr,
                      (const float4*)nullptr);
    }
    if (e != cudaSuccess) return e;
    *launches += 1;
    {
      const bool own_tiles = !dg && n_dep_tiles > 0;
      const int parts = own_tiles ? 1 : dkv_parts(p, n_sm, overlap, overlap && dg);
      auto kern = parts > 1 ? dkv_kernel<T, D, true> : dkv_kernel<T, D, false>;
      if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dkv_smem)) != cudaSuccess) return e;
      const dim3 grid((n_seq + (own_tiles ? n_dep_tiles : 0)) * parts, p.H, p.B);
      prof::Scope ps(parts > 1 ? prof::kDkvSplitTc : prof::kDkvTc, st);
      e = launch_next(kern, grid, kDkvThreads, dkv_smem, parts, overlap, st, p, m.dkv, (const float*)delta_t, (const float*)lse_t, T_qp, n_seq);
    }
    if (e != cudaSuccess) return e;
    *launches += 1;
  }
  if (dg) {
    auto kern = depth_grad_kernel<T, D>;
    constexpr uint32_t smem = dg_smem<D>();
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
    const int64_t n_blocks = (int64_t)((p.T_q + kStep - 1) / kStep) * p.H * p.B;
    dim3 grid((unsigned)(n_blocks < n_sm ? n_blocks : n_sm));
    {
      prof::Scope ps(prof::kDepthGradTc, st);
      e = launch_next(kern, grid, kDgThreads, smem, 1, overlap, st, p, m.dkv, m.out, (const float*)delta_t, (const float*)lse_t, T_qp);
    }
    if (e != cudaSuccess) return e;
    *launches += 1;
  }
  return cudaSuccess;
}

inline int bwd(const Params& p, const moda_problem* pr, void* extra, int n_sm, cudaStream_t st, int* launches, int* cuda_err) {
  const int T_qp = padded_rows(p.T_q);
  const BwdWorkspace ws(pr);
  const bool fused = bwd_is_fused(pr);
  unsigned char* base = reinterpret_cast<unsigned char*>(extra);
  BwdBuffers w{};
  w.delta_t = reinterpret_cast<float*>(base);
  w.lse_t = reinterpret_cast<float*>(base + ws.stat);
  if (fused) {
    w.norm_t = reinterpret_cast<float*>(base + 2 * ws.stat);
    w.scale_blk = reinterpret_cast<float4*>(base + 3 * ws.stat);
    w.kvmax = reinterpret_cast<int*>(base + 3 * ws.stat + ws.scale);
    w.dq_acc = reinterpret_cast<int*>(base + 3 * ws.stat + ws.scale + ws.kvmax);
    w.acc_bytes = ws.acc;
    w.kvmax_bytes = ws.kvmax;
  }
  const bool dep = p.L > 0;
  const int D = pr->D, dt = pr->dtype;

  BwdMaps m;
  memset(&m, 0, sizeof(m));
  bool ok = make_map_rows(&m.dq.k, p.k, dt, p.B, p.T_kv, p.H, D, 64) &&
            make_map_rows(&m.dq.v, p.v, dt, p.B, p.T_kv, p.H, D, 64) &&
            make_map_rows(&m.dkv.k, p.k, dt, p.B, p.T_kv, p.H, D, 128) &&
            make_map_rows(&m.dkv.v, p.v, dt, p.B, p.T_kv, p.H, D, 128) &&
            make_map_rows(&m.dkv.q, p.q, dt, p.B, p.T_q, p.H, D, 64) &&
            make_map_rows(&m.dkv.dout, p.dout, dt, p.B, p.T_q, p.H, D, 64);
  if (ok && dep) {
    ok = make_map_depth(&m.dq.kd, p.kd, dt, p, D, 64) && make_map_depth(&m.dq.vd, p.vd, dt, p, D, 64) &&
         make_map_depth(&m.dkv.kd, p.kd, dt, p, D, 128) && make_map_depth(&m.dkv.vd, p.vd, dt, p, D, 128);
  } else if (ok) {
    m.dq.kd = m.dq.k; m.dq.vd = m.dq.v; m.dkv.kd = m.dkv.k; m.dkv.vd = m.dkv.v;
  }
  if (!ok) return MODA_ERR_UNSUPPORTED;
  const bool dg = depth_grad_applies(p, pr);
  const bool boxes = p.Ls == p.L || (dep && 32 % p.L == 0);      // depth_grad_kernel stores boxes of 32 rows, or row by row
  if (dg && boxes && !(make_map_depth(&m.out.dkd, p.dkd, dt, p, D, 32) && make_map_depth(&m.out.dvd, p.dvd, dt, p, D, 32)))
    return MODA_ERR_UNSUPPORTED;
  if ((int64_t)((p.T_q + kStep - 1) / kStep) * p.H * p.B > 0x7fffffff || n_sm <= 0) return MODA_ERR_UNSUPPORTED;

  cudaError_t e;
  const bool bf = dt == MODA_BF16;
  if (D == 128) e = bf ? launch_bwd<__nv_bfloat16, 128>(p, m, w, T_qp, dg, fused, n_sm, st, launches)
                       : launch_bwd<__half, 128>(p, m, w, T_qp, dg, fused, n_sm, st, launches);
  else e = bf ? launch_bwd<__nv_bfloat16, 64>(p, m, w, T_qp, dg, false, n_sm, st, launches)
              : launch_bwd<__half, 64>(p, m, w, T_qp, dg, false, n_sm, st, launches);
  if (e != cudaSuccess) { *cuda_err = (int)e; return MODA_ERR_CUDA; }
  return MODA_OK;
}

}  // namespace tc
}  // namespace moda
