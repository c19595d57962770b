// Fused triangular sweeps for the FP32 refinement: the whole forward (L, with
// the stored per-panel row moves) or backward (U) substitution of a group of
// right-hand-side columns runs in one thread-block cluster per (matrix, column
// group), with the right-hand sides resident in the shared memories of its
// CTAs.  One launch replaces the ~2 x n/NB small launches of the blocked
// sweep, and each cluster streams its triangle exactly once.
//
// Reference: the solve half of complex32_faer_lu_solve
// (crates/refeff-linalg/src/lu.rs:474-529), applied to the elimination's
// factors and row moves.
//
// The NB-row blocks are dealt round robin to the CTAs.  A step: the block's
// owner solves it with the block's triangle (a warp a column; the triangle is
// brought in by cp.async one of its blocks ahead) and writes the solved rows
// into every CTA's buffer (distributed shared memory); after one cluster
// barrier each CTA subtracts their contribution from its own rows.  The first
// factor entries of that update are loaded before the barrier.  Row moves
// (forward) are pushed by the CTAs that hold the source rows, one more barrier
// where a panel has any.  A row's arithmetic does not depend on the number of
// CTAs.
//
// A step is bound by its chain: the 64 dependent rows of the solve, the
// barrier, and the loads and multiply-adds of one panel's rows.  At n = 4112 in
// 8 CTAs, backward, it takes 15 us: solve 5, barrier 1.5, update 6.  Measured
// and not taken: prefetches of the next panel into L2 (2 us a step to issue),
// two rows a thread (fewer loads in flight), 8-row blocks of the solve by their
// inverses (the inverses cost what they save).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "batched_lu.cuh"
#include "cplx.cuh"
#include "fms_plan.cuh"

namespace cg = cooperative_groups;

namespace rfx {
namespace {

constexpr int kSwUnroll = 16, kSwLists = 2;

__device__ __forceinline__ void sw_cp_async16(void* dst, const void* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// Shared memory of one CTA: Y[CG][ldl] (its rows), T[NB][NB] (a block's triangle, by columns), the reciprocal diagonal,
// X[2][NB][CG] (solved rows, by step parity), tmp[2][2 NB][CG] (moved rows), the step's moves [2][2 NB].
template <int NB, int CG>
struct SweepSmem {
  static int ldl(int n, int cl) { return ((n + NB - 1) / NB + cl - 1) / cl * NB; }
  static size_t bytes(int n, int cl) {
    return (size_t(ldl(n, cl)) * CG + size_t(NB) * NB + NB + size_t(2 * NB) * CG + size_t(4 * NB) * CG) * sizeof(float2) + kSwLists * (2 * NB) * sizeof(int2);
  }
};

// Y[r] -= sum_j T(r, j) X[j] over the CTA's rows [l_begin, l_end) (numbered within the CTA), j < kb, T column j at
// panel + lda j.  Each thread walks its rows in batches of kSwUnroll columns and loads the next batch (of the same row
// or of its next row) before it multiplies the current one; the first batch is loaded by the constructor, which does
// not need X.
template <int NB, int CG, int kThreads>
struct SweepUpdate {
  const float2* panel;
  size_t lda;
  int kb, nfull, l, l_end, rank, shift, bi = 0;
  float2 cur[kSwUnroll];

  __device__ __forceinline__ int row(int local) const { return (((local / NB) << shift) + rank) * NB + local % NB; }
  __device__ __forceinline__ void load(int local, int batch, float2 (&v)[kSwUnroll]) const {
    const float2* p = panel + row(local) + lda * size_t(batch * kSwUnroll);
#pragma unroll
    for (int u = 0; u < kSwUnroll; ++u) v[u] = p[lda * u];
  }
  __device__ __forceinline__ SweepUpdate(const float2* panel_, size_t lda_, int kb_, int l_begin, int l_end_, int rank_,
                                         int shift_)
      : panel(panel_), lda(lda_), kb(kb_), nfull(kb_ / kSwUnroll), l(l_begin + int(threadIdx.x)), l_end(l_end_),
        rank(rank_), shift(shift_) {
    if (nfull > 0 && l < l_end) load(l, 0, cur);
  }
  __device__ __forceinline__ static void madd(float2 (&acc)[CG], float2 v, const float2* x) {
    if constexpr (CG == 1) {
      cfma(acc[0], v, x[0]);
    } else {
#pragma unroll
      for (int c = 0; c < CG; c += 2) {
        const float4 q = *reinterpret_cast<const float4*>(x + c);
        cfma(acc[c], v, make_float2(q.x, q.y));
        cfma(acc[c + 1], v, make_float2(q.z, q.w));
      }
    }
  }
  __device__ __forceinline__ void run(const float2* X, float2* Y, int ldl) {
    if (l >= l_end) return;
    float2 acc[CG];
#pragma unroll
    for (int c = 0; c < CG; ++c) acc[c] = make_float2(0.f, 0.f);
    auto rest = [&] {  // the columns past the full batches, then the row
      for (int j = nfull * kSwUnroll; j < kb; ++j) madd(acc, panel[row(l) + lda * size_t(j)], X + j * CG);
#pragma unroll
      for (int c = 0; c < CG; ++c) {
        float2& y = Y[c * ldl + l];
        y = csub(y, acc[c]);
        acc[c] = make_float2(0.f, 0.f);
      }
    };
    if (nfull == 0) {
      for (; l < l_end; l += kThreads) rest();
      return;
    }
    for (;;) {
      int ln = l, bn = bi + 1;
      if (bn == nfull) {
        ln = l + kThreads;
        bn = 0;
      }
      const bool more = ln < l_end;
      float2 nxt[kSwUnroll];
      if (more) load(ln, bn, nxt);
      const float2* x = X + bi * kSwUnroll * CG;
#pragma unroll
      for (int u = 0; u < kSwUnroll; ++u) madd(acc, cur[u], x + u * CG);
      if (bn == 0) rest();
      if (!more) break;
      l = ln;
      bi = bn;
#pragma unroll
      for (int u = 0; u < kSwUnroll; ++u) cur[u] = nxt[u];
    }
  }
};

// shift: log2 of the cluster size
template <bool kForward, int NB, int CG, int kThreads>
__global__ void __launch_bounds__(kThreads, kThreads == 256 ? 2 : 1)
    sweep_kernel(BatchLayout lay, float2* __restrict__ M, LuWork w, int shift, const int* skip) {
  cg::cluster_group cluster = cg::this_cluster();
  const int cl = 1 << shift, rank = cl > 1 ? int(cluster.block_rank()) : 0;
  const int b = blockIdx.y, cg0 = int(blockIdx.x >> shift) * CG;
  if (skip && skip[b]) return;
  const int n = lay.n, ncols = min(CG, lay.m - cg0), nblk = (n + NB - 1) / NB;
  const int ldl = (nblk + cl - 1) / cl * NB;
  extern __shared__ __align__(16) float2 sw_sm[];
  float2* Y = sw_sm;                            // [CG][ldl]
  float2* T = Y + size_t(ldl) * CG;             // [NB][NB], column p at T + NB p
  float2* dinv = T + NB * NB;                   // [NB]: reciprocals of the block's diagonal (0 for a zero pivot)
  float2* X = dinv + NB;                        // [2][NB][CG]
  float2* tmp = X + 2 * NB * CG;                // [2][2 NB][CG]
  int2* mvs = reinterpret_cast<int2*>(tmp + 4 * NB * CG);  // [2][2 NB]: the moves of the step
  __shared__ int nmv[kSwLists];
  float2* Mb = M + size_t(b) * lay.stride;
  const size_t lda = size_t(lay.lda);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  auto owner = [&](int r) { return (r / NB) & (cl - 1); };
  auto local = [&](int r) { return ((r / NB) >> shift) * NB + r % NB; };
  // this CTA's rows: blocks rank, rank + cl, ...; the matrix's last block may be partial
  const int slots = nblk > rank ? (nblk - rank - 1) / cl + 1 : 0;
  const int lrows = slots * NB - (slots > 0 && ((nblk - 1) & (cl - 1)) == rank ? nblk * NB - n : 0);
  auto global_row = [&](int l) { return (((l / NB) << shift) + rank) * NB + l % NB; };
  auto barrier = [&] {
    if (cl > 1) cluster.sync();
    else __syncthreads();
  };
  // the triangle of block blk (16-byte row pairs: lda is even); zeros beyond a partial block
  auto fetch = [&](int blk) {
    if (blk >= 0 && blk < nblk) {
      const int k = blk * NB, kb = min(NB, n - k);
      for (int idx = tid; idx < NB * (NB / 2); idx += kThreads) {
        const int r = 2 * (idx % (NB / 2)), c = idx / (NB / 2);
        const float2* src = Mb + size_t(k + r) + lda * size_t(k + c);
        if (r + 1 < kb && c < kb) {
          sw_cp_async16(T + c * NB + r, src);
        } else {
          T[c * NB + r] = r < kb && c < kb ? *src : make_float2(0.f, 0.f);
          T[c * NB + r + 1] = make_float2(0.f, 0.f);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the triangle fetched last is there; the reciprocals of its diagonal
  auto prepare = [&] {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (!kForward && tid < NB) {
      const float2 v = T[tid * NB + tid];
      dinv[tid] = (v.x == 0.f && v.y == 0.f) ? make_float2(0.f, 0.f) : cdiv(make_float2(1.f, 0.f), v);
    }
  };
  // row moves of a step (forward): with paired blocks both blocks' moves come before the first block of the pair is
  // solved (the second block's moves only touch rows below the first block)
  auto lists = [&](int blk) {
    const bool pair = w.pair128 && NB == 64;
    return !kForward || blk >= nblk ? 0 : !pair ? 1 : (blk % 2 == 1 ? 0 : (blk + 1 < nblk ? 2 : 1));
  };
  int2 mv_next = make_int2(0, 0);
  int nmv_next = 0;
  const int mq = tid / (2 * NB), mi = tid % (2 * NB);
  auto load_moves = [&](int blk) {
    nmv_next = 0;
    if (mq < lists(blk)) {
      const size_t pidx = size_t(b) * w.npanels + blk + mq;
      nmv_next = w.nperm[pidx];
      mv_next = w.perm[pidx * (2 * NB) + mi];
    }
  };
  auto store_moves = [&] {
    if (mq < kSwLists) {
      mvs[mq * 2 * NB + mi] = mv_next;
      if (mi == 0) nmv[mq] = nmv_next;
    }
  };
  // the first block of this CTA in the order of the sweep
  fetch(kForward ? rank : nblk - 1 - ((nblk - 1 - rank) & (cl - 1)));
#pragma unroll
  for (int c = 0; c < CG; ++c)
    for (int l = tid; l < lrows; l += kThreads)
      Y[c * ldl + l] = c < ncols ? Mb[size_t(global_row(l)) + lda * size_t(n + cg0 + c)] : make_float2(0.f, 0.f);
  load_moves(0);
  store_moves();
  if (((kForward ? 0 : nblk - 1) & (cl - 1)) == rank) prepare();
  barrier();
  for (int step = 0; step < nblk; ++step) {
    const int blk = kForward ? step : nblk - 1 - step, k = blk * NB, kb = min(NB, n - k);
    float2* Xs = X + (step & 1) * NB * CG;
    if constexpr (kForward) {
      for (int q = 0; q < kSwLists; ++q) {
        const int np = nmv[q];
        if (np == 0) continue;
        const int2* pm = mvs + q * 2 * NB;
        float2* buf = tmp + q * 2 * NB * CG;
        for (int idx = tid; idx < np * CG; idx += kThreads) {
          const int2 mv = pm[idx / CG];
          if (owner(mv.y) == rank) {
            float2* dst = buf + idx;
            if (cl > 1) dst = cluster.map_shared_rank(dst, owner(mv.x));
            *dst = Y[(idx % CG) * ldl + local(mv.y)];
          }
        }
        barrier();
        for (int idx = tid; idx < np * CG; idx += kThreads) {
          const int d = pm[idx / CG].x;
          if (owner(d) == rank) Y[(idx % CG) * ldl + local(d)] = buf[idx];
        }
        __syncthreads();
      }
    }
    const bool mine = (blk & (cl - 1)) == rank;
    if (mine) {
      // the block's solve, one warp per column; unrolled, so that the triangle's entries are read ahead of the chain
      if (wid < CG) {
        constexpr int kR = NB / 32;
        float2* y = Y + wid * ldl + (blk >> shift) * NB;
        float2 x[kR];
#pragma unroll
        for (int t = 0; t < kR; ++t) x[t] = lane + 32 * t < kb ? y[lane + 32 * t] : make_float2(0.f, 0.f);
#pragma unroll
        for (int pp = 0; pp < NB; ++pp) {
          const int p = kForward ? pp : NB - 1 - pp, ot = p >> 5, ol = p & 31;
          if constexpr (!kForward)
            if (lane == ol) x[ot] = cmul(x[ot], dinv[p]);
          const float2 xp = make_float2(__shfl_sync(0xffffffffu, x[ot].x, ol), __shfl_sync(0xffffffffu, x[ot].y, ol));
#pragma unroll
          for (int t = 0; t < kR; ++t) {
            if (kForward ? t < ot : t > ot) continue;
            const int i = lane + 32 * t;
            if (t != ot || (kForward ? i > p : i < p)) cfms(x[t], T[p * NB + i], xp);
          }
        }
#pragma unroll
        for (int t = 0; t < kR; ++t) {
          const int i = lane + 32 * t;
          if (i < kb) {
            y[i] = x[t];
            for (int q = 0; q < cl; ++q) {
              float2* dst = Xs + i * CG + wid;
              if (cl > 1) dst = cluster.map_shared_rank(dst, q);
              *dst = x[t];
            }
          }
        }
      }
    }
    // rows of the blocks still to be solved
    const int l_begin = kForward ? (blk >= rank ? ((blk - rank) >> shift) + 1 : 0) * NB : 0;
    const int l_end = kForward ? lrows : (blk > rank ? ((blk - rank - 1) >> shift) + 1 : 0) * NB;
    SweepUpdate<NB, CG, kThreads> up(Mb + lda * size_t(k), lda, kb, l_begin, l_end, rank, shift);
    const int next = kForward ? blk + 1 : blk - 1;
    const bool mine_next = next >= 0 && next < nblk && (next & (cl - 1)) == rank;
    if (cl > 1 && mine_next) prepare();  // while the owner solves
    barrier();
    if (mine) fetch(kForward ? blk + cl : blk - cl);
    if constexpr (kForward) load_moves(blk + 1);
    up.run(Xs, Y, ldl);
    if constexpr (kForward) store_moves();
    if (cl == 1 && mine_next) prepare();
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  for (int c = 0; c < ncols; ++c)
    for (int l = tid; l < lrows; l += kThreads) Mb[size_t(global_row(l)) + lda * size_t(n + cg0 + c)] = Y[c * ldl + l];
}

constexpr size_t kSwSmemBudget = 224 * 1024;

template <bool kForward, int NB, int CG, int kThreads>
bool launch_sweep_threads(const BatchLayout& lay, int batch, int groups, int shift, size_t smem, float2* M,
                          const LuWork& w, const int* skip, cudaStream_t s) {
  auto kern = sweep_kernel<kForward, NB, CG, kThreads>;
  ensure_smem_limit(reinterpret_cast<const void*>(kern), smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(groups) << shift, unsigned(batch), 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1u << shift;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  count_launch();
  cudaLaunchKernelEx(&cfg, kern, lay, M, w, shift, skip);
  return true;
}

template <bool kForward, int NB, int CG>
bool launch_sweep_cg(const BatchLayout& lay, int batch, float2* M, const LuWork& w, const int* skip, cudaStream_t s) {
  const int groups = (lay.m + CG - 1) / CG, sms = current_sm_count();
  int shift = 0;
  while (shift < 3 && SweepSmem<NB, CG>::bytes(lay.n, 1 << shift) > kSwSmemBudget) ++shift;
  // More CTAs while there are fewer than four an SM and each keeps some 512 rows.  Backward / forward sweep, 1 CTA of 512
  // threads against a cluster: n = 4112 x 12, 16 columns 2.14 / 1.81 ms (4 columns a CTA), 8 CTAs 0.98 / 1.02; n = 2256
  // x 100 2.29 / 1.88, 2 CTAs 1.87 / 1.90, 4 CTAs 1.59 / 1.62; n = 1392 x 60 0.56 / 0.44, 2 CTAs 0.40 / 0.40, 4 CTAs
  // 0.53 / 0.52; n = 688 x 60 0.14 / 0.14, 2 CTAs 0.14 / 0.15.
  while (shift < 3 && (long long)groups * batch << shift < 4 * sms && lay.n >= (1024 << shift)) ++shift;
  const size_t smem = SweepSmem<NB, CG>::bytes(lay.n, 1 << shift);
  if (smem > kSwSmemBudget) return false;
  if constexpr (NB == 64)
    if (shift > 0) return launch_sweep_threads<kForward, NB, CG, 256>(lay, batch, groups, shift, smem, M, w, skip, s);
  return launch_sweep_threads<kForward, NB, CG, 512>(lay, batch, groups, shift, smem, M, w, skip, s);
}

// 64-row blocks: 8 right-hand sides a cluster; 4 where there are no more, or where 8 leave one CTA an SM and 4 two
// (n = 15000 x 4, 25 columns: 12.8 ms with 8, two rounds of 16 clusters, 6.6 ms with 4).
template <bool kForward>
bool launch_sweep64(const BatchLayout& lay, int batch, float2* M, const LuWork& w, const int* skip, cudaStream_t s) {
  constexpr size_t kTwoPerSm = 113 * 1024;
  const bool four = lay.m <= 4 || (SweepSmem<64, 8>::bytes(lay.n, 8) > kTwoPerSm &&
                                   SweepSmem<64, 4>::bytes(lay.n, 8) <= kTwoPerSm);
  return (!four && launch_sweep_cg<kForward, 64, 8>(lay, batch, M, w, skip, s)) ||
         launch_sweep_cg<kForward, 64, 4>(lay, batch, M, w, skip, s);
}

}  // namespace

bool fused_forward_sweep(int nb, const BatchLayout& lay, int batch, float2* M, const LuWork& w, const int* skip,
                         cudaStream_t s) {
  if (nb == 64) return launch_sweep64<true>(lay, batch, M, w, skip, s);
  if (nb == 32) return launch_sweep_cg<true, 32, 8>(lay, batch, M, w, skip, s);
  return false;
}

bool fused_backward_sweep(int nb, const BatchLayout& lay, int batch, float2* M, const int* skip, cudaStream_t s) {
  if (nb == 64) return launch_sweep64<false>(lay, batch, M, LuWork(), skip, s);
  if (nb == 32) return launch_sweep_cg<false, 32, 8>(lay, batch, M, LuWork(), skip, s);
  return false;
}

}  // namespace rfx
