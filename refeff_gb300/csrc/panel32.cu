// Panel factorisation of the FP32 elimination with the panel in registers: the
// rows [k, n) are split over a thread-block cluster, a thread holds one or two
// rows of all NB columns, and nothing but pivot candidates goes through shared
// memory.  A column is a chain of latencies (rank, reduce, barrier, select,
// update), so the kernel shortens the chain:
//
//   * every warp writes its candidate (rank and row) into all CTAs of the
//     cluster before the barrier and keeps the candidate's entries in its own
//     CTA, so one barrier a column suffices, and the selection reads local
//     memory only;
//   * ranks are compared as integers with redux instead of shuffle trees;
//   * multipliers are products with the pivot's reciprocal;
//   * a row's entries rotate by one register a column (entry 0 is the current
//     column, finished multipliers come in at the end), so that the loop over
//     columns stays rolled and 15, 7, 3 or 1 columns are updated without branches;
//   * only rows that start among the panel's first NB positions can be displaced
//     without being pivots, so the row bookkeeping is NB entries in shared
//     memory, kept by one thread of every CTA, off the other warps' path.
//
// The factors do not depend on the cluster size.  panel_kernel (batched_lu.cu),
// which keeps the panel in shared memory, serves the panels too tall for this one.
#include <cooperative_groups.h>
#include <algorithm>
#include <climits>
#include <type_traits>
#include "batched_lu.cuh"
#include "cplx.cuh"

namespace cg = cooperative_groups;

namespace rfx {

namespace {

constexpr int kMaxThreads = 512, kMaxWarps = kMaxThreads / 32;

// |re| + |im| as an ordered integer; a NaN competes as zero, so that a valid row is always chosen
__device__ __forceinline__ uint32_t rank_of(float2 v) {
  const uint32_t b = __float_as_uint(cabs1(v)) & 0x7fffffffu;
  return b > 0x7f800000u ? 0u : b;
}
// no candidate: rank 0 in row INT_MAX, which loses to any row
__device__ __forceinline__ void rank_merge(uint32_t& v, int& r, uint32_t ov, int orow) {
  if (ov > v || (ov == v && orow < r)) { v = ov; r = orow; }
}
// the largest rank of the warp and the lowest row that has it, in every lane
__device__ __forceinline__ void rank_warp(uint32_t& v, int& r) {
  const uint32_t m = __reduce_max_sync(0xffffffffu, v);
  r = __reduce_min_sync(0xffffffffu, v == m ? r : INT_MAX);
  v = m;
}

template <int NB, int kRpt, int kThreadsMax, int kBlocks>
__global__ void __launch_bounds__(kThreadsMax, kBlocks)
    panel32_kernel(BatchLayout lay, int k, float2* __restrict__ M, LuWork w) {
  cg::cluster_group cluster = cg::this_cluster();
  const int CL = int(cluster.num_blocks()), rank = int(cluster.block_rank());
  const int b = blockIdx.y, n = lay.n, R = n - k, kb = min(NB, R), panel = k / NB;
  const int rpc = (R + CL - 1) / CL, row_lo = rank * rpc;
  const int nloc = max(0, min(R, row_lo + rpc) - row_lo);
  const int threads = int(blockDim.x), warps = threads / 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  __shared__ uint2 slots[2][16 * kMaxWarps];          // (rank, row) of every warp of the cluster, by column parity
  // this CTA's candidates' entries from the current column on (zero past the panel's last)
  __shared__ __align__(16) float2 cand[2][kMaxWarps][NB];
  __shared__ __align__(16) float2 ubuf[kMaxWarps][NB];
  __shared__ int piv[NB], tpos[NB], occ[NB];          // pivot rows; position of top row i; top row at position i
  __shared__ int nmoves;

  const size_t lda = size_t(lay.lda);
  float2* Mb = M + size_t(b) * lay.stride + size_t(k) + lda * size_t(k);
  // x[i][q]: column (j + q) mod NB of row tid + i threads, j the current column
  float2 x[kRpt][NB];
  int state[kRpt];     // -1 open, j pivot of column j, NB no row
#pragma unroll
  for (int i = 0; i < kRpt; ++i) {
    const int r = tid + i * threads;
    state[i] = r < nloc ? -1 : NB;
#pragma unroll
    for (int q = 0; q < NB; ++q) x[i][q] = r < nloc && q < kb ? Mb[size_t(row_lo + r) + lda * q] : make_float2(0.f, 0.f);
  }
  for (int i = tid; i < NB; i += threads) tpos[i] = occ[i] = i;
  if (tid == 0) nmoves = 0;
  __syncthreads();
  const uint32_t magic = 0xffffffffu / uint32_t(rpc) + 1u;  // row / rpc for rows below 65536 as a high product

#pragma unroll 1
  for (int j = 0; j < kb; ++j) {
    const int par = j & 1, left = kb - j;
    uint32_t wv = 0;
    int wrow = INT_MAX;
#pragma unroll
    for (int i = 0; i < kRpt; ++i)
      if (state[i] < 0) rank_merge(wv, wrow, rank_of(x[i][0]), row_lo + tid + i * threads);
    rank_warp(wv, wrow);
#pragma unroll
    for (int i = 0; i < kRpt; ++i)
      if (state[i] < 0 && row_lo + tid + i * threads == wrow) {
#pragma unroll
        for (int q = 0; q < NB; ++q) cand[par][wid][q] = q < left ? x[i][q] : make_float2(0.f, 0.f);
      }
    if (lane < CL) {
      uint2* dst = &slots[par][rank * warps + wid];
      if (CL > 1) dst = cluster.map_shared_rank(dst, lane);
      *dst = make_uint2(wv, uint32_t(wrow));
    }
    if (CL > 1) cluster.sync();
    else __syncthreads();
    wv = 0;
    wrow = INT_MAX;
    for (int q = lane; q < CL * warps; q += 32) rank_merge(wv, wrow, slots[par][q].x, int(slots[par][q].y));
    rank_warp(wv, wrow);
    wrow = min(wrow, R - 1);  // always a row of the panel: every open row ranks at least zero
    const int owner = int(__umulhi(uint32_t(wrow), magic)), lr = wrow - owner * rpc;
    const float2* us = &cand[par][(lr % threads) / 32][0];
    if (CL > 1) {
      const float2* src = cluster.map_shared_rank(us, owner);
      if (lane < NB) ubuf[wid][lane] = src[lane];
      us = &ubuf[wid][0];
      __syncwarp();
    }
    if (tid == threads - 1) {
      piv[j] = wrow;
      // the pivot sits at its own index unless it is a displaced top row; the row at position j takes its place
      const int q = wrow < NB ? tpos[wrow] : wrow, pj = occ[j];
      if (pj != wrow) {
        tpos[pj] = q;
        if (q < NB) occ[q] = pj;
      }
      if (rank == 0) {
        w.ipiv[size_t(b) * n + k + j] = k + q;
        if (wv == 0) {
          atomicMax(w.status + b, int(kDevSingular));
          atomicCAS(w.info + b, 0, k + j + 1);
        }
      }
    }
    // multipliers by the pivot's reciprocal (by division where |pivot|^2 could leave the FP32 range, zero for a zero or
    // NaN pivot)
    const float2 u0 = us[0];
    const int field = int(max(__float_as_uint(u0.x) & 0x7fffffffu, __float_as_uint(u0.y) & 0x7fffffffu) >> 23);
    const int mode = wv == 0 ? 0 : field > 127 - 60 && field < 127 + 60 ? 1 : 2;
    float2 pr = u0;
    if (mode == 1) {
      const float inv = 1.0f / fmaf(u0.x, u0.x, u0.y * u0.y);
      pr = make_float2(u0.x * inv, -u0.y * inv);
    }
#pragma unroll
    for (int i = 0; i < kRpt; ++i) {
      if (state[i] < 0 && row_lo + tid + i * threads == wrow) state[i] = j;
      // a row that is a pivot already only rotates: multiplier 0, its own entry comes in at the end
      const float2 l = state[i] >= 0 || mode == 0 ? make_float2(0.f, 0.f) : mode == 1 ? cmul(x[i][0], pr) : cdiv(x[i][0], pr);
      const float2 last = state[i] >= 0 ? x[i][0] : l;
      auto columns = [&](auto count) {
        constexpr int kCount = decltype(count)::value;
#pragma unroll
        for (int q = 1; q < NB; ++q) {
          float2 v = x[i][q];
          if (q <= kCount) cfms(v, l, us[q]);
          x[i][q - 1] = v;
        }
        x[i][NB - 1] = last;
      };
      if (NB > 16 && left > 16) columns(std::integral_constant<int, NB - 1>());
      else if (left > 8) columns(std::integral_constant<int, 15>());
      else if (left > 4) columns(std::integral_constant<int, 7>());
      else if (left > 2) columns(std::integral_constant<int, 3>());
      else columns(std::integral_constant<int, 1>());
    }
  }
  // a narrower last panel turns on to the full circle
#pragma unroll 1
  for (int j = kb; j < NB; ++j)
#pragma unroll
    for (int i = 0; i < kRpt; ++i) {
      const float2 first = x[i][0];
#pragma unroll
      for (int q = 1; q < NB; ++q) x[i][q - 1] = x[i][q];
      x[i][NB - 1] = first;
    }
  // no CTA leaves while another may read its candidates; and the bookkeeping is complete
  if (CL > 1) cluster.sync();
  else __syncthreads();
#pragma unroll
  for (int i = 0; i < kRpt; ++i) {
    const int r = tid + i * threads;
    if (r >= nloc) continue;
    const int row = row_lo + r, dst = state[i] >= 0 ? state[i] : row < NB ? tpos[row] : row;
#pragma unroll
    for (int q = 0; q < NB; ++q)
      if (q < kb) Mb[size_t(dst) + lda * q] = x[i][q];
  }
  if (rank == 0) {
    // the panel's row moves: pivots to their positions, displaced top rows to theirs
    int2* pm = w.perm + (size_t(b) * w.npanels + panel) * (2 * NB);
    for (int t = tid; t < 2 * NB; t += threads) {
      int dst = 0, src = 0;
      if (t < NB) {
        if (t < kb) {
          dst = t;
          src = piv[t];
        }
      } else if (t - NB < R) {
        src = t - NB;
        dst = tpos[src];
        for (int j = 0; j < kb; ++j)
          if (piv[j] == src) dst = src;  // a pivot: listed above
      }
      if (dst != src) pm[atomicAdd(&nmoves, 1)] = make_int2(k + dst, k + src);
    }
    __syncthreads();
    if (tid == 0) w.nperm[size_t(b) * w.npanels + panel] = nmoves;
  }
}

template <int NB, int kRpt, int kThreadsMax, int kBlocks>
cudaError_t launch_shape(int cl, int rows, const BatchLayout& lay, int batch, int k, float2* M, const LuWork& w,
                         cudaStream_t s) {
  auto kern = panel32_kernel<NB, kRpt, kThreadsMax, kBlocks>;
  if (cl > 8) {
    const cudaError_t err = ensure_nonportable_clusters(reinterpret_cast<const void*>(kern));
    if (err != cudaSuccess) return err;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(cl), unsigned(batch), 1);
  cfg.blockDim = dim3(unsigned(std::max(32, ((rows + kRpt - 1) / kRpt + 31) / 32 * 32)), 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(cl);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kern, lay, k, M, w);
}

}  // namespace

// Rows a CTA can hold in registers.
constexpr int kRows16 = 1024, kRows32 = 512;

cudaError_t launch_panel32(int nb, int max_cluster, const BatchLayout& lay, int batch, int k, float2* M,
                           const LuWork& w, cudaStream_t s, bool& served) {
  const int R = lay.n - k, cap = nb == 16 ? kRows16 : kRows32;
  served = (nb == 16 || nb == 32) && (R + max_cluster - 1) / max_cluster <= cap;
  if (!served) return cudaSuccess;
  const int sms = current_sm_count();
  int cl = 1;
  while (cl < max_cluster && (R + cl - 1) / cl > cap) cl *= 2;
  while (cl < 8 && R > 256 * cl && (long long)batch * cl * 2 <= sms) cl *= 2;
  const int rows = (R + cl - 1) / cl;
  // two smaller CTAs per SM (96 registers) where there are more CTAs than SMs
  if (nb == 32 && rows <= 320 && (long long)batch * cl > sms) return launch_shape<32, 1, 320, 2>(cl, rows, lay, batch, k, M, w, s);
  if (nb == 32) return launch_shape<32, 1, 512, 1>(cl, rows, lay, batch, k, M, w, s);
  if (rows <= 512) return launch_shape<16, 1, 512, 2>(cl, rows, lay, batch, k, M, w, s);
  return launch_shape<16, 2, 512, 1>(cl, rows, lay, batch, k, M, w, s);
}

}  // namespace rfx
