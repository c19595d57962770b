// Panel factorisation of the FP64 elimination: the (n - k) x NB panel in the
// distributed shared memory of a thread-block cluster, like panel_kernel of the
// FP32 form (batched_lu.cu), but built around GB300's FP64 rate of two
// multiply-adds per SM and cycle, which a plain right-looking panel saturates
// (measured at n = 304: 180 us for 32 columns, the same with one row per thread
// as with two).
//
//   * the panel is taken in blocks of 8 columns: the rank-1 updates stay inside
//     the block (3.5 columns of FP64 multiply-adds on average instead of 15.5),
//     and the block's rank-8 update of the remaining columns runs on the tensor
//     path in exact 8-bit digit products (digits64.cuh, mma.sync on 16-row tiles
//     that lie at the same rows whatever the cluster size, so that the result
//     does not depend on it);
//   * the pivot's reciprocal is formed once per column, by one thread, instead
//     of two divisions per row;
//   * pivot candidates are ranked as integers (the bit patterns of non-negative
//     doubles), not by comparisons on the FP64 pipe.
//
// Pivot rule, ties, row bookkeeping and outputs are those of panel_kernel.
#include <cooperative_groups.h>
#include <climits>
#include "batched_lu.cuh"
#include "cplx.cuh"
#include "digits64.cuh"

namespace cg = cooperative_groups;

namespace rfx {

namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kSub = 8;  // columns per block

// |re| + |im| as an ordered, non-negative integer; a NaN (whose sign bit may be set) competes as zero, so that a valid
// row is always chosen
__device__ __forceinline__ long long rank_of(double2 v) {
  const long long b = __double_as_longlong(cabs1(v)) & 0x7fffffffffffffffll;
  return b > 0x7ff0000000000000ll ? 0 : b;
}
__device__ __forceinline__ void rank_merge(long long& v, int& r, long long ov, int orow) {
  if (ov > v || (ov == v && orow < r)) { v = ov; r = orow; }
}
struct alignas(16) RankSlot {
  long long val;
  int row;
};

template <int NB>
__global__ void __launch_bounds__(kThreads) panel64_kernel(BatchLayout lay, int k, double2* __restrict__ M, LuWork w,
                                                           int rpc_max) {
  constexpr int kRest = NB > kSub ? NB - kSub : 1;        // most columns a block updates
  constexpr int kGroups = (kRest + 7) / 8;
  cg::cluster_group cluster = cg::this_cluster();
  const int CL = int(cluster.num_blocks());
  const int rank = int(cluster.block_rank());
  const int b = blockIdx.y;
  const int n = lay.n;
  const int R = n - k;
  const int kb = min(NB, R);
  const int panel = k / NB;
  const int rpc = ((R + CL - 1) / CL + 15) / 16 * 16;  // whole 16-row tiles
  const int row_lo = rank * rpc;
  const int nloc = max(0, min(R, row_lo + rpc) - row_lo);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;

  extern __shared__ __align__(16) unsigned char smraw[];
  double2* pan = reinterpret_cast<double2*>(smraw);
  double2* urow = pan + size_t(NB) * rpc_max;                 // pivot row; then one unused slot's width of padding
  int* done = reinterpret_cast<int*>(urow + NB) + 8;
  const bool pos_global = w.pos_scratch != nullptr;
  int* row2pos = pos_global ? w.pos_scratch + size_t(b) * 2 * n : done + rpc_max;
  int* pos2row = row2pos + n;
  int* scratch = pos_global ? done + rpc_max : pos2row + n;  // [2] move count
  __shared__ RankSlot wslot[2][kWarps];
  __shared__ double2 prec;          // the pivot's reciprocal, or the pivot itself where that would leave the range
  __shared__ int pmode;             // 0 zero pivot, 1 reciprocal, 2 division
  __shared__ int piv[kSub];         // the block's pivot rows
  __shared__ double2 L11[kSub][kSub], U12[kSub][kRest];
  __shared__ uint32_t words[kGroups][2 * kDig * 32];
  __shared__ int ecol[kGroups][8];

  double2* Mb = M + size_t(b) * lay.stride;
  for (int idx = tid; idx < nloc * kb; idx += kThreads) {
    const int r = idx % nloc, c = idx / nloc;
    pan[size_t(c) * rpc_max + r] = Mb[size_t(k + row_lo + r) + size_t(lay.lda) * (k + c)];
  }
  for (int r = tid; r < nloc; r += kThreads) done[r] = 0;
  if (rank == 0) {
    for (int q = tid; q < R; q += kThreads) { row2pos[q] = q; pos2row[q] = q; }
    if (tid == 0) scratch[2] = 0;
  }
  __syncthreads();

  long long best = -1;
  int brow = INT_MAX;
  for (int c0 = 0; c0 < kb; c0 += kSub) {
    const int ce = min(c0 + kSub, kb);
    best = -1;
    brow = INT_MAX;
    for (int r = tid; r < nloc; r += kThreads)
      if (!done[r]) rank_merge(best, brow, rank_of(pan[size_t(c0) * rpc_max + r]), row_lo + r);
    for (int j = c0; j < ce; ++j) {
      for (int off = 16; off > 0; off >>= 1) {
        const long long ov = __shfl_down_sync(0xffffffffu, best, off);
        const int orow = __shfl_down_sync(0xffffffffu, brow, off);
        rank_merge(best, brow, ov, orow);
      }
      if (lane == 0) {
        wslot[j & 1][wid].val = best;
        wslot[j & 1][wid].row = brow;
      }
      cluster.sync();
      if (j == c0 && c0 > 0) {
        // the previous block's rows of U beyond its columns, now that no CTA reads their old values any more
        for (int idx = tid; idx < kSub * (kb - c0); idx += kThreads) {
          const int p = idx % kSub, c = idx / kSub, own = piv[p] / rpc;
          if (own == rank) pan[size_t(c0 + c) * rpc_max + (piv[p] - row_lo)] = U12[p][c];
        }
        __syncthreads();  // piv is written again below
      }
      long long wv = -1;
      int wrow = INT_MAX;
      for (int q = lane; q < CL * kWarps; q += 32) {
        const RankSlot* rs = cluster.map_shared_rank(&wslot[j & 1][0], q / kWarps);
        rank_merge(wv, wrow, rs[q % kWarps].val, rs[q % kWarps].row);
      }
      for (int off = 16; off > 0; off >>= 1) {
        const long long ov = __shfl_xor_sync(0xffffffffu, wv, off);
        const int orow = __shfl_xor_sync(0xffffffffu, wrow, off);
        rank_merge(wv, wrow, ov, orow);
      }
      wrow = min(wrow, R - 1);  // always a row of the panel: every undecided row ranks at least zero
      const int owner = wrow / rpc, lr = wrow % rpc;
      const double2* opan = cluster.map_shared_rank(pan, owner);
      if (tid < ce - j) {
        const double2 v = opan[size_t(j + tid) * rpc_max + lr];
        urow[j + tid] = v;
        if (tid == 0) {
          const double d = v.x * v.x + v.y * v.y;
          if (!(cabs1(v) > 0.0)) {
            pmode = 0;
          } else if (d > 1e-280 && d < 1e280) {
            pmode = 1;
            prec = make_double2(v.x / d, -v.y / d);
          } else {
            pmode = 2;
            prec = v;
          }
          piv[j - c0] = wrow;
        }
      }
      if (rank == owner && tid == lr % kThreads) done[lr] = 1;
      if (rank == 0 && tid == kThreads - 1) {
        const int q = row2pos[wrow];
        const int pj = pos2row[j];
        pos2row[j] = wrow;
        pos2row[q] = pj;
        row2pos[wrow] = j;
        row2pos[pj] = q;
        w.ipiv[size_t(b) * n + k + j] = k + q;
        if (!(wv > 0)) {
          atomicMax(w.status + b, int(kDevSingular));
          atomicCAS(w.info + b, 0, k + j + 1);
        }
      }
      __syncthreads();
      // multipliers, rank-1 update of the block's own columns, and the local arg-max of column j + 1
      const double2 pr = prec;
      const int mode = pmode;
      best = -1;
      brow = INT_MAX;
      for (int r = tid; r < nloc; r += kThreads) {
        if (done[r]) continue;
        double2 l = pan[size_t(j) * rpc_max + r];
        l = mode == 1 ? cmul(l, pr) : mode == 2 ? cdiv(l, pr) : make_double2(0.0, 0.0);
        pan[size_t(j) * rpc_max + r] = l;
        for (int c = j + 1; c < ce; ++c) {
          double2 v = pan[size_t(c) * rpc_max + r];
          cfms(v, l, urow[c]);
          pan[size_t(c) * rpc_max + r] = v;
          if (c == j + 1) rank_merge(best, brow, rank_of(v), row_lo + r);
        }
      }
    }
    if constexpr (NB > kSub) {
      const int rest = kb - ce;
      if (rest <= 0) break;
      // U12 = L11^-1 A12 of the block's pivot rows, in every CTA: their multipliers and untouched columns have been
      // final since the barrier of the block's last column
      __syncthreads();
      for (int idx = tid; idx < kSub * (kSub + rest); idx += kThreads) {
        const int p = idx % kSub, c = idx / kSub;
        const double2* src = cluster.map_shared_rank(pan, piv[p] / rpc) + piv[p] % rpc;
        if (c < kSub) L11[p][c] = src[size_t(c0 + c) * rpc_max];
        else U12[p][c - kSub] = src[size_t(ce + c - kSub) * rpc_max];
      }
      __syncthreads();
      if (tid < rest) {
        double2 x[kSub];
#pragma unroll
        for (int p = 0; p < kSub; ++p) x[p] = U12[p][tid];
#pragma unroll
        for (int p = 0; p < kSub; ++p)
#pragma unroll
          for (int q = p + 1; q < kSub; ++q) cfms(x[q], L11[q][p], x[p]);
#pragma unroll
        for (int p = 0; p < kSub; ++p) U12[p][tid] = x[p];
      }
      __syncthreads();
      const int groups = (rest + 7) / 8, g = lane >> 2, t = lane & 3;
      if (wid < groups) {
        double2 v[2];
#pragma unroll
        for (int q = 0; q < 2; ++q)
          v[q] = 8 * wid + g < rest ? U12[2 * t + q][8 * wid + g] : make_double2(0.0, 0.0);
        cut_tile_b(v, words[wid], ecol[wid]);
      }
      __syncthreads();
      for (int tile = wid; tile * 16 < nloc; tile += kWarps) {
        const int r0 = tile * 16;
        double2 v[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int r = r0 + g + 8 * h;
            v[h][q] = r < nloc && !done[r] ? pan[size_t(c0 + 2 * t + q) * rpc_max + r] : make_double2(0.0, 0.0);
          }
        DigitTileA a;
        const bool fits = cut_tile_a(v, a);
        for (int gr = 0; gr < groups; ++gr) {
          int bad = 0;
#pragma unroll
          for (int q = 0; q < 8; ++q) bad |= ecol[gr][q] == kNonfinite;
          double2 p[2][2];
          if (fits && !bad) {
            tile_product(a, words[gr], ecol[gr], p);
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const int r = r0 + g + 8 * h, c = 8 * gr + 2 * t + q;
                p[h][q] = make_double2(0.0, 0.0);
                if (r < nloc && !done[r] && c < rest)
                  for (int i = 0; i < kSub; ++i) cfma(p[h][q], pan[size_t(c0 + i) * rpc_max + r], U12[i][c]);
              }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int r = r0 + g + 8 * h, c = 8 * gr + 2 * t + q;
              if (r < nloc && !done[r] && c < rest) {
                double2& z = pan[size_t(ce + c) * rpc_max + r];
                z = csub(z, p[h][q]);
              }
            }
        }
      }
      __syncthreads();
    }
  }
  cluster.sync();
  // write back in pivoted order; rank 0 publishes the row moves of this panel
  const int* r2p0 = pos_global ? row2pos : cluster.map_shared_rank(row2pos, 0);
  for (int idx = tid; idx < nloc * kb; idx += kThreads) {
    const int r = idx % nloc, c = idx / nloc;
    const int dst = k + r2p0[row_lo + r];
    Mb[size_t(dst) + size_t(lay.lda) * (k + c)] = pan[size_t(c) * rpc_max + r];
  }
  if (rank == 0) {
    int2* pm = w.perm + (size_t(b) * w.npanels + panel) * (2 * NB);
    for (int q = tid; q < R; q += kThreads) {
      if (pos2row[q] != q) {
        const int si = atomicAdd(&scratch[2], 1);
        if (si < 2 * NB) pm[si] = make_int2(k + q, k + pos2row[q]);
      }
    }
    __syncthreads();
    if (tid == 0) w.nperm[size_t(b) * w.npanels + panel] = min(scratch[2], 2 * NB);
  }
  cluster.sync();
}

template <int NB>
cudaError_t launch_panel64_nb(const PanelConfig& pc, const BatchLayout& lay, int batch, int k, double2* M,
                              const LuWork& w, cudaStream_t s) {
  auto kern = panel64_kernel<NB>;
  cudaError_t err = ensure_smem_limit(reinterpret_cast<const void*>(kern), size_t(pc.smem));
  if (err != cudaSuccess) return err;
  if (pc.cluster > 8) {
    err = ensure_nonportable_clusters(reinterpret_cast<const void*>(kern));
    if (err != cudaSuccess) return err;
  }
  // the smallest cluster whose CTAs hold the trailing rows in whole 16-row tiles
  int cl = pc.cluster;
  const int R = lay.n - k;
  while (cl > 1 && ((R + cl / 2 - 1) / (cl / 2) + 15) / 16 * 16 <= pc.rpc_max) cl /= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(cl), unsigned(batch), 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = size_t(pc.smem);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(cl);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kern, lay, k, M, w, pc.rpc_max);
}

}  // namespace

cudaError_t launch_panel64(const PanelConfig& pc, int nb, const BatchLayout& lay, int batch, int k, double2* M,
                           const LuWork& w, cudaStream_t s) {
  switch (nb) {
    case 32: return launch_panel64_nb<32>(pc, lay, batch, k, M, w, s);
    case 16: return launch_panel64_nb<16>(pc, lay, batch, k, M, w, s);
    case 8: return launch_panel64_nb<8>(pc, lay, batch, k, M, w, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace rfx
