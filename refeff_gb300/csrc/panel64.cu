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
//     does not depend on it), with FP64 multiply-adds for the sums that the
//     digits' grid may have lost (structural zeros, sparse or badly scaled
//     systems: a panel of 688 rows takes 115 us without such sums, up to 180
//     with many);
//   * the block's columns of a thread's row stay in registers (NB = 32; the
//     narrower panels of large systems hold several rows a thread and work in
//     shared memory); each warp publishes its pivot candidate's row with its
//     rank, so a column takes one (cluster) barrier;
//   * multipliers are products with the pivot's reciprocal (7 FP64 operations a
//     column) instead of two divisions per row;
//   * pivot candidates are ranked as integers (the bit patterns of non-negative
//     doubles), not by comparisons on the FP64 pipe.
//
// Pivot rule, ties, row bookkeeping and outputs are those of panel_kernel.
#include <cooperative_groups.h>
#include <algorithm>
#include <climits>
#include <type_traits>
#include "batched_lu.cuh"
#include "cplx.cuh"
#include "digits64.cuh"

namespace cg = cooperative_groups;

namespace rfx {

namespace {

constexpr int kSub = 8;  // columns per block
// |re| + |im| as an ordered, non-negative integer; a NaN (whose sign bit may be set) competes as zero, so that a valid
// row is always chosen
__device__ __forceinline__ unsigned long long rank_of(double2 v) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(cabs1(v))) & 0x7fffffffffffffffull;
  return b > 0x7ff0000000000000ull ? 0 : b;
}
// no candidate: rank 0 in row INT_MAX, which loses to any row
__device__ __forceinline__ void rank_merge(unsigned long long& v, int& r, unsigned long long ov, int orow) {
  if (ov > v || (ov == v && orow < r)) { v = ov; r = orow; }
}
// the largest rank of the warp and the lowest row that has it, in every lane
__device__ __forceinline__ void rank_warp(unsigned long long& v, int& r) {
  const uint32_t hi = uint32_t(v >> 32), lo = uint32_t(v);
  const uint32_t mh = __reduce_max_sync(0xffffffffu, hi);
  const uint32_t ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  r = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? r : INT_MAX);
  v = (static_cast<unsigned long long>(mh) << 32) | ml;
}
struct alignas(16) RankSlot {
  unsigned long long val;
  int row;
};
// kRpt rows per thread: kRpt * blockDim.x >= rpc_max, blockDim.x <= kMaxThreads
template <int NB, int kMaxThreads, int kRpt>
__global__ void __launch_bounds__(kMaxThreads, kMaxThreads == 256 ? 2 : 1)
    panel64_kernel(BatchLayout lay, int k, double2* __restrict__ M, LuWork w, int rpc_max) {
  constexpr int kMaxWarps = kMaxThreads / 32;
  const int kThreads = int(blockDim.x), kWarps = kThreads / 32;
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
  int* done = reinterpret_cast<int*>(pan + size_t(NB) * rpc_max + NB) + 8;
  const bool pos_global = w.pos_scratch != nullptr;
  int* row2pos = pos_global ? w.pos_scratch + size_t(b) * 2 * n : done + rpc_max;
  int* pos2row = row2pos + n;
  int* scratch = pos_global ? done + rpc_max : pos2row + n;  // [2] move count
  // candidates of every warp of the cluster (each warp writes its own into all CTAs), by column parity, and this CTA's
  // candidates' entries from the current column on
  __shared__ RankSlot wslot[2][16 * kMaxWarps];
  __shared__ double2 wrowv[2][kMaxWarps][kSub];
  __shared__ double2 ubuf[kMaxWarps][kSub];
  __shared__ int pivs[2][kSub];                  // the block's pivot rows, by block parity
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

  // a single CTA needs no cluster barrier
  auto sync_all = [&] {
    if (CL > 1) cluster.sync();
    else __syncthreads();
  };
  // wrow / rpc for wrow < 65536 as a high product
  const uint32_t magic = 0xffffffffu / uint32_t(rpc) + 1u;
  bool open[kRpt];  // rows of this thread that are not pivots yet
#pragma unroll
  for (int i = 0; i < kRpt; ++i) open[i] = tid + i * kThreads < nloc;
  for (int c0 = 0; c0 < kb; c0 += kSub) {
    const int ce = min(c0 + kSub, kb);
    int* const piv = pivs[(c0 / kSub) & 1];
    // x[i][q]: column j + q of row tid + i kThreads, j the current column (in the panel itself where a thread has more
    // rows than fit in registers)
    constexpr bool kRegs = kRpt == 1;
    double2 x[kRegs ? kRpt : 1][kSub];
    if constexpr (kRegs)
#pragma unroll
      for (int i = 0; i < kRpt; ++i)
#pragma unroll
        for (int q = 0; q < kSub; ++q)
          x[i][q] = open[i] && c0 + q < ce ? pan[size_t(c0 + q) * rpc_max + tid + i * kThreads] : make_double2(0.0, 0.0);
#pragma unroll 1
    for (int j = c0; j < ce; ++j) {
      const int par = j & 1, left = ce - j;
      auto entry = [&](int i, int q) {
        if constexpr (kRegs) return x[i][q];
        else return q < left ? pan[size_t(j + q) * rpc_max + tid + i * kThreads] : make_double2(0.0, 0.0);
      };
      unsigned long long wv = 0;
      int wrow = INT_MAX;
#pragma unroll
      for (int i = 0; i < kRpt; ++i)
        if (open[i]) rank_merge(wv, wrow, rank_of(entry(i, 0)), row_lo + tid + i * kThreads);
      rank_warp(wv, wrow);
#pragma unroll
      for (int i = 0; i < kRpt; ++i)
        if (row_lo + tid + i * kThreads == wrow && open[i])
#pragma unroll
          for (int q = 0; q < kSub; ++q) wrowv[par][wid][q] = entry(i, q);
      if (lane < CL) {
        RankSlot* dst = &wslot[par][rank * kWarps + wid];
        if (CL > 1) dst = cluster.map_shared_rank(dst, lane);
        RankSlot mine;
        mine.val = wv;
        mine.row = wrow;
        *dst = mine;
      }
      sync_all();
      if (j == c0 && c0 > 0) {
        // the previous block's rows of U beyond its columns, now that no CTA reads their old values any more
        const int* old = pivs[((c0 / kSub) & 1) ^ 1];
        for (int idx = tid; idx < kSub * (kb - c0); idx += kThreads) {
          const int p = idx % kSub, c = idx / kSub, lp = old[p] - row_lo;
          if (lp >= 0 && lp < rpc) pan[size_t(c0 + c) * rpc_max + lp] = U12[p][c];
        }
      }
      wv = 0;
      wrow = INT_MAX;
      for (int q = lane; q < CL * kWarps; q += 32) rank_merge(wv, wrow, wslot[par][q].val, wslot[par][q].row);
      rank_warp(wv, wrow);
      wrow = min(wrow, R - 1);  // always a row of the panel: every open row ranks at least zero
      const int owner = int(__umulhi(uint32_t(wrow), magic)), lr = wrow - owner * rpc;
      // the pivot row's entries, from its warp's slot in its CTA
      const double2* us = &wrowv[par][(kRpt == 1 ? lr : lr % kThreads) / 32][0];
      if (CL > 1) {
        const double2* src = cluster.map_shared_rank(us, owner);
        if (lane < kSub) ubuf[wid][lane] = src[lane];
        us = &ubuf[wid][0];
        __syncwarp();
      }
      double2 u[kSub];
#pragma unroll
      for (int q = 0; q < kSub; ++q) u[q] = us[q];
      if (tid == kThreads - 1) {
        piv[j - c0] = wrow;
        if (rank == 0) {
          const int q = row2pos[wrow];
          const int pj = pos2row[j];
          pos2row[j] = wrow;
          pos2row[q] = pj;
          row2pos[wrow] = j;
          row2pos[pj] = q;
          w.ipiv[size_t(b) * n + k + j] = k + q;
          if (wv == 0) {
            atomicMax(w.status + b, int(kDevSingular));
            atomicCAS(w.info + b, 0, k + j + 1);
          }
        }
      }
      // the pivot row is final: its entries in the block go back to the panel
#pragma unroll
      for (int i = 0; i < kRpt; ++i)
        if (open[i] && row_lo + tid + i * kThreads == wrow) {
          open[i] = false;
          done[lr] = 1;
          if constexpr (kRegs)
#pragma unroll
            for (int q = 0; q < kSub; ++q)
              if (q < left) pan[size_t(j + q) * rpc_max + lr] = x[i][q];
        }
      // multipliers by the pivot's reciprocal (by division where |pivot|^2 could leave the FP64 range, zero for a zero
      // or NaN pivot), and the rank-1 update of the block's own columns
      const int field = max(field_of(u[0].x), field_of(u[0].y));
      double2 pr = u[0];
      int mode = wv == 0 ? 0 : 2;
      bool any = false;
#pragma unroll
      for (int i = 0; i < kRpt; ++i) any = any || open[i];
      if (mode && any && field > 1023 - 440 && field < 1023 + 440) {
        mode = 1;
        const double inv = 1.0 / fma(u[0].x, u[0].x, u[0].y * u[0].y);
        pr = make_double2(u[0].x * inv, -u[0].y * inv);
      }
#pragma unroll
      for (int i = 0; i < kRpt; ++i) {
        if (!open[i]) continue;
        const double2 a = entry(i, 0);
        const double2 l = mode == 1 ? cmul(a, pr) : mode == 2 ? cdiv(a, pr) : make_double2(0.0, 0.0);
        pan[size_t(j) * rpc_max + tid + i * kThreads] = l;
        // the columns left without branches between them: a dependent FP64 operation waits about 140 cycles, so they have
        // to overlap (rounding their number up to 7, 3 or 1 issued a quarter more multiply-adds, 1% of a call)
        auto columns = [&](auto count) {
          constexpr int kCount = decltype(count)::value;
          double2 v[kCount];
#pragma unroll
          for (int q = 0; q < kCount; ++q) v[q] = entry(i, q + 1);
#pragma unroll
          for (int q = 0; q < kCount; ++q) cfms(v[q], l, u[q + 1]);
#pragma unroll
          for (int q = 0; q < kCount; ++q) {
            if constexpr (kRegs) x[i][q] = v[q];
            else if (q + 1 < left) pan[size_t(j + q + 1) * rpc_max + tid + i * kThreads] = v[q];
          }
        };
        switch (left) {
          case 8: columns(std::integral_constant<int, 7>()); break;
          case 7: columns(std::integral_constant<int, 6>()); break;
          case 6: columns(std::integral_constant<int, 5>()); break;
          case 5: columns(std::integral_constant<int, 4>()); break;
          case 4: columns(std::integral_constant<int, 3>()); break;
          case 3: columns(std::integral_constant<int, 2>()); break;
          case 2: columns(std::integral_constant<int, 1>()); break;
          default: break;
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
      // eight lanes a column, one row each
      for (int idx = tid; idx < (rest + 3) / 4 * 32; idx += kThreads) {
        const int p = idx % kSub, c = idx / kSub;
        double2 x = c < rest ? U12[p][c] : make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < kSub - 1; ++i) {
          const double2 xi = make_double2(__shfl_sync(0xffffffffu, x.x, (lane & 24) + i), __shfl_sync(0xffffffffu, x.y, (lane & 24) + i));
          if (p > i) cfms(x, L11[p][i], xi);
        }
        if (c < rest) U12[p][c] = x;
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
        const bool fits = w.digits && cut_tile_a(v, a);
        for (int gr = 0; gr < groups; ++gr) {
          int bad = 0;
#pragma unroll
          for (int q = 0; q < 8; ++q) bad |= ecol[gr][q] == kNonfinite;
          double2 p[2][2];
          uint32_t weak = 0, direct = 0;
          if (fits && !bad) {
            weak = tile_product(a, words[gr], ecol[gr], p);
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
                const double2 old = z;
                if ((weak >> (2 * h + q) & 1u) && below(old, a.e[h] + ecol[gr][2 * t + q] - kWeak)) direct |= 1u << (2 * h + q);
                else z = csub(old, p[h][q]);
              }
            }
          // in FP64 multiply-adds: sums whose products may have been lost on their grid (below kWeak of it, as C is)
          for (; direct; direct &= direct - 1) {
            const int bit = __ffs(direct) - 1, r = r0 + g + 8 * (bit >> 1), c = 8 * gr + 2 * t + (bit & 1);
            double2 s = make_double2(0.0, 0.0);
#pragma unroll
            for (int i = 0; i < kSub; ++i) cfma(s, pan[size_t(c0 + i) * rpc_max + r], U12[i][c]);
            double2& z = pan[size_t(ce + c) * rpc_max + r];
            z = csub(z, s);
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

template <int NB, int kMaxThreads, int kRpt>
cudaError_t launch_panel64_shape(const PanelConfig& pc, const BatchLayout& lay, int batch, int k, double2* M,
                                 const LuWork& w, cudaStream_t s) {
  if (pc.rpc_max > kMaxThreads * kRpt) return cudaErrorInvalidValue;
  auto kern = panel64_kernel<NB, kMaxThreads, kRpt>;
  cudaError_t err = ensure_smem_limit(reinterpret_cast<const void*>(kern), size_t(pc.smem));
  if (err != cudaSuccess) return err;
  if (pc.cluster > 8) {
    err = ensure_nonportable_clusters(reinterpret_cast<const void*>(kern));
    if (err != cudaSuccess) return err;
  }
  // the smallest cluster whose CTAs hold the trailing rows in whole 16-row tiles; then more CTAs while SMs would stay
  // idle and a CTA has more than a warp of rows for each quarter of its SM (the FP64 pipe, which bounds the panel,
  // takes as long for a part of a warp).  The factors do not depend on the cluster size.
  int cl = pc.cluster;
  const int R = lay.n - k, sms = current_sm_count();
  while (cl > 1 && ((R + cl / 2 - 1) / (cl / 2) + 15) / 16 * 16 <= pc.rpc_max) cl /= 2;
  while (cl < 8 && R > 128 * cl && (long long)batch * cl * 2 <= sms) cl *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(cl), unsigned(batch), 1);
  // a thread per row (kRpt = 1), at least four warps
  const int rows = ((R + cl - 1) / cl + 15) / 16 * 16, threads = std::max(128, (rows + 31) / 32 * 32);
  cfg.blockDim = dim3(unsigned(kRpt == 1 ? threads : kMaxThreads), 1, 1);
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
  // rows per CTA: at most 208 in the 100 KB panels of 32 columns (two CTAs per SM), 400, 800 and 1552 in the 200 KB ones
  switch (nb) {
    case 32:
      if (pc.rpc_max <= 256) return launch_panel64_shape<32, 256, 1>(pc, lay, batch, k, M, w, s);
      return launch_panel64_shape<32, 512, 1>(pc, lay, batch, k, M, w, s);
    case 16: return launch_panel64_shape<16, 512, 2>(pc, lay, batch, k, M, w, s);
    case 8: return launch_panel64_shape<8, 512, 4>(pc, lay, batch, k, M, w, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace rfx
