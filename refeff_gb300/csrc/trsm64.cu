// Block row and block column solves of the FP64 elimination and back
// substitution: U12 = L11^-1 (P A12) for the columns right of a panel (with the
// panel's row moves), and X = U11^-1 Y on the right-hand sides.
//
// A substitution of 32 steps takes 128 FP64 instructions a column (4 a step,
// one row a lane), and a warp's FP64 instruction occupies its quarter of the
// SM for 64 cycles, so the column-by-column form is bound by the FP64 pipe.
// Here a warp takes 16 columns in blocks of 8 rows: substitution inside a
// block (28 instructions a column in all), and the update of the other blocks
// in exact 8-bit digit products (digits64.cuh) from the digits of the 8 x 8
// blocks of the triangle, cut once per CTA.  The product is formed transposed,
// C^T -= X^T L^T, so that X, the operand X^T and C^T share one register layout
// (lane (g, t): columns g and g + 8, rows 2t and 2t + 1 of the block) and
// nothing moves between lanes but the substitution's own broadcasts.  Sums that
// the digits' grid may have lost are formed again in FP64 multiply-adds.
#include <cuda_runtime.h>
#include "batched_lu.cuh"
#include "cplx.cuh"
#include "digits64.cuh"

namespace rfx {

namespace {

constexpr int kBlk = 8;                // rows per block
constexpr int kMaxBlocks = 4;          // kb <= 32
constexpr int kPairs = kMaxBlocks * (kMaxBlocks - 1) / 2;
constexpr int kWarps = 4, kWarpCols = 16;

__device__ __forceinline__ double2 shfl2(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// Columns [c_begin, c_end) of every matrix, rows [k, k + kb).  kUpper: X = U11^-1 Y.  Else: the panel's row moves, then
// L11^-1.
template <bool kUpper>
__global__ void __launch_bounds__(32 * kWarps) trsm64_kernel(BatchLayout lay, int k, int kb, int c_begin, int c_end,
                                                             double2* __restrict__ M, LuWork w, int panel,
                                                             const int* skip) {
  const int b = blockIdx.y;
  if (skip && skip[b]) return;
  // T[r][c]: the triangle's rows (kUpper: each divided by its diagonal entry inside the diagonal blocks)
  __shared__ double2 T[kMaxBlocks * kBlk][kMaxBlocks * kBlk + 1];
  __shared__ double2 rdiag[kMaxBlocks * kBlk];             // kUpper: reciprocals of the diagonal
  __shared__ uint32_t words[kPairs][2 * kDig * 32];        // digits of block (p, q)^T, p != q, as B operands
  __shared__ int ecol[kPairs][8];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, t = lane & 3;
  const int nblk = (kb + kBlk - 1) / kBlk;
  const size_t lda = size_t(lay.lda);
  double2* Mb = M + size_t(b) * lay.stride;
  for (int idx = tid; idx < nblk * kBlk * nblk * kBlk; idx += 32 * kWarps) {
    const int r = idx % (nblk * kBlk), c = idx / (nblk * kBlk);
    T[r][c] = r < kb && c < kb ? Mb[size_t(k + r) + lda * size_t(k + c)] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  // the block of T that multiplies block q's solution in block p's rows: below the diagonal, or above it for kUpper
  auto pair_of = [](int p, int q) { return kUpper ? q * (q - 1) / 2 + p : p * (p - 1) / 2 + q; };
  {
    int at = 0;
    for (int hi = 1; hi < nblk; ++hi)
      for (int lo = 0; lo < hi; ++lo, ++at) {
        if (at % kWarps != wid) continue;
        const int p = kUpper ? lo : hi, q = kUpper ? hi : lo;
        double2 v[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) v[i] = T[p * kBlk + g][q * kBlk + 2 * t + i];  // B[k = 2t + i][n = g] = T_pq[n][k]
        cut_tile_b(v, words[pair_of(p, q)], ecol[pair_of(p, q)]);
      }
  }
  if constexpr (kUpper) {
    if (tid < kb) {
      const double2 d = T[tid][tid];
      rdiag[tid] = d.x == 0.0 && d.y == 0.0 ? make_double2(0.0, 0.0) : cdiv(make_double2(1.0, 0.0), d);
    }
    __syncthreads();
    for (int idx = tid; idx < nblk * kBlk * kBlk; idx += 32 * kWarps) {
      const int r = idx / kBlk, c = r / kBlk * kBlk + idx % kBlk;
      if (r < kb && c < kb && c > r) T[r][c] = cmul(T[r][c], rdiag[r]);
    }
  }
  __syncthreads();
  const int first = c_begin + (blockIdx.x * kWarps + wid) * kWarpCols;
  if (first >= c_end) return;
  if constexpr (!kUpper) {
    // the panel's row moves: every source is read before any row is written, eight columns at a time
    const size_t pidx = size_t(b) * w.npanels + panel;
    const int np = w.nperm[pidx];
    const int2* pm = w.perm + pidx * (2 * w.nb);
    int2 mv[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) mv[i] = lane + 32 * i < np ? pm[lane + 32 * i] : make_int2(-1, 0);
#pragma unroll 1
    for (int c0 = 0; c0 < kWarpCols; c0 += 8) {
      double2 v[8][2];
#pragma unroll
      for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (mv[i].x >= 0 && first + c0 + c < c_end) v[c][i] = Mb[size_t(mv[i].y) + lda * size_t(first + c0 + c)];
      __syncwarp();
#pragma unroll
      for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (mv[i].x >= 0 && first + c0 + c < c_end) Mb[size_t(mv[i].x) + lda * size_t(first + c0 + c)] = v[c][i];
    }
    __syncwarp();
  }
  // x[p][h][i]: row 8p + 2t + i, column g + 8h
  double2 x[kMaxBlocks][2][2];
#pragma unroll
  for (int p = 0; p < kMaxBlocks; ++p)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = p * kBlk + 2 * t + i, c = first + g + 8 * h;
        x[p][h][i] = r < kb && c < c_end ? Mb[size_t(k + r) + lda * size_t(c)] : make_double2(0.0, 0.0);
      }
#pragma unroll
  for (int s = 0; s < kMaxBlocks; ++s) {
    const int q = kUpper ? kMaxBlocks - 1 - s : s;
    if (q >= nblk) continue;
    // the diagonal block, a row a step
    if constexpr (kUpper) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int r = q * kBlk + 2 * t + i;
          x[q][h][i] = r < kb ? cmul(x[q][h][i], rdiag[r]) : make_double2(0.0, 0.0);
        }
    }
#pragma unroll
    for (int step = 0; step < kBlk - 1; ++step) {
      const int j = kUpper ? kBlk - 1 - step : step;
      double2 xj[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) xj[h] = shfl2(x[q][h][j & 1], (lane & 28) + (j >> 1));
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = 2 * t + i;
        if (kUpper ? r < j : r > j) {
          const double2 m = T[q * kBlk + r][q * kBlk + j];
#pragma unroll
          for (int h = 0; h < 2; ++h) cfms(x[q][h][i], m, xj[h]);
        }
      }
    }
    // the other blocks' rows
    if (kUpper ? q == 0 : q + 1 >= nblk) continue;
    DigitTileA a;
    const bool fits = w.digits && cut_tile_a(x[q], a);
#pragma unroll
    for (int p = 0; p < kMaxBlocks; ++p) {
      if (kUpper ? p >= q : p <= q || p >= nblk) continue;
      const int at = pair_of(p, q);
      int bad = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) bad |= ecol[at][i] == kNonfinite;
      double2 d[2][2];
      // entries (bit 2 h + i) to be summed in FP64 multiply-adds: all of a tile that the digits cannot hold, and those
      // whose products may have been lost on their grid (below kWeak of it, as C is)
      uint32_t direct = 15;
      if (fits && !bad) {
        direct = tile_product(a, words[at], ecol[at], d);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (!below(x[p][h][i], a.e[h] + ecol[at][2 * t + i] - kWeak)) direct &= ~(1u << (2 * h + i));
      }
      if (__any_sync(0xffffffffu, direct)) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (!__any_sync(0xffffffffu, direct >> (2 * h + i) & 1u)) continue;
            double2 s = make_double2(0.0, 0.0);
#pragma unroll 2
            for (int j = 0; j < kBlk; ++j) {
              const double2 xj = shfl2(j & 1 ? x[q][h][1] : x[q][h][0], (lane & 28) + (j >> 1));
              cfma(s, T[p * kBlk + 2 * t + i][q * kBlk + j], xj);
            }
            if (direct >> (2 * h + i) & 1u) d[h][i] = s;
          }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 2; ++i) x[p][h][i] = csub(x[p][h][i], d[h][i]);
    }
  }
#pragma unroll
  for (int p = 0; p < kMaxBlocks; ++p)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = p * kBlk + 2 * t + i, c = first + g + 8 * h;
        if (r < kb && c < c_end) Mb[size_t(k + r) + lda * size_t(c)] = x[p][h][i];
      }
}

}  // namespace

void launch_trsm64(bool upper, const BatchLayout& lay, int batch, int k, int kb, int c_begin, int c_end, double2* M,
                   const LuWork& w, const int* skip, cudaStream_t s) {
  const int ncols = c_end - c_begin;
  if (ncols <= 0) return;
  const dim3 grid(unsigned((ncols + kWarps * kWarpCols - 1) / (kWarps * kWarpCols)), unsigned(batch));
  count_launch();
  if (upper) trsm64_kernel<true><<<grid, 32 * kWarps, 0, s>>>(lay, k, kb, c_begin, c_end, M, w, 0, skip);
  else trsm64_kernel<false><<<grid, 32 * kWarps, 0, s>>>(lay, k, kb, c_begin, c_end, M, w, k / w.nb, skip);
}

}  // namespace rfx
