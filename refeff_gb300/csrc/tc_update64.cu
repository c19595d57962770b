// Tensor-core (tcgen05, sm_103a) block update of the FP64 elimination and of
// the FP64 triangular sweeps over many right-hand sides:
//     C[r, c] -= sum_k A[r, k] B[k, c]      (complex FP64, K <= 32)
// with C, A and B blocks of one matrix.
//
// The FP64 pipe of GB300 runs 2 multiply-adds per SM and cycle (1.15 TFLOP/s
// measured in this update); the bf16 tensor path runs about 1600 times that.
// The products are therefore formed exactly on the tensor path from signed
// 8-bit digits, an error-free splitting after Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication by using fast routines
// of matrix multiplication and its applications", Numer. Algorithms 59 (2012):
//
//   * column k of A is multiplied by 2^g_k and row k of B by 2^-g_k so that no
//     column of A is small in every row (graded systems: without it a system
//     whose columns span 24 orders of magnitude loses every digit in the back
//     substitution); row r of A is then scaled by a power of two 2^-e_r so that
//     its real and imaginary parts lie in (-1, 1), column c of B by 2^-f_c; a
//     row of B that meets a zero column of A takes no part in f_c;
//   * each scaled value is rounded to a 62-bit fixed-point number and cut into
//     eight signed digits of weights 2^-6, 2^-14, ..., 2^-62 (|t| <= 128, exact
//     in bf16);
//   * tcgen05.mma kind::f16 with FP32 accumulation sums the digit products of
//     one level s = i + j (2 .. 9, 36 pairs) without rounding: at most 8 pairs
//     x 2 real products x 32 columns x 2^14 = 2^23 < 2^24;
//   * the epilogue adds the eight exact level sums in 64-bit integers, converts
//     the total to FP64 (one rounding) and subtracts it from C (one rounding);
//   * where neither the sum nor C reaches 2^-7 of 2^(e_r + f_c), the products may
//     be too small for the grid (sparse and badly scaled systems): unless large
//     entries of the row and the column meet, the epilogue lists the entry, and
//     tc64_recheck_kernel looks up its largest product and forms the sum again
//     in FP64 multiply-adds where that is below 2^-6 of it.
//
// Dropped and cut parts weigh about 2^-62 of 2^(e_r + f_c) per product and the
// join keeps 2^-57 of it, less than what the FMA chain it replaces rounds away in
// its 32 steps: on 40 FMS systems of n = 117 .. 688 and 8 random ones the error
// of the solution is 0.23 .. 0.70 of the chain's, 0.51 in the geometric mean
// (seven digits, 28 pairs, measured up to twice the chain's error).
//
// Layout of the work: a CTA owns a 128-row tile of A, whose digits for all 32
// columns (128 KB) stay in shared memory while it walks 16-column tiles of B
// and C.  One MMA multiplies one digit plane of A by the adjacent digit slots
// of B (N = 32 (9 - i)) into the adjacent level accumulators, so the 36 x 4
// real products of a K step take 16 instructions.  Two sets of 256 TMEM columns
// alternate, and sixteen epilogue warps finish one tile while the next is
// multiplied.  The tensor work per tile (2304 cycles), its C traffic (64 KB)
// and its 4096 FP64 subtractions (2048 cycles) are of the same size, so neither
// a deeper K nor a wider tile would win much.
//
// Every wait on an mbarrier is bounded.  A CTA whose waits ran out drains its
// copies and MMAs, and its epilogue warps finish their remaining tiles with
// FP64 multiply-adds from the matrix, so the update is complete in any case;
// rows and columns that hold an infinity or NaN, or whose products lie near the
// ends of the FP64 range, take the same path.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include "cplx.cuh"
#include "batched_lu.cuh"
#include "digits64.cuh"

namespace rfx {

namespace {

constexpr int kRows = 128;                       // rows per tile (MMA M)
constexpr int kCols = 16;                        // columns per tile
constexpr int kPlane = kRows * 32;               // one digit plane of A, one K step (16 columns): 4 KB
constexpr int kAHalf = 2 * kDig * kPlane;        // re and im digits of one K step: 64 KB
constexpr int kATile = 2 * kAHalf;               // 128 KB
constexpr int kBSide = kDig * 2 * kCols * 32;    // eight slots of 32 rows of 16 bf16: 8 KB
constexpr int kBHalf = 2 * kBSide;               // P = [Br | Bi] and Q = [-Bi | Br], one K step: 16 KB
constexpr int kBTile = 2 * kBHalf;               // 32 KB
constexpr int kBStages = 3;
constexpr int kEpiWarps = 16;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr uint32_t kTmemCols = 512;              // two accumulator sets of 8 levels x [re | im] x 16 columns
constexpr int kBarOff = kATile + kBStages * kBTile;
constexpr int kSmem = kBarOff + 256 + 1024;      // + alignment of the base to 1 KB
static_assert(kSmem <= 227 * 1024, "dynamic shared memory per CTA");

// barriers: A halves full / empty, B stages full / empty, accumulators full / empty, drain
enum : int { kAFull = 0, kAEmpty = 2, kBFull = 4, kBEmpty = 4 + kBStages, kAccFull = 4 + 2 * kBStages,
             kAccEmpty = 6 + 2 * kBStages, kDrain = 8 + 2 * kBStages, kBars = 9 + 2 * kBStages };
static_assert(kBars * 8 <= 128, "barrier area");

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// Byte offset of 16-byte chunk `chunk` of row `row` in a K-major tile of 32-byte rows with the 32-byte swizzle.
__device__ __forceinline__ int sw32(int row, int chunk) { return row * 32 + ((chunk ^ ((row >> 2) & 1)) << 4); }
// start >> 4, LBO 1 (unused when swizzled), SBO = 8 rows x 32 B, version 1, 32-byte swizzle (layout 6)
__device__ __forceinline__ uint64_t desc_sw32(uint32_t saddr) {
  return uint64_t((saddr >> 4) & 0x3FFFu) | (uint64_t(1) << 16) | (uint64_t(256 >> 4) << 32) | (uint64_t(1) << 46) |
         (uint64_t(6) << 61);
}
// kind::f16, D = F32, A = B = BF16, both K-major, M = 128, N columns
__device__ __forceinline__ uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(kRows >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// Bounded wait of one role on another (poll budget, or 1 s); gives up early once the CTA's abort flag is up,
// and raises that flag when it runs out.
__device__ __forceinline__ bool role_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, long long polls) {
  uint64_t t0 = 0;  // the clock is read after 256 polls: its read takes longer than most waits
  for (long long it = 0; it < polls; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255) == 255) {
      if (*abort_flag) return false;
      const uint64_t t = global_ns();
      if (t0 == 0) t0 = t;
      else if (t - t0 > 1000000000ull) break;
    }
  }
  *abort_flag = 1;
  return false;
}
// Drain wait for work this thread issued itself (the full default budget, no abort exit).
__device__ __forceinline__ void drain_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return;
  const uint64_t t0 = global_ns();
  for (long long it = 0; it < kTcWaitPolls; ++it)
    if (mbar_try(bar, parity) || ((it & 1023) == 1023 && global_ns() - t0 > 1000000000ull)) return;
}

// sum_k A[row, k] B[k, col] in FP64 multiply-adds: the path of rows and columns that the digits cannot hold, and
// of tiles whose waits ran out.
__device__ __forceinline__ double2 direct_sum(const double2* arow, const double2* bcol, int lda, int kb) {
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 1
  for (int k = 0; k < kb; ++k) cfma(acc, arow[size_t(lda) * k], bcol[k]);
  return acc;
}

// Most small sums are of large products that cancel: masks of the k at which a row's entries reach 2^-kLostPart of its
// largest, and a column's of its, tell it by a common bit.
constexpr int kLostPart = kLost / 2;
constexpr int kZero = 127;  // a sum of two deficits from here on: a product that is zero
// An entry whose sum the grid may have lost: C at (row, col) of matrix b is untouched yet; p the digit sum, of grid 2^e.
struct alignas(16) Tc64Entry {
  double2 p;
  int row, col, b, e;
};
// Entries a block of tc64_recheck_kernel takes at a time: each CTA lists its own ones (counted in shared memory: a global
// counter's latency held the epilogues up, 28.6 instead of 26.8 ms of updates of 16 systems of n = 2256) and hands them
// on as chunks (first entry, count), since a few CTAs have most.
constexpr int kChunk = 64;

}  // namespace

// alpha[b][k] = 2048 + max over the rows of (exponent of A[row, k] - exponent of the row's largest entry), 0 where column k
// is zero in every row without infinities and NaN: g_k = 2048 - alpha.  The table is zero before and is cleared again by the update kernel.
__global__ void __launch_bounds__(kRows) tc64_scale_kernel(BatchLayout lay, int r_begin, int r_end, int ka, int kb,
                                                           const double2* __restrict__ M, int* __restrict__ alpha,
                                                           int* __restrict__ chunks) {
  __shared__ int cmax[32];
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *chunks = 0;  // of the update that follows
  const int b = blockIdx.y, lane = threadIdx.x & 31, row = r_begin + blockIdx.x * kRows + int(threadIdx.x);
  if (threadIdx.x < 32) cmax[threadIdx.x] = 0;
  const double2* A = M + size_t(b) * lay.stride + size_t(row) + size_t(lay.lda) * ka;
  int f[32], top = 0;
#pragma unroll
  for (int k = 0; k < 32; ++k) f[k] = row < r_end && k < kb ? field_of(A[size_t(lay.lda) * k]) : -1;
#pragma unroll
  for (int k = 0; k < 32; ++k) top = max(top, f[k]);
  int mine = 0;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const int v = __reduce_max_sync(0xffffffffu, f[k] >= 0 && top < 0x7ff ? max(f[k], 1) - max(top, 1) + 2048 : 0);
    if (lane == k) mine = v;
  }
  __syncthreads();
  atomicMax(&cmax[lane], mine);
  __syncthreads();
  if (threadIdx.x < 32 && cmax[lane] > 0) atomicMax(alpha + b * 32 + lane, cmax[lane]);
}

// Digits of both operands.  Blocks x < nbm: a row tile of A, image[b][bm][K step][re 1..8, im 1..8][128 rows of 16 bf16]
// and the row exponents, two threads per row, 16 columns each.  The others: a column tile of B,
// image[b][bn][K step][P, Q][digit 1..8][32 rows of 16 bf16] with P = [Br | Bi], Q = [-Bi | Br] (16 columns each) and the
// column exponents, one warp per column, one lane per row, each exponent with its mask of large entries.  rdef and cdef:
// 32 bytes a row of A and a column of B, how many powers of two each (balanced) entry lies below the grid (63: 63 or more;
// kZero: zero, or meeting only zeros).
__global__ void __launch_bounds__(256) tc64_split_kernel(BatchLayout lay, int r_begin, int r_end, int c_begin, int c_end,
                                                         int ka, int kb, const double2* __restrict__ M,
                                                         const int* __restrict__ alpha, uint8_t* __restrict__ aimg,
                                                         uint8_t* __restrict__ bimg, int2* __restrict__ rexp,
                                                         int2* __restrict__ cexp, uint8_t* __restrict__ rdef,
                                                         uint8_t* __restrict__ cdef, int nbm, int nbm_all, int nbn_all) {
  __shared__ __align__(16) uint8_t sm[kBTile];
  __shared__ int gk[32];  // kNoEntry: column k of A is zero
  const int b = blockIdx.y;
  if (threadIdx.x < 32) {
    const int a = alpha[b * 32 + int(threadIdx.x)];
    gk[threadIdx.x] = a > 0 ? 2048 - a : kNoEntry;
  }
  __syncthreads();
  const double2* Mb = M + size_t(b) * lay.stride;
  if (int(blockIdx.x) < nbm) {
    int* rowmax = reinterpret_cast<int*>(sm);
    const int bm = blockIdx.x, r = threadIdx.x & (kRows - 1), h = threadIdx.x >> 7;
    const int row = r_begin + bm * kRows + r;
    const double2* A = Mb + size_t(row) + size_t(lay.lda) * (ka + 16 * h);
    double2 v[16];
    int e = kNoEntry;
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = row < r_end && 16 * h + i < kb ? A[size_t(lay.lda) * i] : make_double2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int f = field_of(v[i]);
      if (f >= 0) e = max(e, f == 0x7ff ? kNonfinite : max(f, 1) - 1022 + gk[16 * h + i]);
    }
    if (h == 0) rowmax[r] = e;
    __syncthreads();
    if (h == 1) rowmax[r] = max(rowmax[r], e);
    __syncthreads();
    e = rowmax[r];
    const size_t at = (size_t(b) * nbm_all + bm) * kRows + r;
    uint32_t below_grid[4] = {}, large = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int f = field_of(v[i]), d = f < 0 ? kZero : min(max(e - (max(f, 1) - 1022 + gk[16 * h + i]), 0), 63);
      below_grid[i / 4] |= uint32_t(d) << (8 * (i % 4));
      large |= d <= kLostPart ? 1u << i : 0u;
    }
    uint16_t* const half_mask = reinterpret_cast<uint16_t*>(&rexp[at].y);
    half_mask[h] = uint16_t(large);
    if (h == 0) rexp[at].x = e;
    *reinterpret_cast<uint4*>(rdef + at * 32 + 16 * h) = make_uint4(below_grid[0], below_grid[1], below_grid[2], below_grid[3]);
    if (h * 16 >= kb) return;  // a K step that is not multiplied
    const bool none = e == kNonfinite || e == kNoEntry;
    uint8_t* out = aimg + (size_t(b) * nbm_all + bm) * kATile + size_t(h) * kAHalf;
#pragma unroll
    for (int ch = 0; ch < 2; ++ch)
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint2 y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const double x = part ? v[8 * ch + i].y : v[8 * ch + i].x;
          const int g = gk[16 * h + 8 * ch + i];
          y[i] = none || g == kNoEntry ? biased_digits(0.0, 0) : biased_digits(x, e - g);
        }
#pragma unroll
        for (int d = 0; d < kDig; ++d) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) w[i] = pack_bf16(digit_of(y[2 * i], d), digit_of(y[2 * i + 1], d));
          *reinterpret_cast<uint4*>(out + (part * kDig + d) * kPlane + sw32(r, ch)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    return;
  }
  const int bn = int(blockIdx.x) - nbm, k = threadIdx.x & 31;
  uint8_t* const p = sm + (k >> 4) * kBHalf;
  uint8_t* const q = p + kBSide;
  const int ch = (k >> 3) & 1, kk = (k & 7) * 2;
  for (int c = threadIdx.x >> 5; c < kCols; c += 8) {
    const int col = c_begin + bn * kCols + c;
    double2 v = make_double2(0.0, 0.0);
    if (col < c_end && k < kb) v = Mb[size_t(ka + k) + size_t(lay.lda) * col];
    // an entry that meets only zeros of A must not set the column's grid (an infinity or NaN still marks the column)
    const int f = field_of(v), g = gk[k];
    const int e = __reduce_max_sync(0xffffffffu, f == 0x7ff ? kNonfinite : f < 0 || g == kNoEntry ? kNoEntry : max(f, 1) - 1022 - g);
    const bool none = e == kNonfinite || e == kNoEntry || g == kNoEntry;
    const int d = none || f < 0 ? kZero : min(e - (max(f, 1) - 1022 - g), 63);
    const size_t at = (size_t(b) * nbn_all + bn) * kCols + c;
    cdef[at * 32 + k] = uint8_t(d);
    const uint32_t large = __ballot_sync(0xffffffffu, d <= kLostPart);
    if (k == 0) cexp[at] = make_int2(e, int(large));
    if (none) v = make_double2(0.0, 0.0);
    const uint2 yr = biased_digits(v.x, none ? 0 : e + g), yi = biased_digits(v.y, none ? 0 : e + g);
#pragma unroll
    for (int d = 0; d < kDig; ++d) {
      const float re = digit_of(yr, d), im = digit_of(yi, d);
      auto put = [&](uint8_t* base, int row, float x) {
        *reinterpret_cast<uint16_t*>(base + sw32(row, ch) + kk) = uint16_t(__float_as_uint(x) >> 16);
      };
      put(p, d * 32 + c, re);
      put(p, d * 32 + 16 + c, im);
      put(q, d * 32 + c, -im);
      put(q, d * 32 + 16 + c, re);
    }
  }
  __syncthreads();
  uint4* out = reinterpret_cast<uint4*>(bimg + (size_t(b) * nbn_all + bn) * kBTile);
  const int bytes = kb > 16 ? kBTile : kBHalf;
  for (int i = threadIdx.x; i < bytes / 16; i += 256) out[i] = reinterpret_cast<const uint4*>(sm)[i];
}

// The walk of a CTA: units (matrix, row tile, segment of `chunk` column tiles), every gridDim.x-th, and the column
// tiles inside each.
struct Tc64Work {
  int nbm, nbn, nseg, chunk, units;
};
struct Tc64Tile {
  int u, bn, bn_end, b, bm;
  __device__ __forceinline__ void unit(const Tc64Work& w) {
    const int seg = u % w.nseg, rest = u / w.nseg;
    bm = rest % w.nbm;
    b = rest / w.nbm;
    bn = seg * w.chunk;
    bn_end = min(bn + w.chunk, w.nbn);
  }
  __device__ __forceinline__ bool start(const Tc64Work& w) {
    u = blockIdx.x;
    if (u >= w.units) return false;
    unit(w);
    return true;
  }
  __device__ __forceinline__ bool next(const Tc64Work& w) {
    if (++bn < bn_end) return true;
    u += gridDim.x;
    if (u >= w.units) return false;
    unit(w);
    return true;
  }
};

__global__ void __launch_bounds__(kThreads, 1)
    tc64_update_kernel(BatchLayout lay, int r_begin, int r_end, int c_begin, int c_end, int ka, int kb,
                       double2* __restrict__ M, const uint8_t* __restrict__ aimg, const uint8_t* __restrict__ bimg,
                       const int2* __restrict__ rexp, const int2* __restrict__ cexp, int nbm_all, int nbn_all,
                       Tc64Work w, int* __restrict__ alpha, int alpha_n, Tc64Entry* __restrict__ list,
                       int2* __restrict__ chunk, int* __restrict__ chunks, int capacity, long long polls) {
  extern __shared__ uint8_t smraw[];
  const uint32_t raw = smem_u32(smraw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* const meta = smraw + (sbase - raw) + kBarOff;
  auto bar = [&](int i) { return smem_u32(meta) + 8u * uint32_t(i); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(meta + 128);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(meta + 132);
  int* const entries = reinterpret_cast<int*>(meta + 136);  // listed by this CTA, and those that found no room
  const int list0 = blockIdx.x * capacity;                  // this CTA's part of the list
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nk = kb > 16 ? 2 : 1;  // K steps
  if (blockIdx.x == 0)
    for (int i = tid; i < alpha_n; i += kThreads) alpha[i] = 0;  // read by the split kernel before; for the next update

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    for (int i = 0; i < kBars; ++i)
      mbar_init(bar(i), i == kAccEmpty || i == kAccEmpty + 1 ? uint32_t(kEpiWarps) : 1u);
    *abort_flag = 0;
    *entries = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---- producer: the digits of A once per unit, those of B per tile ----
    if (lane == 0) {
      uint32_t units = 0, tiles = 0;
      Tc64Tile t;
      bool more = t.start(w), ok = true;
      uint32_t a_issued[2] = {0, 0};
      while (more && ok && !*abort_flag) {
        const uint8_t* ab = aimg + (size_t(t.b) * nbm_all + t.bm) * kATile;
        for (int h = 0; h < nk && ok; ++h) {
          ok = role_wait(bar(kAEmpty + h), (units & 1) ^ 1, abort_flag, polls);
          if (!ok) break;
          mbar_expect_tx(bar(kAFull + h), kAHalf);
          for (int i = 0; i < 4; ++i)
            bulk_copy(sbase + h * kAHalf + i * (kAHalf / 4), ab + h * kAHalf + i * (kAHalf / 4), kAHalf / 4, bar(kAFull + h));
          ++a_issued[h];
        }
        const int u = t.u;
        while (more && t.u == u && ok) {
          const int st = int(tiles % kBStages);
          ok = role_wait(bar(kBEmpty + st), ((tiles / kBStages) & 1) ^ 1, abort_flag, polls);
          if (!ok) break;
          mbar_expect_tx(bar(kBFull + st), uint32_t(nk * kBHalf));
          bulk_copy(sbase + kATile + st * kBTile, bimg + (size_t(t.b) * nbn_all + t.bn) * kBTile, uint32_t(nk * kBHalf),
                    bar(kBFull + st));
          ++tiles;
          more = t.next(w);
        }
        ++units;
      }
      // every copy has landed before the CTA ends
      for (int h = 0; h < nk; ++h)
        if (a_issued[h]) drain_wait(bar(kAFull + h), (a_issued[h] - 1) & 1);
      for (uint32_t q = tiles > uint32_t(kBStages) ? tiles - kBStages : 0; q < tiles; ++q)
        drain_wait(bar(kBFull + int(q % kBStages)), (q / kBStages) & 1);
    }
  } else if (warp == 1) {
    // ---- MMA issuer ----
    if (lane == 0) {
      uint32_t units = 0, tiles = 0;
      bool issued = false, ok = true;
      Tc64Tile t;
      bool more = t.start(w), first = true;
      while (more && ok && !*abort_flag) {
        const uint32_t buf = tiles & 1;
        const int st = int(tiles % kBStages);
        ok = role_wait(bar(kAccEmpty + int(buf)), ((tiles >> 1) & 1) ^ 1, abort_flag, polls) &&
             role_wait(bar(kBFull + st), (tiles / kBStages) & 1, abort_flag, polls);
        if (!ok) break;
        Tc64Tile nx = t;
        const bool nmore = nx.next(w);
        const bool last = !nmore || nx.u != t.u;  // of the unit
        for (int h = 0; h < nk; ++h) {
          if (first && !(ok = role_wait(bar(kAFull + h), units & 1, abort_flag, polls))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sA = sbase + h * kAHalf, sP = sbase + kATile + st * kBTile + h * kBHalf;
          const uint64_t dp = desc_sw32(sP), dq = desc_sw32(sP + kBSide);
#pragma unroll 1
          for (int i = 0; i < kDig; ++i) {
            // digit i + 1 of A against digits 1 .. 8 - i of B: levels i + 2 .. 9
            const uint32_t d = tmem + buf * 256 + uint32_t(32 * i), id = idesc_bf16(32 * (kDig - i));
            mma_bf16(d, desc_sw32(sA + i * kPlane), dp, id, h || i ? 1u : 0u);
            mma_bf16(d, desc_sw32(sA + (kDig + i) * kPlane), dq, id, 1u);
          }
          issued = true;
          if (last) mma_commit(bar(kAEmpty + h));
        }
        if (!ok) break;
        mma_commit(bar(kBEmpty + st));
        mma_commit(bar(kAccFull + int(buf)));
        ++tiles;
        first = last;
        if (last) ++units;
        t = nx;
        more = nmore;
      }
      if (issued) {  // every MMA has completed before the tensor memory is freed
        mma_commit(bar(kDrain));
        drain_wait(bar(kDrain), 0);
      }
    }
  } else {
    // ---- epilogue: warp (quarter, g) finishes rows [32 quarter, + 32), columns [4 g, + 4) of every tile ----
    const int g = (warp - 2) >> 2, quarter = warp & 3;
    const uint32_t lane_off = uint32_t(quarter * 32) << 16;
    const int lda = lay.lda;
    uint32_t tiles = 0;
    bool direct = false;  // the waits ran out: the remaining tiles in FP64 multiply-adds
    Tc64Tile t;
    bool more = t.start(w);
    // C of this thread's four entries, each loaded again for the next tile once it has been used
    double2 cn[4];
    auto c_ptr = [&](const Tc64Tile& q) {
      return M + size_t(q.b) * lay.stride + size_t(r_begin + q.bm * kRows + quarter * 32 + lane) +
             size_t(lda) * size_t(c_begin + q.bn * kCols + 4 * g);
    };
    // columns of the tile that this thread has: 0 where its row lies outside the block
    auto c_count = [&](const Tc64Tile& q) {
      return r_begin + q.bm * kRows + quarter * 32 + lane < r_end ? c_end - (c_begin + q.bn * kCols + 4 * g) : 0;
    };
    double2* cur = M;
    int have = 0;
    if (more) {
      cur = c_ptr(t);
      have = c_count(t);
#pragma unroll
      for (int j = 0; j < 4; ++j) cn[j] = j < have ? cur[size_t(lda) * j] : make_double2(0.0, 0.0);
    }
    while (more) {
      const int2 erm = rexp[(size_t(t.b) * nbm_all + t.bm) * kRows + quarter * 32 + lane];
      int er = erm.x;
      const int4* const ec4 = reinterpret_cast<const int4*>(cexp + (size_t(t.b) * nbn_all + t.bn) * kCols + 4 * g);
      const int4 ec01 = ec4[0], ec23 = ec4[1];
      const int ec[4] = {ec01.x, ec01.z, ec23.x, ec23.z}, cmask[4] = {ec01.y, ec01.w, ec23.y, ec23.w};
      const int tb = t.b, tcol = c_begin + t.bn * kCols + 4 * g, trow = r_begin + t.bm * kRows + quarter * 32 + lane;
      more = t.next(w);
      double2* const nxt = more ? c_ptr(t) : M;
      const int nhave = more ? c_count(t) : 0;
      const uint32_t buf = tiles & 1;
      if (!direct) {
        const bool ready = role_wait(bar(kAccFull + int(buf)), (tiles >> 1) & 1, abort_flag, polls);
        direct = !__all_sync(0xffffffffu, ready);
      }
      if (direct) er = kNonfinite;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // one column at a time: the level sums of more would not fit in registers beside C, and C spilled to local
      // memory stalls on its own loads (4 us a tile)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t lv[2 * kDig];
        __syncwarp();
        if (!direct) {
          const uint32_t ta = tmem + buf * 256 + lane_off + uint32_t(4 * g + c);
#pragma unroll
          for (int s = 0; s < kDig; ++s) {
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(lv[s]) : "r"(ta + uint32_t(32 * s)));
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];"
                         : "=r"(lv[kDig + s])
                         : "r"(ta + uint32_t(32 * s + 16)));
          }
          // the loaded registers pass through the wait, so that nothing reads them before it
          asm volatile("tcgen05.wait::ld.sync.aligned;"
                       : "+r"(lv[0]), "+r"(lv[1]), "+r"(lv[2]), "+r"(lv[3]), "+r"(lv[4]), "+r"(lv[5]), "+r"(lv[6]),
                         "+r"(lv[7]), "+r"(lv[8]), "+r"(lv[9]), "+r"(lv[10]), "+r"(lv[11]), "+r"(lv[12]),
                         "+r"(lv[13]), "+r"(lv[14]), "+r"(lv[15])::"memory");
          if (c == 3) {  // the accumulators are in registers: they may be overwritten
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (lane == 0) mbar_arrive(bar(kAccEmpty + int(buf)));
          }
        }
        if (c < have) {
          double2 p = make_double2(0.0, 0.0);
          bool store = true;
          auto direct_entry = [&] {
            const double2* Mb = M + size_t(tb) * lay.stride;
            return direct_sum(Mb + size_t(trow) + size_t(lda) * ka, Mb + size_t(ka) + size_t(lda) * (tcol + c), lda, kb);
          };
          const int e = er + ec[c];  // kNonfinite or more with an infinity or NaN, or where the waits ran out
          if (unsigned(e + kSafeExp) <= 2u * kSafeExp) {
            int ur, ui;
            const long long vr = join_levels<true>(lv, ur), vi = join_levels<true>(lv + kDig, ui);
            p = make_double2(normal_double(vr, e + ur), normal_double(vi, e + ui));
            if (ur + ui == 2 * kFineUnit && !(erm.y & cmask[c]) && below(cn[c], e - kWeak)) {
              // a full list is not counted on: the counter stays within the threads that race for its last places
              const int at = *static_cast<volatile int*>(entries) < capacity ? atomicAdd(entries, 1) : capacity;
              store = at >= capacity;
              if (store) {  // no room
                p = direct_entry();
              } else {
                Tc64Entry entry;
                entry.p = p;
                entry.row = trow;
                entry.col = tcol + c;
                entry.b = tb;
                entry.e = e;
                list[list0 + at] = entry;
              }
            }
          } else if (e > kNoEntry / 2) {  // else a row or column of zeros
            p = direct_entry();
          }
          if (store) cur[size_t(lda) * c] = make_double2(cn[c].x - p.x, cn[c].y - p.y);
        }
        cn[c] = c < nhave ? nxt[size_t(lda) * c] : make_double2(0.0, 0.0);
      }
      ++tiles;
      cur = nxt;
      have = nhave;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    const int have = min(*entries, capacity), mine = (have + kChunk - 1) / kChunk;
    int at = 0;
    if (mine > 0 && lane == 0) at = atomicAdd(chunks, mine);
    at = __shfl_sync(0xffffffffu, at, 0);
    for (int q = lane; q < mine; q += 32) chunk[at + q] = make_int2(list0 + q * kChunk, min(kChunk, have - q * kChunk));
  }
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// The listed entries: C -= p where a product reaches 2^(e - kLost) or all are zero, else C -= the sum in FP64 multiply-adds.  Four lanes
// an entry, eight terms each.  A kernel of its own: these entries gather in few rows of few tiles (0.3 .. 0.6% of all on
// symmetric clusters, whose structural zeros are rounding noise in C), where warps that summed their own ones would hold
// their tiles up.  Most are sound, and the bytes of rdef and cdef tell it without A and B.
__global__ void __launch_bounds__(4 * kChunk, 2) tc64_recheck_kernel(BatchLayout lay, int r_begin, int c_begin, int ka, int kb,
                                                                     double2* __restrict__ M, const uint8_t* __restrict__ rdef,
                                                                     const uint8_t* __restrict__ cdef, int nbm_all, int nbn_all,
                                                                     const Tc64Entry* __restrict__ list,
                                                                     const int2* __restrict__ chunk,
                                                                     const int* __restrict__ chunks) {
  const int total = *chunks, i = int(threadIdx.x) / 4, part = threadIdx.x & 3;
  const size_t lda = size_t(lay.lda);
  for (int ch = blockIdx.x; ch < total; ch += gridDim.x) {
    const int2 cc = chunk[ch];
    const Tc64Entry q = list[cc.x + min(i, cc.y - 1)];
    double2* const Mb = M + size_t(q.b) * lay.stride;
    double2* const c = Mb + size_t(q.row) + lda * size_t(q.col);
    double2 z = *c, p = q.p;
    const uint2 da = *reinterpret_cast<const uint2*>(rdef + (size_t(q.b) * nbm_all * kRows + (q.row - r_begin)) * 32 + 8 * part);
    const uint2 db = *reinterpret_cast<const uint2*>(cdef + (size_t(q.b) * nbn_all * kCols + (q.col - c_begin)) * 32 + 8 * part);
    uint32_t d = __vminu4(da.x + db.x, da.y + db.y);  // at most 254 a byte
    d = __vminu4(d, __shfl_xor_sync(0xffffffffu, d, 1));
    d = __vminu4(d, __shfl_xor_sync(0xffffffffu, d, 2));
    d = __vminu4(d, d >> 16);
    const uint32_t least = min(d & 255u, (d >> 8) & 255u);
    const bool again = least > uint32_t(kLost) && least < uint32_t(kZero);
    if (__any_sync(0xffffffffu, again)) {
      const double2* const a = Mb + size_t(q.row) + lda * size_t(ka);
      const double2* const b = Mb + size_t(ka) + lda * size_t(q.col);
      double2 va[8], vb[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = part + 4 * j;
        va[j] = again && k < kb ? a[lda * size_t(k)] : make_double2(0.0, 0.0);
        vb[j] = again && k < kb ? b[k] : make_double2(0.0, 0.0);
      }
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int j = 0; j < 8; ++j) cfma(s, va[j], vb[j]);
#pragma unroll
      for (int w = 1; w < 4; w *= 2) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, w);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, w);
      }
      if (again) p = s;
    }
    if (part == 0 && i < cc.y) *c = csub(z, p);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {
struct Tc64Images {
  int nbm, nbn;
  size_t a, b, r, c, rd, cd, list, chunk, chunks, total;  // byte offsets: A and B images, row and column exponents, rdef, cdef, listed entries
  int capacity;                                           // entries a CTA may list
};
Tc64Images tc64_images(int n, int m, int batch) {
  Tc64Images v;
  v.nbm = (n + kRows - 1) / kRows;
  v.nbn = (n + m + kCols - 1) / kCols;
  v.a = 0;
  v.b = v.a + size_t(batch) * v.nbm * kATile;
  v.r = v.b + size_t(batch) * v.nbn * kBTile;
  v.c = v.r + size_t(batch) * v.nbm * kRows * sizeof(int2);
  v.rd = v.c + size_t(batch) * v.nbn * kCols * sizeof(int2);
  v.cd = v.rd + size_t(batch) * v.nbm * kRows * 32;
  v.list = v.cd + size_t(batch) * v.nbn * kCols * 32;
  const int sms = current_sm_count();
  // a tile's entries at least, a quarter of the share of a CTA, 128 MB in all at most
  const size_t share = size_t(batch) * n * (n + m) / 4 / sms;
  v.capacity = int(std::max<size_t>(kRows * kCols, std::min<size_t>((size_t(1) << 22) / sms, share))) / kChunk * kChunk;
  v.chunk = v.list + size_t(sms) * v.capacity * sizeof(Tc64Entry);
  v.chunks = v.chunk + size_t(sms) * v.capacity / kChunk * sizeof(int2);
  v.total = v.chunks + 16;
  return v;
}
}  // namespace

size_t tc64_image_bytes(int n, int m, int batch) { return tc64_images(n, m, batch).total; }

void tc64_update(const BatchLayout& lay, int batch, int r_begin, int r_end, int c_begin, int c_end, int ka, int kb,
                 double2* M, uint8_t* images, int* alpha, int image_batch, long long wait_polls, cudaStream_t s) {
  const int rows = r_end - r_begin, cols = c_end - c_begin;
  if (rows <= 0 || cols <= 0 || kb <= 0 || image_batch <= 0) return;
  const Tc64Images im = tc64_images(lay.n, lay.m, image_batch);
  int2* rexp = reinterpret_cast<int2*>(images + im.r);
  int2* cexp = reinterpret_cast<int2*>(images + im.c);
  Tc64Entry* list = reinterpret_cast<Tc64Entry*>(images + im.list);
  int2* chunk = reinterpret_cast<int2*>(images + im.chunk);
  int* chunks = reinterpret_cast<int*>(images + im.chunks);
  const int sms = current_sm_count();
  ensure_smem_limit(reinterpret_cast<const void*>(tc64_update_kernel), size_t(kSmem));
  for (int b0 = 0; b0 < batch; b0 += image_batch) {
    const int nb = std::min(image_batch, batch - b0);
    double2* Mb = M + size_t(b0) * lay.stride;
    Tc64Work w;
    w.nbm = (rows + kRows - 1) / kRows;
    w.nbn = (cols + kCols - 1) / kCols;
    // Column tiles per unit: a unit loads the 128 KB of A digits once (about one tile's time), so up to 24 tiles
    // share them; fewer where that would leave SMs without a unit.
    const long long tiles = (long long)nb * w.nbm * w.nbn;
    const int want = int(std::max<long long>(1, std::min<long long>(24, (tiles + sms - 1) / sms)));
    w.nseg = (w.nbn + want - 1) / want;
    w.chunk = (w.nbn + w.nseg - 1) / w.nseg;
    w.units = nb * w.nbm * w.nseg;
    count_launch();
    tc64_scale_kernel<<<dim3(unsigned(w.nbm), unsigned(nb)), kRows, 0, s>>>(lay, r_begin, r_end, ka, kb, Mb, alpha, chunks);
    count_launch();
    tc64_split_kernel<<<dim3(unsigned(w.nbm + w.nbn), unsigned(nb)), 256, 0, s>>>(
        lay, r_begin, r_end, c_begin, c_end, ka, kb, Mb, alpha, images + im.a, images + im.b, rexp, cexp,
        images + im.rd, images + im.cd, w.nbm, im.nbm, im.nbn);
    count_launch();
    const unsigned ctas = unsigned(std::min(w.units, sms));
    tc64_update_kernel<<<ctas, kThreads, kSmem, s>>>(
        lay, r_begin, r_end, c_begin, c_end, ka, kb, Mb, images + im.a, images + im.b, rexp, cexp, im.nbm, im.nbn, w,
        alpha, nb * 32, list, chunk, chunks, im.capacity, wait_polls > 0 ? wait_polls : kTcWaitPolls);
    count_launch();
    tc64_recheck_kernel<<<unsigned(2 * sms), 4 * kChunk, 0, s>>>(lay, r_begin, c_begin, ka, kb, Mb, images + im.rd, images + im.cd,
                                                                 im.nbm, im.nbn, list, chunk, chunks);
  }
}

}  // namespace rfx
