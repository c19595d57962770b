// Tensor-core (tcgen05, sm_103a) trailing update of the FP32 LU:
//     C[r, c] -= sum_k A[r, k] B[k, c]      (complex, K <= 128)
// with A = L21 (rows below the block) and B = U12 (block rows, trailing
// columns); K is one 64-column block, or two when the elimination pairs them.
//
// Each complex product is formed from real FP16 MMAs with FP32 accumulation in
// tensor memory, using a two-term split x = hi + lo (hi = fp16(x), lo =
// fp16(x - hi)) and the three products hi*hi + hi*lo + lo*hi, which keeps the
// update at about FP32 accuracy:
//     Cr += Ar Br + Ai (-Bi)        Ci += Ar Bi + Ai Br
// FP16 carries the same 11 significant bits as TF32 at twice the rate and half
// the operand bytes; what it lacks is exponent range, which power-of-two scales
// give back: column k of A and row k of B are balanced by 2^g_k (so that no
// column of A is small in every row; a row of B that meets a zero column of A
// counts as zeros), each row of A and each column of B is scaled to a largest
// entry in [2^13, 2^14), and the epilogue takes the scales out again.  Entries
// more than 2^16 below their row's largest keep 2^-39 of that instead of their
// 22 bits, some 2^-35 of the largest product of row and column in a sum of 128.
// Where neither the sum nor C reaches 2^-13 of that product (2^28 in the scaled
// operands: the error stays below 2^-22 of the sum or C, what two terms keep of a
// value) the epilogue looks the entry's largest product up and, below 2^-11 of it,
// forms the sum again in FP32 multiply-adds (recheck_columns).  Most such entries
// are sums of large products that cancel (2% of a symmetric cluster's), and a bit
// mask of the row's and the column's large entries tells it at once.
// The operands are first written by tc_split_kernel into tile images that are
// already in the UMMA shared-memory layout (K-major, 64-byte rows, 64-byte
// swizzle), so the update kernel moves them with plain cp.async.bulk copies
// completed on mbarriers.  The update runs as one persistent, warp-specialised
// CTA per SM over 128 x 64 complex tiles (tc_update_persistent_kernel below).
// Every wait on an mbarrier is bounded; on timeout the kernel records an error
// flag, ends every role, waits for its copies and MMAs in flight, frees its
// tensor memory and returns.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "cplx.cuh"
#include "batched_lu.cuh"

namespace rfx {

namespace {

constexpr int BM = kTcBM;         // 128 rows per tile (MMA M)
constexpr int BN = kTcBN;         // 64 columns per tile (MMA N)
// Operand rows of 64 bytes with the 64-byte swizzle: a K chunk holds KC = 32
// FP16 values per row (56 KB of planes), and four chunks are in flight.
constexpr int kRowBytes = 64;
constexpr int KC = kRowBytes / 2;          // K elements per chunk
constexpr int A_PLANE = BM * kRowBytes;    // bytes per A plane per chunk (8 KB)
constexpr int B_PLANE = BN * kRowBytes;    // bytes per B plane per chunk (4 KB)
constexpr int A_PLANES = 4;       // re_hi, re_lo, im_hi, im_lo
// B slots -im_hi, re_hi, im_hi, -im_lo, re_lo, im_lo: each adjacent pair is one 2 BN-row B operand
constexpr int B_PLANES = 6;
constexpr int SMEM_OPS = A_PLANES * A_PLANE + B_PLANES * B_PLANE;  // 56 KB
constexpr long long kWaitLimit = kTcWaitPolls;  // drains of copies and MMAs in flight
constexpr int kChunks = kTcKMax / KC;  // K chunks per tile image (K up to 128)

// Byte offset of element (row, k) (k < KC, 2 bytes) in a K-major tile of 64-byte rows with the 64-byte swizzle: the
// 16-byte chunk index XOR (row / 2) % 4.
__device__ __forceinline__ int sw_offset(int row, int k) {
  return row * 64 + ((((k >> 3) ^ ((row >> 1) & 3))) << 4) + ((k & 7) << 1);
}

// 2^e, e clamped to the normal range
__device__ __forceinline__ float pow2(int e) { return __int_as_float(min(max(e + 127, 1), 254) << 23); }
// 2^-shift, also below the normal range (exact: shift_of ends at 140)
__device__ __forceinline__ float unscale(int shift) { return shift <= 126 ? pow2(-shift) : __int_as_float(1 << (149 - shift)); }
// v 2^x for |x| beyond what one factor holds
__device__ __forceinline__ float scaled(float v, int x) { return v * pow2(x >> 1) * pow2(x - (x >> 1)); }
// the shift that brings values below 2^e below 2^14 (denormals alone: all their bits above FP16's last)
__device__ __forceinline__ int shift_of(int e) { return min(14 - e, 140); }
// larger exponent field of the two parts (0: zero; denormals as 1)
__device__ __forceinline__ int field_of(float2 v) {
  const uint32_t m = max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu);
  return int(max(m >> 23, min(m, 1u)));
}
constexpr int kNone = -(1 << 20);  // exponent of a row or column of zeros, balance of a zero column of A
// the FP16 terms of a scaled value
__device__ __forceinline__ void split2(float x, __half& hi, __half& lo) {
  hi = __float2half_rn(x);
  lo = __float2half_rn(x - __half2float(hi));
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t umma_desc_sw(uint32_t saddr) {
  // start address >> 4 (14 bits), LBO = 1 (unused for swizzled K-major), SBO = 8 rows (the 8-row groups),
  // descriptor version 1, base offset 0, layout type 4 = 64-byte swizzle.
  return uint64_t((saddr >> 4) & 0x3FFFu) | (uint64_t(1) << 16) | (uint64_t((8 * kRowBytes) >> 4) << 32) |
         (uint64_t(1) << 46) | (uint64_t(4) << 61);
}

// kind::f16, D = F32, A = B = F16, both K-major, M = BM, N = 2 BN: one A plane against two adjacent B
// slots, into the adjacent accumulators [Cr | Ci].
constexpr uint32_t kIdesc = (1u << 4) | (uint32_t((2 * BN) >> 3) << 17) | (uint32_t(BM >> 4) << 24);

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(kIdesc), "r"(accumulate));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

constexpr float kWeakSum = 32768.f;  // 2^(28 - 13)
constexpr int kLost = 11, kLostRow = 5, kLostCol = kLost - kLostRow;
// How many powers of two a scaled value lies below 2^14 (63: 63 or more), kZero for a zero: a sum of two from kZero on means
// a product that is zero.
constexpr uint32_t kZero = 127;
__device__ __forceinline__ uint32_t deficit(float2 v) {
  const int f = field_of(v);
  return f == 0 ? kZero : uint32_t(min(max(140 - f, 0), 63));
}
// Eight columns of a warp's 32 rows, a row a lane, in the columns marked in `mine` (any: in some lane of the warp), whose
// sums are small: C -= the sum (in tensor memory at tr and ti) where the entry's largest product reaches 2^(28 - kLost),
// all are zero or C is not small, else C -= the sum in FP32 multiply-adds: an entry at a time by the whole warp while
// they are few (a lane alone would wait for 128 loads one after another), else the eight columns beside each other, a row
// a lane.  c: the lane's C in the first column; cs: the columns' scales; rdef, cdef: the deficits of the lane's row and of
// the first column; a0: A's first row of the warp; bcol: B's first column.  13 atoms with two spin channels (n = 416, up
// to half of the entries couplings of 1e-8 and less), 116 systems: updates 4.6 ms entry by entry, 1.6 ms so (0.37 where
// nothing is formed again).
__device__ __forceinline__ void recheck_columns(uint32_t any, uint32_t mine, uint32_t tr, uint32_t ti, float2* c, float rs,
                                                const float2* cs, const uint8_t* rdef, const uint8_t* cdef, const float2* a0,
                                                const float2* bcol, int lda, int kb) {
  const int lane = threadIdx.x & 31;
  uint32_t ur[8], ui[8], d[8];  // d: the smallest sums of two bytes (at most 254 each)
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    ur[j] = ui[j] = 0;
    d[j] = 0xfefefefeu;
    if (any >> j & 1u) {
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(ur[j]) : "r"(tr + uint32_t(j)));
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(ui[j]) : "r"(ti + uint32_t(j)));
    }
  }
  float2 v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = mine >> j & 1u ? c[size_t(lda) * j] : make_float2(0.f, 0.f);
#pragma unroll 1
  for (int q = 0; q < (kb + 15) / 16; ++q) {
    const uint4 x = reinterpret_cast<const uint4*>(rdef)[q];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (any >> j & 1u) {
        const uint4 y = reinterpret_cast<const uint4*>(cdef + j * kTcKMax)[q];
        d[j] = __vminu4(__vminu4(d[j], x.x + y.x), __vminu4(x.y + y.y, __vminu4(x.z + y.z, x.w + y.w)));
      }
  }
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(ur[0]), "+r"(ur[1]), "+r"(ur[2]), "+r"(ur[3]), "+r"(ur[4]), "+r"(ur[5]), "+r"(ur[6]), "+r"(ur[7]),
                 "+r"(ui[0]), "+r"(ui[1]), "+r"(ui[2]), "+r"(ui[3]), "+r"(ui[4]), "+r"(ui[5]), "+r"(ui[6]), "+r"(ui[7])::"memory");
  uint32_t again = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t pair = __vminu4(d[j], d[j] >> 16), least = min(pair & 255u, pair >> 8 & 255u);
    if (!(mine >> j & 1u)) continue;
    const float cf = cs[j].x;
    if (least > uint32_t(kLost) && least < kZero && fmaxf(fabsf(v[j].x), fabsf(v[j].y)) < (kWeakSum * rs) * cf)
      again |= 1u << j;
    else
      c[size_t(lda) * j] = make_float2(fmaf(-(__uint_as_float(ur[j]) * rs), cf, v[j].x),
                                       fmaf(-(__uint_as_float(ui[j]) * rs), cf, v[j].y));
  }
  const uint32_t lanes = __ballot_sync(0xffffffffu, again != 0);
  if (lanes == 0) return;
  if (__reduce_add_sync(0xffffffffu, __popc(again)) * 12 <= kb) {
    for (uint32_t rows = lanes; rows; rows &= rows - 1) {
      const int r = __ffs(rows) - 1;
      for (uint32_t cols = __shfl_sync(0xffffffffu, again, r); cols; cols &= cols - 1) {
        const int j = __ffs(cols) - 1;
        float2 acc = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < kTcKMax / 32; ++i) {
          const int k = 32 * i + lane;
          if (k < kb) cfma(acc, a0[size_t(lda) * k + r], bcol[size_t(lda) * j + k]);
        }
#pragma unroll
        for (int w = 16; w > 0; w /= 2) {
          acc.x += __shfl_xor_sync(0xffffffffu, acc.x, w);
          acc.y += __shfl_xor_sync(0xffffffffu, acc.y, w);
        }
        if (lane == r) c[size_t(lda) * j] = csub(c[size_t(lda) * j], acc);
      }
    }
    return;
  }
  const uint32_t cols = __reduce_or_sync(0xffffffffu, again);
  float2 acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int k0 = 0; k0 < kb; k0 += 32) {
    // 32 terms of the columns, one a lane, handed round by shuffles: the loads of all are in flight at once
    float2 bl[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      bl[j] = (cols >> j & 1u) && k0 + lane < kb ? bcol[size_t(lda) * j + k0 + lane] : make_float2(0.f, 0.f);
#pragma unroll 1
    for (int h = 0; h < 32 && k0 + h < kb; h += 8) {
      float2 a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = again && k0 + h + i < kb ? a0[size_t(lda) * (k0 + h + i) + lane] : make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (cols >> j & 1u)
#pragma unroll
          for (int i = 0; i < 8; ++i)
            cfma(acc[j], a[i], make_float2(__shfl_sync(0xffffffffu, bl[j].x, h + i), __shfl_sync(0xffffffffu, bl[j].y, h + i)));
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (again >> j & 1u) c[size_t(lda) * j] = csub(c[size_t(lda) * j], acc[j]);
}

// Bit j of a row's or column's mask stands for g consecutive k from g j on, g = 1, 2 or 4 for kb <= 32, 64 or 128: all of
// the row's entries lie within 2^kLostRow of its largest, one of the column's within 2^kLostCol; a common bit means a
// product above 2^(28 - kLost).  (A row or column of zeros has every bit: its sums are exact.)
__device__ __forceinline__ uint32_t large_mask(const uint8_t* def, int kb, bool row) {
  const uint32_t limit = 0x01010101u * uint32_t(row ? kLostRow : kLostCol);
  const uint32_t* d = reinterpret_cast<const uint32_t*>(def);
  uint32_t mask = 0;
#pragma unroll 4
  for (int q = 0; q < (kb + 3) / 4; ++q) {  // the bytes of a chunk beyond kb are 127
    const uint32_t in = __vcmpleu4(d[q], limit);
    if (kb <= 32) {
      mask |= (in & 1u | in >> 7 & 2u | in >> 14 & 4u | in >> 21 & 8u) << (4 * q);
    } else if (kb <= 64) {
      const uint32_t lo = in & 0xffffu, hi = in >> 16;
      mask |= (row ? uint32_t(lo == 0xffffu) | uint32_t(hi == 0xffffu) << 1 : uint32_t(lo != 0) | uint32_t(hi != 0) << 1) << (2 * q);
    } else {
      mask |= uint32_t(row ? in == 0xffffffffu : in != 0) << q;
    }
  }
  return mask;
}

}  // namespace

// ---------------------------------------------------------------------------
// scales and operand images: A[b][bm][chunk][plane] (8 KB), B[b][bn][chunk][plane] (4 KB), chunks of KC = 32; rdef and
// cdef, the deficit of each entry of A and B, a byte each, kTcKMax a row of A and a column of B
// ---------------------------------------------------------------------------
// alpha[b][k] = 256 + max over the rows of (exponent of A[row, k] - exponent of the row's largest entry), 0 where column k
// is zero in every row without infinities and NaN: g_k = 256 - alpha.  The table is zero before and is cleared again by the update kernel.
template <int kK>  // kb <= kK, a multiple of 32
__global__ void __launch_bounds__(BM) tc_scale_kernel(BatchLayout lay, int k, int kb, const float2* __restrict__ M,
                                                      int* __restrict__ alpha) {
  __shared__ int cmax[kTcKMax];
  const int b = blockIdx.y, lane = threadIdx.x & 31, row = k + kb + blockIdx.x * BM + int(threadIdx.x);
  cmax[threadIdx.x] = 0;
  const float2* A = M + size_t(b) * lay.stride + size_t(row) + size_t(lay.lda) * k;
  uint32_t f[kK / 4];  // exponent fields, four to a word
  int top = 0;
#pragma unroll
  for (int q = 0; q < kK / 32; ++q) {
    float2 v[32];  // (loaded first: 32 loads in flight)
#pragma unroll
    for (int i = 0; i < 32; ++i)
      v[i] = row < lay.n && 32 * q + i < kb ? A[size_t(lay.lda) * (32 * q + i)] : make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int x = field_of(v[i]), w = 8 * q + i / 4;
      f[w] = (i % 4 ? f[w] : 0u) | uint32_t(x) << (8 * (i % 4));
      top = max(top, x);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kK / 32; ++q) {
    int mine = 0;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int v = int(f[8 * q + i / 4] >> (8 * (i % 4))) & 255;
      const int m = __reduce_max_sync(0xffffffffu, v > 0 && top < 255 ? v - top + 256 : 0);
      if (lane == i) mine = m;
    }
    if (mine > 0) atomicMax(&cmax[32 * q + lane], mine);
  }
  __syncthreads();
  if (cmax[threadIdx.x] > 0) atomicMax(alpha + b * kTcKMax + threadIdx.x, cmax[threadIdx.x]);
}
static_assert(BM == kTcKMax, "one thread a column of the table");

__device__ __forceinline__ void load_balance(const int* alpha, int* gk) {
  if (threadIdx.x < kTcKMax) {
    const int a = alpha[threadIdx.x];
    gk[threadIdx.x] = a > 0 ? 256 - a : kNone;
  }
  __syncthreads();
}

// Operand images: blocks x < nbm take a row tile of A, the others a column tile of B.
__device__ __forceinline__ void split_a_tile(const BatchLayout& lay, int k, int kb, const float2* __restrict__ M,
                                             const int* gk, uint8_t* __restrict__ img, float2* __restrict__ rscale,
                                             uint8_t* rdef, int nbm, uint8_t* smem) {
  // The tile is read down the columns (coalesced in the column-major matrix),
  // turned around in shared memory, and written as 16-byte chunks of the
  // swizzled K-major rows.
  constexpr int TS = BM + 1;  // padded row of the transposed tile
  float2* T = reinterpret_cast<float2*>(smem);
  int(*rowe)[BM] = reinterpret_cast<int(*)[BM]>(smem + KC * TS * sizeof(float2));
  const int nch = (kb + KC - 1) / KC;
  const int bm = blockIdx.x, b = blockIdx.y;
  const int n = lay.n, r0 = k + kb + bm * BM;
  const float2* Mb = M + size_t(b) * lay.stride + size_t(lay.lda) * k;
  {
    const int r = threadIdx.x & (BM - 1), h = threadIdx.x / BM;
    int e = kNone;
    if (r0 + r < n)
#pragma unroll 8
      for (int kk = h; kk < kb; kk += 2) {
        const int f = field_of(Mb[size_t(r0 + r) + size_t(lay.lda) * kk]);
        if (f > 0) e = max(e, gk[kk] == kNone ? 129 : f - 126 + gk[kk]);  // (129: a row with an infinity or NaN)
      }
    rowe[h][r] = e;
    __syncthreads();
    if (h == 0) {
      e = max(e, rowe[1][r]);
      const int shift = e == kNone ? 0 : shift_of(e);  // |A| 2^g < 2^e along the row
      rowe[0][r] = shift;
      rscale[(size_t(b) * nbm + bm) * BM + r].x = e == kNone ? 0.f : unscale(shift);
    }
    __syncthreads();
  }
  for (int chunk = 0; chunk < nch; ++chunk) {
    for (int e = threadIdx.x; e < BM * KC; e += 256) {
      const int r = e % BM, kk = e / BM, kcol = chunk * KC + kk;
      float2 v = make_float2(0.f, 0.f);
      if (r0 + r < n && kcol < kb) {
        v = Mb[size_t(r0 + r) + size_t(lay.lda) * kcol];
        const int g = gk[kcol], x = rowe[0][r] + (g == kNone ? 0 : g);
        v = make_float2(scaled(v.x, x), scaled(v.y, x));
      }
      T[kk * TS + r] = v;
    }
    __syncthreads();
    uint8_t* base = img + ((size_t(b) * nbm + bm) * kChunks + chunk) * size_t(A_PLANES) * A_PLANE;
    for (int e = threadIdx.x; e < BM * (KC / 8); e += 256) {
      const int k8 = e % (KC / 8), r = e / (KC / 8);
      __align__(16) __half q[A_PLANES][8];
      uint32_t d[2] = {0, 0};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 v = T[(8 * k8 + i) * TS + r];
        split2(v.x, q[0][i], q[1][i]);
        split2(v.y, q[2][i], q[3][i]);
        d[i / 4] |= deficit(v) << (8 * (i % 4));
      }
      *reinterpret_cast<uint2*>(rdef + ((size_t(b) * nbm + bm) * BM + r) * kTcKMax + chunk * KC + 8 * k8) = make_uint2(d[0], d[1]);
      const int off = sw_offset(r, 8 * k8);
#pragma unroll
      for (int p = 0; p < A_PLANES; ++p)
        *reinterpret_cast<uint4*>(base + size_t(p) * A_PLANE + off) = *reinterpret_cast<const uint4*>(q[p]);
    }
    __syncthreads();
  }
  if (threadIdx.x < BM) {
    const size_t at = (size_t(b) * nbm + bm) * BM + threadIdx.x;
    rscale[at].y = __uint_as_float(rscale[at].x == 0.f ? ~0u : large_mask(rdef + at * kTcKMax, kb, true));
  }
}

__device__ __forceinline__ void split_b_tile(const BatchLayout& lay, int bn, int k, int kb, int col_end,
                                             const float2* __restrict__ M, const int* gk, uint8_t* __restrict__ img,
                                             float2* __restrict__ cscale, uint8_t* cdef, int nbn, uint8_t* smem) {
  int* cole = reinterpret_cast<int*>(smem);
  const int b = blockIdx.y, c0 = k + kb + bn * BN;
  const float2* Mb = M + size_t(b) * lay.stride + size_t(k);
  // column exponents: one warp a column, lanes down its rows
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int c = wid; c < BN; c += 8) {
    int e = kNone;
    if (c0 + c < col_end)
      for (int kk = lane; kk < kb; kk += 32) {
        // an entry that meets only zeros of A must not set the column's scale
        const int f = field_of(Mb[size_t(kk) + size_t(lay.lda) * (c0 + c)]);
        if (f > 0 && gk[kk] != kNone) e = max(e, f - 126 - gk[kk]);
        else if (f == 255) e = max(e, 129);  // an infinity or NaN reaches every row
      }
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) {
      const int shift = e == kNone ? 0 : shift_of(e);  // |B| 2^-g < 2^e along the column
      cole[c] = shift;
      cscale[(size_t(b) * nbn + bn) * BN + c].x = e == kNone ? 0.f : unscale(shift);
    }
  }
  __syncthreads();
  const int nch = (kb + KC - 1) / KC;
  // a thread takes eight consecutive rows of a column: one 16-byte chunk of each slot
  for (int e = threadIdx.x; e < BN * nch * (KC / 8); e += 256) {
    const int k8 = e % (nch * (KC / 8)), c = e / (nch * (KC / 8)), chunk = k8 / (KC / 8), kin = 8 * (k8 % (KC / 8));
    __align__(16) __half q[B_PLANES][8];
    uint32_t d[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int krow = 8 * k8 + i;
      float2 v = make_float2(0.f, 0.f);
      if (c0 + c < col_end && krow < kb) {
        v = Mb[size_t(krow) + size_t(lay.lda) * (c0 + c)];
        const int g = gk[krow], x = g == kNone ? 0 : cole[c] - g;
        v = g == kNone && field_of(v) < 255 ? make_float2(0.f, 0.f) : make_float2(scaled(v.x, x), scaled(v.y, x));
      }
      __half rh, rl, ih, il;
      split2(v.x, rh, rl);
      split2(v.y, ih, il);
      q[0][i] = __hneg(ih);
      q[1][i] = rh;
      q[2][i] = ih;
      q[3][i] = __hneg(il);
      q[4][i] = rl;
      q[5][i] = il;
      d[i / 4] |= deficit(v) << (8 * (i % 4));
    }
    *reinterpret_cast<uint2*>(cdef + ((size_t(b) * nbn + bn) * BN + c) * kTcKMax + 8 * k8) = make_uint2(d[0], d[1]);
    uint8_t* base = img + ((size_t(b) * nbn + bn) * kChunks + chunk) * size_t(B_PLANES) * B_PLANE + sw_offset(c, kin);
#pragma unroll
    for (int p = 0; p < B_PLANES; ++p)
      *reinterpret_cast<uint4*>(base + size_t(p) * B_PLANE) = *reinterpret_cast<const uint4*>(q[p]);
  }
  __syncthreads();
  if (threadIdx.x < BN) {
    const size_t at = (size_t(b) * nbn + bn) * BN + threadIdx.x;
    cscale[at].y = __uint_as_float(cscale[at].x == 0.f ? ~0u : large_mask(cdef + at * kTcKMax, kb, false));
  }
}

__global__ void __launch_bounds__(256) tc_split_kernel(BatchLayout lay, int k, int kb, int col_end,
                                                       const float2* __restrict__ M, const int* __restrict__ alpha,
                                                       uint8_t* __restrict__ aimg, uint8_t* __restrict__ bimg,
                                                       float2* __restrict__ rscale, float2* __restrict__ cscale,
                                                       uint8_t* rdef, uint8_t* cdef, int nbm,
                                                       int nbm_all, int nbn_all) {
  __shared__ __align__(16) uint8_t smem[KC * (BM + 1) * sizeof(float2) + 2 * BM * sizeof(int)];
  __shared__ int gk[kTcKMax];
  load_balance(alpha + blockIdx.y * kTcKMax, gk);
  if (int(blockIdx.x) < nbm) split_a_tile(lay, k, kb, M, gk, aimg, rscale, rdef, nbm_all, smem);
  else split_b_tile(lay, int(blockIdx.x) - nbm, k, kb, col_end, M, gk, bimg, cscale, cdef, nbn_all, smem);
}

// ---------------------------------------------------------------------------
// the update, persistent and warp-specialised
// ---------------------------------------------------------------------------
// One CTA per SM walks the tiles t = blockIdx.x, blockIdx.x + gridDim.x, ...
// (t -> matrix b, row tile bm, column tile bn, bn fastest).  Roles:
//   warp 0   producer: bulk-copies each K-chunk (56 KB of planes) into a
//            four-stage ring, waiting for the stage to be released;
//   warp 1   MMA: 12 tcgen05.mma (N = 128: [Cr | Ci]) per chunk into one of four TMEM accumulators
//            (128 columns each), releasing the stage with tcgen05.commit and
//            signalling the tile's accumulator the same way;
//   warps 2-17   four epilogue groups of four warps, group g taking the tiles
//            i = g mod 4 of the CTA: C of the tile is loaded into registers
//            16 columns ahead, then tcgen05.ld, subtract, store, release.
// The copies of tile i + 1, its MMAs and the epilogues of the previous tiles
// overlap; four epilogues are in flight per SM, which keeps enough C loads
// outstanding to approach the bandwidth of moving C.  Every wait is bounded; a timeout sets
// the error flag and a shared abort flag that ends every role's loop, then
// the producer waits (bounded) for its copies still in flight and the MMA
// thread for its MMAs before the tensor memory is freed.
constexpr int kPStages = 4;                    // operand ring depth (4 x 56 KB)
constexpr int kPGroups = 4;                     // epilogue groups of 4 warps, one accumulator each
constexpr int kPThreads = 64 + kPGroups * 128;  // producer warp, MMA warp, epilogue groups
constexpr uint32_t kPTmemCols = 512;  // kPGroups * 128 columns, rounded up to a power of two
// barriers: full[kPStages], empty[kPStages], acc_full[kPGroups], acc_empty[kPGroups], drain
constexpr int kBarFull = 0, kBarEmpty = kPStages, kBarAccFull = 2 * kPStages, kBarAccEmpty = 2 * kPStages + kPGroups,
              kBarDrain = 2 * kPStages + 2 * kPGroups;
static_assert((kBarDrain + 1) * 8 <= 256, "barrier area");
constexpr int kPSmem = kPStages * SMEM_OPS + 1024 + 512;
static_assert(kPSmem <= 227 * 1024, "dynamic shared memory per CTA");

__device__ __forceinline__ bool mbar_wait_or_abort(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                                   int* err_flag, long long polls) {
  const uint64_t t0 = global_ns();
  for (long long it = 0; it < polls; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 255) == 255) {
      if (*abort_flag) return false;
      if (global_ns() - t0 > 1000000000ull) break;
    }
  }
  *abort_flag = 1;
  atomicExch(err_flag, 1);
  return false;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__global__ void __launch_bounds__(kPThreads, 1) tc_update_persistent_kernel(
    BatchLayout lay, int k, int kb, int col_end, float2* __restrict__ M, const uint8_t* __restrict__ aimg,
    const uint8_t* __restrict__ bimg, const float2* __restrict__ rscale, const float2* __restrict__ cscale,
    const uint8_t* __restrict__ rdef, const uint8_t* __restrict__ cdef, int nbm_all, int nbn_all, int nbm, int nbn, int batch, int* __restrict__ alpha, int* __restrict__ err_flag, const int* skip,
    long long polls) {
  extern __shared__ uint8_t smraw[];
  const uint32_t raw = smem_u32(smraw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* const gbase = smraw + (sbase - raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(gbase + kPStages * SMEM_OPS);
  // bars at kBarFull / kBarEmpty / kBarAccFull / kBarAccEmpty / kBarDrain; then the TMEM slot and flags
  auto bar = [&](int i) { return smem_u32(&bars[i]); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + kPStages * SMEM_OPS + 256);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + kPStages * SMEM_OPS + 260);
  int* consumed = reinterpret_cast<int*>(gbase + kPStages * SMEM_OPS + 264);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = lay.n;
  const int per_matrix = nbm * nbn;
  const int total = per_matrix * batch;  // the host keeps this below 2^31
  const int nchunks = (kb + KC - 1) / KC;  // 1 .. kChunks
  // the balance table, read by the split kernels before: zero again for the next update
  for (int i = blockIdx.x * kPThreads + tid; i < batch * kTcKMax; i += gridDim.x * kPThreads) alpha[i] = 0;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kPTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    for (int i = 0; i < kPStages; ++i) {
      mbar_init(bar(kBarFull + i), 1);   // full: the producer's expect_tx
      mbar_init(bar(kBarEmpty + i), 1);  // empty: one commit
    }
    for (int a = 0; a < kPGroups; ++a) {
      mbar_init(bar(kBarAccFull + a), 1);     // accumulator full: one commit
      mbar_init(bar(kBarAccEmpty + a), 128);  // accumulator empty: the 128 threads of one epilogue group
    }
    mbar_init(bar(kBarDrain), 1);  // drain
    *abort_flag = 0;
    *consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  auto tile_of = [&](int t, int& b, int& bm, int& bn) {
    b = t / per_matrix;
    const int rem = t - b * per_matrix;
    bm = rem / nbn;
    bn = rem - bm * nbn;
  };

  if (warp == 0) {
    // ---- producer ----
    if (lane == 0) {
      long long c = 0;  // chunks issued
      for (int t = blockIdx.x; t < total && !*abort_flag; t += gridDim.x) {
        int b, bm, bn;
        tile_of(t, b, bm, bn);
        if (skip && skip[b]) continue;
        const uint8_t* ab = aimg + (size_t(b) * nbm_all + bm) * kChunks * size_t(A_PLANES) * A_PLANE;
        const uint8_t* bb = bimg + (size_t(b) * nbn_all + bn) * kChunks * size_t(B_PLANES) * B_PLANE;
        bool ok = true;
        for (int ch = 0; ch < nchunks; ++ch, ++c) {
          const int st = int(c % kPStages);
          const uint32_t ph = uint32_t((c / kPStages) & 1);
          if (!mbar_wait_or_abort(bar(kBarEmpty + st), ph ^ 1u, abort_flag, err_flag, polls)) { ok = false; break; }
          const uint32_t sA = sbase + uint32_t(st) * SMEM_OPS, sB = sA + A_PLANES * A_PLANE;
          mbar_expect_tx(bar(kBarFull + st), uint32_t(SMEM_OPS));
          const uint8_t* ach = ab + size_t(ch) * A_PLANES * A_PLANE;
          const uint8_t* bch = bb + size_t(ch) * B_PLANES * B_PLANE;
          for (int p = 0; p < A_PLANES; ++p) bulk_copy(sA + p * A_PLANE, ach + size_t(p) * A_PLANE, A_PLANE, bar(kBarFull + st));
          for (int p = 0; p < B_PLANES; ++p) bulk_copy(sB + p * B_PLANE, bch + size_t(p) * B_PLANE, B_PLANE, bar(kBarFull + st));
        }
        if (!ok) break;
      }
      if (*abort_flag) {
        // copies issued but not yet seen complete by the MMA thread: wait for them (bounded)
        for (long long q = *(volatile int*)consumed; q < c; ++q) {
          const uint64_t t0 = global_ns();
          for (long long it = 0; it < kWaitLimit; ++it) {
            uint32_t done;
            asm volatile(
                "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                : "=r"(done)
                : "r"(bar(kBarFull + int(q % kPStages))), "r"(uint32_t((q / kPStages) & 1))
                : "memory");
            if (done || ((it & 1023) == 1023 && global_ns() - t0 > 1000000000ull)) break;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ----
    if (lane == 0) {
      long long c = 0, i = 0;  // chunks consumed, tiles of this CTA
      bool issued = false;
      for (int t = blockIdx.x; t < total && !*abort_flag; t += gridDim.x) {
        int b, bm, bn;
        tile_of(t, b, bm, bn);
        if (skip && skip[b]) continue;
        const int a = int(i % kPGroups);
        if (!mbar_wait_or_abort(bar(kBarAccEmpty + a), uint32_t(((i / kPGroups) & 1) ^ 1), abort_flag, err_flag, polls))
          break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_r = tmem + uint32_t(a * 128), tmem_i = tmem_r + 64;
        bool ok = true;
        for (int ch = 0; ch < nchunks; ++ch, ++c) {
          const int st = int(c % kPStages);
          if (!mbar_wait_or_abort(bar(kBarFull + st), uint32_t((c / kPStages) & 1), abort_flag, err_flag, polls)) { ok = false; break; }
          *(volatile int*)consumed = int(c + 1);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sA = sbase + uint32_t(st) * SMEM_OPS, sB = sA + A_PLANES * A_PLANE;
          for (int ks = 0; ks < KC / 16; ++ks) {
            const uint32_t koff = uint32_t(ks * 32);
            auto ad = [&](int p) { return umma_desc_sw(sA + p * A_PLANE + koff); };
            auto bd = [&](int p) { return umma_desc_sw(sB + p * B_PLANE + koff); };
            const uint32_t acc0 = (ch == 0 && ks == 0) ? 0u : 1u;
            // [Cr | Ci] += Ar hi [Br hi | Bi hi] + Ar hi [Br lo | Bi lo] + Ar lo [Br hi | Bi hi]
            //            + Ai hi [-Bi hi | Br hi] + Ai hi [-Bi lo | Br lo] + Ai lo [-Bi hi | Br hi],
            // i.e. Cr += Ar Br + Ai (-Bi), Ci += Ar Bi + Ai Br, each hi*hi + hi*lo + lo*hi
            (void)tmem_i;
            mma_f16(tmem_r, ad(0), bd(1), acc0);
            mma_f16(tmem_r, ad(0), bd(4), 1u);
            mma_f16(tmem_r, ad(1), bd(1), 1u);
            mma_f16(tmem_r, ad(2), bd(0), 1u);
            mma_f16(tmem_r, ad(2), bd(3), 1u);
            mma_f16(tmem_r, ad(3), bd(0), 1u);
          }
          issued = true;
          umma_commit(bar(kBarEmpty + st));  // the stage is free once these MMAs have read it
        }
        if (!ok) break;
        umma_commit(bar(kBarAccFull + a));  // the accumulator is complete
        ++i;
      }
      if (issued) {
        // every MMA of this CTA has completed before the tensor memory is freed
        umma_commit(bar(kBarDrain));
        const uint64_t t0 = global_ns();
        for (long long it = 0; it < kWaitLimit; ++it) {
          uint32_t done;
          asm volatile(
              "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
              : "=r"(done)
              : "r"(bar(kBarDrain))
              : "memory");
          if (done || ((it & 1023) == 1023 && global_ns() - t0 > 1000000000ull)) break;
        }
      }
    }
  } else {
    // ---- epilogue groups ----
    const int g = (warp - 2) >> 2;     // group g: warps 2 + 4g .. 5 + 4g
    const int quarter = warp & 3;      // tensor-memory lanes [32 quarter, 32 quarter + 32)
    const uint32_t lane_off = uint32_t(quarter * 32) << 16;
    long long i = 0;                   // tiles of this CTA
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
      // every branch below is uniform across the warp (tcgen05.ld is .sync.aligned)
      if (__shfl_sync(0xffffffffu, *abort_flag, 0)) break;
      int b, bm, bn;
      tile_of(t, b, bm, bn);
      if (skip && skip[b]) continue;
      const long long mine = i++;
      if (mine % kPGroups != g) continue;
      const int r0 = k + kb + bm * BM, c0 = k + kb + bn * BN;
      const int row = r0 + quarter * 32 + lane;
      const bool row_ok = row < n;
      const int ld = lay.lda;  // column offsets within a tile stay far below 2^31 elements
      const float2 rsm = rscale[(size_t(b) * nbm_all + bm) * BM + quarter * 32 + lane];
      const float rs = rsm.x;
      const uint32_t rmask = __float_as_uint(rsm.y);
      const float2* cs = cscale + (size_t(b) * nbn_all + bn) * BN;
      float2* crow = M + size_t(b) * lay.stride + size_t(row) + size_t(lay.lda) * size_t(c0);
      // C of 16 columns at a time, an entry of the next part loaded as soon as this one's is used
      float2 cn[16];
#pragma unroll
      for (int j = 0; j < 16; ++j)
        cn[j] = (row_ok && c0 + j < col_end) ? crow[j * ld] : make_float2(0.f, 0.f);
      const bool ready = mbar_wait_or_abort(bar(kBarAccFull + g), uint32_t((mine / kPGroups) & 1), abort_flag, err_flag, polls);
      if (!__all_sync(0xffffffffu, ready)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_r = tmem + uint32_t(g * 128) + lane_off, tmem_i = tmem_r + 64;
      unsigned long long weak_cols = 0;
#pragma unroll 1
      for (int part = 0; part < BN / 16; ++part) {
        uint32_t lost = 0;  // columns of the part whose sums may have lost their terms: C stays as it is
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t cr[8], ci[8];
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                       : "=r"(cr[0]), "=r"(cr[1]), "=r"(cr[2]), "=r"(cr[3]), "=r"(cr[4]), "=r"(cr[5]), "=r"(cr[6]),
                         "=r"(cr[7])
                       : "r"(tmem_r + uint32_t(part * 16 + h * 8)));
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                       : "=r"(ci[0]), "=r"(ci[1]), "=r"(ci[2]), "=r"(ci[3]), "=r"(ci[4]), "=r"(ci[5]), "=r"(ci[6]),
                         "=r"(ci[7])
                       : "r"(tmem_i + uint32_t(part * 16 + h * 8)));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int i = h * 8 + j, off = part * 16 + i;
            if (row_ok && c0 + off < col_end) {
              float2 v = cn[i];
              // the row's factor first: the column's may be 2^115, and either may be denormal
              const float2 csm = cs[off];
              const float cf = csm.x, pr = __uint_as_float(cr[j]), pi = __uint_as_float(ci[j]);
              // (no branch here: it would part the loads of C from one another)
              const bool weak = (fmaxf(fabsf(pr), fabsf(pi)) < kWeakSum) & ((rmask & __float_as_uint(csm.y)) == 0);
              lost |= weak ? 1u << i : 0u;
              crow[off * ld] = make_float2(fmaf(weak ? 0.f : -(pr * rs), cf, v.x), fmaf(weak ? 0.f : -(pi * rs), cf, v.y));
            }
            if (part + 1 < BN / 16)
              cn[i] = (row_ok && c0 + off + 16 < col_end) ? crow[(off + 16) * ld] : make_float2(0.f, 0.f);
          }
        }
        weak_cols |= static_cast<unsigned long long>(lost) << (16 * part);
      }
      // the columns in which a row of this warp has one (the accumulators are still there; C's registers are free)
      const uint32_t weak_lo = uint32_t(weak_cols), weak_hi = uint32_t(weak_cols >> 32);
      const unsigned long long any = (static_cast<unsigned long long>(__reduce_or_sync(0xffffffffu, weak_hi)) << 32) |
                                     __reduce_or_sync(0xffffffffu, weak_lo);
      if (any) {
#pragma unroll 1
        for (int off = 0; off < BN; off += 8) {
          const uint32_t any8 = uint32_t(any >> off) & 255u;
          if (any8 == 0) continue;
          const float2* Mb = M + size_t(b) * lay.stride + size_t(k);
          recheck_columns(any8, uint32_t(weak_cols >> off) & 255u, tmem_r + uint32_t(off), tmem_i + uint32_t(off), crow + off * ld, rs,
                          cs + off, rdef + ((size_t(b) * nbm_all + bm) * BM + quarter * 32 + lane) * kTcKMax,
                          cdef + ((size_t(b) * nbn_all + bn) * BN + off) * kTcKMax,
                          Mb + size_t(ld) * k + size_t(r0 - k + quarter * 32), Mb + size_t(ld) * (c0 + off), ld, kb);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(bar(kBarAccEmpty + g));  // the accumulator may be overwritten
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPTmemCols));
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {
struct TcImages {
  int nbm, nbn;
  size_t a, b, r, c, rd, cd, total;  // byte offsets of the A and B images, the row and column scales (with masks), rdef and cdef
};
TcImages tc_images(int n, int m, int batch) {
  TcImages v;
  v.nbm = (n + BM - 1) / BM;
  v.nbn = (n + m + BN - 1) / BN;
  v.a = 0;
  v.b = v.a + size_t(batch) * v.nbm * kChunks * A_PLANES * A_PLANE;
  v.r = v.b + size_t(batch) * v.nbn * kChunks * B_PLANES * B_PLANE;
  v.c = v.r + size_t(batch) * v.nbm * BM * sizeof(float2);
  v.rd = v.c + size_t(batch) * v.nbn * BN * sizeof(float2);
  v.cd = v.rd + size_t(batch) * v.nbm * BM * kTcKMax;
  v.total = v.cd + size_t(batch) * v.nbn * BN * kTcKMax;
  return v;
}
}  // namespace

size_t tc_image_bytes(int n, int m, int batch) { return tc_images(n, m, batch).total; }

void tc_trailing_update(const BatchLayout& lay, int batch, int k, int kb, int col_end, float2* M, uint8_t* images,
                        int* alpha, int* err_flag, const int* skip, long long wait_polls, KernelSpans* spans,
                        cudaStream_t s) {
  const int rows = lay.n - (k + kb), cols = col_end - (k + kb);
  if (rows <= 0 || cols <= 0 || kb <= 0) return;
  const TcImages im = tc_images(lay.n, lay.m, batch);
  uint8_t *aimg = images + im.a, *bimg = images + im.b;
  float2 *rscale = reinterpret_cast<float2*>(images + im.r), *cscale = reinterpret_cast<float2*>(images + im.c);
  const int nbm_all = im.nbm, nbn_all = im.nbn;
  const int nbm = (rows + BM - 1) / BM, nbn = (cols + BN - 1) / BN;
  const dim3 sgrid{unsigned(nbm), unsigned(batch)};
  count_launch();
  if (kb <= 32) tc_scale_kernel<32><<<sgrid, BM, 0, s>>>(lay, k, kb, M, alpha);
  else if (kb <= 64) tc_scale_kernel<64><<<sgrid, BM, 0, s>>>(lay, k, kb, M, alpha);
  else tc_scale_kernel<kTcKMax><<<sgrid, BM, 0, s>>>(lay, k, kb, M, alpha);
  count_launch();
  tc_split_kernel<<<dim3(unsigned(nbm + nbn), unsigned(batch)), 256, 0, s>>>(lay, k, kb, col_end, M, alpha, aimg, bimg,
                                                                            rscale, cscale, images + im.rd, images + im.cd, nbm,
                                                                            nbm_all, nbn_all);
  const int sms = current_sm_count();
  ensure_smem_limit(reinterpret_cast<const void*>(tc_update_persistent_kernel), size_t(kPSmem));
  const long long tiles = (long long)nbm * nbn * batch;
  if (tiles > 0x7fffffffLL) {  // the kernel numbers tiles with 32-bit integers
    if (err_flag) cudaMemsetAsync(err_flag, 0xff, sizeof(int), s);
    return;
  }
  const unsigned grid = unsigned(tiles < sms ? tiles : sms);
  const bool prof = spans && spans->on;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (prof) {
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
  }
  count_launch();
  tc_update_persistent_kernel<<<grid, kPThreads, kPSmem, s>>>(lay, k, kb, col_end, M, aimg, bimg, rscale, cscale,
                                                              images + im.rd, images + im.cd, nbm_all,
                                                              nbn_all, nbm, nbn, batch, alpha, err_flag, skip,
                                                              wait_polls > 0 ? wait_polls : kTcWaitPolls);
  if (prof) {
    cudaEventRecord(e1, s);
    spans->spans.push_back({e0, e1});
  }
}

}  // namespace rfx
