// Batched right-preconditioned BiCGSTAB for the dense FMS systems.
//
// The reference's iterative form solves each absorber column on its own
// (fms_bicgstab_solve, crates/refeff-core/src/fms/internals/iterative.rs:181-254),
// so every column streams the whole matrix once per matrix-vector product.
// Here the m absorber columns of every energy in a batch advance together:
// one product kernel reads each FP32 system matrix once per product for all m
// columns, and the per-column scalars (rho, alpha, omega) live in FP64 with
// FP64 dot-product accumulation.  Right preconditioning by a diagonal D or a
// block diagonal (one channel block per atom; the learned form) solves
// A P y = b and returns x = P y.
//
// Iteration (van der Vorst), per column:
//   beta = (rho_new / rho)(alpha / omega);  p = r + beta (p - omega v);  p^ = D p
//   v = A p^;  alpha = rho_new / (r~, v);   s = r - alpha v;  s^ = D s
//   t = A s^;  omega = (t, s) / (t, t);     x += alpha p^ + omega s^;  r = s - omega t
//   rho_new = (r~, r);  stop when |r| <= tol |b|.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "bicgstab.cuh"
#include "cplx.cuh"

namespace rfx {
namespace {

// scalar slots per (matrix, column)
// complex values take two slots (re, im)
enum : int { kRho = 0, kAlpha = 2, kOmega = 4, kB2 = 6, kAcc1 = 7, kAcc2 = 9, kAcc3 = 11, kAcc4 = 12 };
static_assert(kAcc4 < kBicgScalars, "scalar slots");
enum : int { kX = 0, kR = 1, kRh = 2, kP = 3, kV = 4, kPh = 5, kSh = 6, kT = 7 };

constexpr int kVecThreads = 256, kVecRowsPerThread = 4, kVecRows = kVecThreads * kVecRowsPerThread;

struct View {
  int n, m, lda, batch;
  float2* vec;
  double* sc;
  int* state;
  int* done;
  float2* part;    // partial products of slices 1..nsplit-1 of the last split product
  int nsplit = 1;  // column slices of that product (1: not split)
  // tensor-core product (image NULL without it): the exponents of A's rows, of X's columns per vector block, and X as
  // the product's operand
  unsigned* amax = nullptr;
  int* xexp = nullptr;
  uint8_t* image = nullptr;
  int xblocks = 0;           // vector blocks of a column
  int tc_n = 0, tc_three = 0;
  const int* act = nullptr;  // running matrices, compacted (-1 past the count); NULL: blockIdx.y is the matrix
  __device__ __forceinline__ int matrix() const { return act ? act[blockIdx.y] : int(blockIdx.y); }
  __device__ float2* v(int k, int b, int c) const {
    return vec + (size_t(k) * batch + b) * size_t(lda) * m + size_t(lda) * c;
  }
  __device__ float2* pv(int slice, int b, int c) const {  // slice >= 1
    return part + ((size_t(slice - 1) * batch + b) * m + c) * size_t(lda);
  }
  __device__ double* s(int b, int c) const { return sc + (size_t(b) * m + c) * kBicgScalars; }
  // y[i] += the other slices' partial products, written back (slice 0 wrote y)
  __device__ __forceinline__ float2 gather(float2* y, int b, int c, int i) const {
    float2 a = y[i];
    if (nsplit > 1) {
      for (int sl = 1; sl < nsplit; ++sl) a = cadd(a, pv(sl, b, c)[i]);
      y[i] = a;
    }
    return a;
  }
};

__device__ __forceinline__ double2 cdot_acc(double2 acc, float2 a, float2 b) {  // acc += conj(a) b
  acc.x += double(a.x) * b.x + double(a.y) * b.y;
  acc.y += double(a.x) * b.y - double(a.y) * b.x;
  return acc;
}

__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < kVecThreads / 32; ++i) t += red[i];
  return t;  // valid on thread 0
}

// Adds the block's partial sums of up to three values to sc slots (one atomic each).
__device__ __forceinline__ void block_accumulate(double* slot0, double a, double* slot1, double b, double* slot2,
                                                 double c) {
  __shared__ double red[kVecThreads / 32];
  const double ta = block_sum(a, red);
  const double tb = slot1 ? block_sum(b, red) : 0.0;
  const double tc = slot2 ? block_sum(c, red) : 0.0;
  if (threadIdx.x == 0) {
    atomicAdd(slot0, ta);
    if (slot1) atomicAdd(slot1, tb);
    if (slot2) atomicAdd(slot2, tc);
  }
}

// The larger |component|'s bits; ordered as the magnitudes are, NaN above all.
__device__ __forceinline__ unsigned abs_bits(float2 v) {
  return max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu);
}
// The exponent s with max 2^s in [2^top, 2^(top + 1)) for a maximum given by its bits (0, infinity and NaN included:
// the power of two stays a normal number).
__device__ __forceinline__ int scale_exponent(unsigned bits, int top) {
  const int e = min(max(int(bits >> 23), 1), 254);
  return min(top + 127 - e, 126);
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float(unsigned(e + 127) << 23); }  // -126 <= e <= 127
// hi / lo FP16 parts of two values
__device__ __forceinline__ void tc_split(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(x0 - f.x, x1 - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// Byte offset of 16-byte chunk `chunk` of row `row` in a K-major tile of 32-byte rows with the 32-byte swizzle.
__device__ __forceinline__ int tc_sw32(int row, int chunk) { return row * 32 + ((chunk ^ ((row >> 2) & 1)) << 4); }
// The scaled maximum lies below 2^(kTcTop + 1): one less for the three-product form, whose sums Ar + Ai double it.
__device__ __forceinline__ int tc_top(bool three) { return three ? 13 : 14; }
__host__ __device__ __forceinline__ constexpr int tc_x_slots(bool three) { return three ? 6 : 8; }

// The block's rows of column c of the next product's X (x[k] = row k kVecThreads + threadIdx.x of the block, 0 past
// n) as the B operand of the tensor-core product: scaled by a power of two that brings the block's largest component
// to [2^14, 2^15), split into two FP16 terms and stored in the slabs' slots (bicg_tc_matvec_kernel).  Neighbouring
// lanes hold neighbouring rows; the even one stores the hi terms of both, the odd one the lo terms, 4 bytes at a time.
// Written here, once a product, the operand costs its 33 row tiles (n = 4112) one bulk copy each instead of a
// conversion each.
__device__ __forceinline__ void store_x_image(const View& w, int b, int c, const float2 (&x)[kVecRowsPerThread]) {
  if (!w.image) return;
  __shared__ unsigned red[kVecThreads / 32];
  unsigned m = 0;
#pragma unroll
  for (int k = 0; k < kVecRowsPerThread; ++k) m = max(m, abs_bits(x[k]));
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kVecThreads / 32; ++i) m = max(m, red[i]);
  const int e = scale_exponent(m, tc_top(w.tc_three));
  if (threadIdx.x == 0) w.xexp[(size_t(b) * w.m + c) * w.xblocks + blockIdx.x] = e;
  const float f = pow2(e);
  const int plane = w.tc_n * 32, slab_bytes = tc_x_slots(w.tc_three) * plane, slabs = (w.n + 15) / 16;
  const bool odd = threadIdx.x & 1;
  uint8_t* img = w.image + size_t(b) * slabs * slab_bytes;
#pragma unroll
  for (int k = 0; k < kVecRowsPerThread; ++k) {
    const int i = blockIdx.x * kVecRows + k * kVecThreads + int(threadIdx.x);
    uint32_t hi, lo, shi, slo;  // (re, im) pairs; of re + im in the low half
    const float re = x[k].x * f, im = x[k].y * f;
    tc_split(re, im, hi, lo);
    tc_split(re + im, 0.f, shi, slo);
    const uint32_t own = odd ? lo : hi, other = __shfl_xor_sync(0xffffffffu, odd ? hi : lo, 1);
    const uint32_t sown = odd ? slo : shi, sother = __shfl_xor_sync(0xffffffffu, odd ? shi : slo, 1);
    if ((i >> 4) >= slabs) continue;
    const uint32_t r0 = odd ? other : own, r1 = odd ? own : other;  // the even row's, the odd row's
    const uint32_t rr = __byte_perm(r0, r1, 0x5410), ii = __byte_perm(r0, r1, 0x7632);
    uint8_t* q = img + size_t(i >> 4) * slab_bytes + tc_sw32(c, (i >> 3) & 1) + 2 * (i & 6);
    auto put = [&](int slot, uint32_t u) { *reinterpret_cast<uint32_t*>(q + slot * plane) = u; };
    if (w.tc_three) {  // Xr hi, lo, Xi hi, lo, (Xr + Xi) hi, lo
      put(odd ? 1 : 0, rr);
      put(odd ? 3 : 2, ii);
      put(odd ? 5 : 4, __byte_perm(odd ? sother : sown, odd ? sown : sother, 0x5410));
    } else {  // Xr, Xi hi; Xr, Xi lo; -Xi, Xr hi; -Xi, Xr lo
      put(odd ? 2 : 0, rr);
      put(odd ? 3 : 1, ii);
      put(odd ? 6 : 4, ii ^ 0x80008000u);
      put(odd ? 7 : 5, rr);
    }
  }
}

__device__ __forceinline__ bool column_idle(const View& w, int b, int c, const int* skip) {
  return (skip && skip[b]) || w.done[b] || w.state[size_t(b) * w.m + c] != 0;
}

// x = 0, r = r~ = b, p = v = 0; |b|^2 and rho = (r~, r) accumulated.
__global__ void bicg_init_kernel(View w, const float2* __restrict__ M32, size_t stride, const int* skip) {
  const int b = blockIdx.y, c = blockIdx.z;
  if (skip && skip[b]) return;
  const float2* rhs = M32 + size_t(b) * stride + size_t(w.lda) * (w.n + c);
  float2 *x = w.v(kX, b, c), *r = w.v(kR, b, c), *rh = w.v(kRh, b, c), *p = w.v(kP, b, c), *v = w.v(kV, b, c);
  double b2 = 0.0;
  for (int k = 0; k < kVecRowsPerThread; ++k) {
    const int i = blockIdx.x * kVecRows + k * kVecThreads + threadIdx.x;
    if (i >= w.n) break;
    const float2 bi = rhs[i];
    x[i] = make_float2(0.f, 0.f);
    r[i] = bi;
    rh[i] = bi;
    p[i] = make_float2(0.f, 0.f);
    v[i] = make_float2(0.f, 0.f);
    b2 += double(bi.x) * bi.x + double(bi.y) * bi.y;
  }
  double* sc = w.s(b, c);
  // rho_new = (r~, r) = |b|^2 at the start
  block_accumulate(sc + kB2, b2, sc + kAcc1, b2, nullptr, 0.0);
}

// p = r + beta (p - omega v);  p^ = D p, which also goes to the product's operand
__global__ void bicg_p_kernel(View w, const float2* __restrict__ D, const int* skip) {
  const int b = w.matrix(), c = blockIdx.z;
  if (b < 0) return;
  if (column_idle(w, b, c, skip)) return;
  const double* sc = w.s(b, c);
  const double2 rho_new = make_double2(sc[kAcc1], sc[kAcc1 + 1]);
  const double2 rho = make_double2(sc[kRho], sc[kRho + 1]);
  const double2 alpha = make_double2(sc[kAlpha], sc[kAlpha + 1]);
  const double2 omega = make_double2(sc[kOmega], sc[kOmega + 1]);
  const double2 beta = cmul(cdiv(rho_new, rho), cdiv(alpha, omega));
  const float2 bf = make_float2(float(beta.x), float(beta.y)), of = make_float2(float(omega.x), float(omega.y));
  const float2 *r = w.v(kR, b, c), *v = w.v(kV, b, c);
  float2 *p = w.v(kP, b, c), *ph = w.v(kPh, b, c);
  const float2* Db = D ? D + size_t(b) * w.lda : nullptr;
  float2 xv[kVecRowsPerThread] = {};
#pragma unroll
  for (int k = 0; k < kVecRowsPerThread; ++k) {
    const int i = blockIdx.x * kVecRows + k * kVecThreads + threadIdx.x;
    if (i >= w.n) break;
    float2 pi = csub(p[i], cmul(of, v[i]));
    pi = cadd(r[i], cmul(bf, pi));
    p[i] = pi;
    const float2 x = Db ? cmul(Db[i], pi) : pi;
    ph[i] = x;
    xv[k] = x;
  }
  store_x_image(w, b, c, xv);
}

// Y = A X for the FP32 system matrices: 128 rows x 16 columns per CTA, each
// thread 4 rows (rg + 32 i) x 4 adjacent columns (read as two 16-byte
// shared loads), A streamed through shared memory in 16-column slabs by a
// three-stage cp.async pipeline (each A entry is read from HBM once per
// product; rows past n and columns past the slice are zero-filled by the
// copies; 55 KB per CTA, four CTAs per SM).  The columns of A are split into
// w.nsplit slices of kchunk (blockIdx.z = column group + groups * slice), so
// that even one running matrix spreads over the SMs: slice 0 writes Y, slice
// s > 0 its partial product, and the next dot kernel sums them in slice order.
constexpr int kMvRows = 128, kMvCols = 16, kMvK = 16, kMvThreads = 128, kMvStages = 3, kMvSliceCols = 512;
constexpr size_t kMvSmem = size_t(kMvStages) * kMvK * (kMvRows + kMvCols) * sizeof(float2);

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src, int bytes) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__global__ void __launch_bounds__(kMvThreads) bicg_matvec_kernel(View w, const float2* __restrict__ M32, size_t stride,
                                                                  int src, int dst, int groups, int kchunk,
                                                                  const int* skip) {
  const int b = w.matrix();
  if (b < 0 || (skip && skip[b]) || w.done[b]) return;
  extern __shared__ __align__(16) float2 mv_smem[];
  float2* As = mv_smem;                                       // [stage][kMvK][kMvRows]
  float2* Xs = mv_smem + size_t(kMvStages) * kMvK * kMvRows;  // [stage][kMvK][kMvCols]
  const int slice = blockIdx.z / groups;
  const int n = w.n, r0 = blockIdx.x * kMvRows, c0 = (blockIdx.z % groups) * kMvCols;
  const int kbeg = slice * kchunk, kend = min(n, kbeg + kchunk);
  const int slabs = (kend - kbeg + kMvK - 1) / kMvK;
  const float2* A = M32 + size_t(b) * stride;
  const int tid = threadIdx.x, rg = tid & 31, cq = tid >> 5;
  // one slab: kMvK columns of A (128 rows as 16-byte row pairs) and of X; a
  // slab past the slice's end commits an empty group (uniform group counts)
  auto load = [&](int slab) {
    if (slab < slabs) {
      const int k0 = kbeg + slab * kMvK, stage = slab % kMvStages;
      float2* as = As + size_t(stage) * kMvK * kMvRows;
      float2* xs = Xs + size_t(stage) * kMvK * kMvCols;
      for (int idx = tid; idx < kMvK * (kMvRows / 2); idx += kMvThreads) {
        const int rr = (idx % (kMvRows / 2)) * 2, kk = idx / (kMvRows / 2), row = r0 + rr;
        const bool in = k0 + kk < kend && row < n;
        const int bytes = in ? (row + 1 < n ? 16 : 8) : 0;
        cp_async16(as + size_t(kk) * kMvRows + rr, in ? A + size_t(row) + size_t(w.lda) * (k0 + kk) : A, bytes);
      }
      for (int idx = tid; idx < kMvK * kMvCols; idx += kMvThreads) {
        const int kk = idx % kMvK, cc = idx / kMvK;
        const bool in = k0 + kk < kend && c0 + cc < w.m;
        const float2* xsrc = in ? w.v(src, b, c0 + cc) + (k0 + kk) : A;
        cp_async8(xs + size_t(kk) * kMvCols + cc, xsrc, in ? 8 : 0);
      }
    }
    cp_async_commit();
  };
  float2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
  for (int sl = 0; sl < kMvStages - 1; ++sl) load(sl);
  for (int sl = 0; sl < slabs; ++sl) {
    cp_async_wait<kMvStages - 2>();  // slab sl has landed (this thread's copies)
    __syncthreads();                 // ... everyone's; and slab sl - 1's stage is free again
    load(sl + kMvStages - 1);
    const int stage = sl % kMvStages;
    const float2* as = As + size_t(stage) * kMvK * kMvRows;
    const float4* xs = reinterpret_cast<const float4*>(Xs + size_t(stage) * kMvK * kMvCols);
#pragma unroll
    for (int kk = 0; kk < kMvK; ++kk) {
      float2 a[4], x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = as[kk * kMvRows + rg + 32 * i];
      const float4 x01 = xs[(kk * kMvCols + 4 * cq) / 2], x23 = xs[(kk * kMvCols + 4 * cq) / 2 + 1];
      x[0] = make_float2(x01.x, x01.y);
      x[1] = make_float2(x01.z, x01.w);
      x[2] = make_float2(x23.x, x23.y);
      x[3] = make_float2(x23.z, x23.w);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) cfma(acc[i][j], a[i], x[j]);
    }
  }
  cp_async_wait<0>();  // no copy outlives the CTA (the trailing groups are empty)
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = c0 + 4 * cq + j;
    if (c >= w.m) continue;
    float2* y = slice == 0 ? w.v(dst, b, c) : w.pv(slice, b, c);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + rg + 32 * i;
      if (r < n) y[r] = acc[i][j];
    }
  }
}

// ---------------------------------------------------------------------------
// Tensor-core product (tcgen05, two FP16 terms a value): the same Y = A X with
// the complex products on the 5th-generation tensor cores.  Every real number
// is scaled by a power of two (one a row of A, from the row's largest entry;
// one a column and vector block of X, store_x_image) so that the largest lands
// in [2^14, 2^15), and taken as hi + lo, two FP16 values: 22 bits, as in a
// split into two TF32 values, for entries down to 2^-17 of the largest, an
// absolute error of 2^-40 of the largest below.  A CTA takes 128 rows and a
// slice of the columns, in slabs of 16 columns:
//   warp 5      bulk copies of X's operand, three or four slabs ahead;
//   warps 0-3   32 rows of A each, by cp.async as far ahead; a row a thread, 16
//               entries from shared memory, scaled and split into the four
//               real planes (re hi, re lo, im hi, im lo) in the K-major
//               32-byte-swizzled UMMA layout (two stages);
//   warp 4      one thread issues 4 MMAs a slab,
//     Ar hi x [Xr | Xi] hi, lo and Ai hi x [-Xi | Xr] hi, lo   (4N columns)
//     Ar lo x [Xr | Xi] hi     and Ai lo x [-Xi | Xr] hi       (2N columns)
//               into TMEM columns [Yr Yi | yr yi]; the second pair takes the
//               three small products, so that they do not disturb the FP32
//               accumulation of the large ones.
// Every 256 columns warps 0-3 take the accumulators, add the two parts, take
// the scales back and add to the row's sums in registers.  Every wait is
// bounded; a timeout sets *err (the solve then hands its matrices to the LU)
// and the CTA drains its copies and MMAs and frees its tensor memory before it
// returns.
// Bound by HBM (A is read once).  The form at n = 4112, 12 matrices, 16 columns
// (576 products and the vector kernels), on one set of inputs: 73.4 ms; with A
// in bulk copies of 1 KB, one a column of a slab, 81.5, bound by their issue
// (1.65 GB in 346 us under a profiler; another ring stage, twice the row warps
// or 1024-column slices changed nothing); FP16 terms with loads in registers
// and 256-column slices 92.8; split by the row's thread into two TF32 terms, 12
// MMAs a slab, 101.9.  Other inputs take other numbers of iterations (164 and
// 117.6 ms in another run); the quotient to the last form stays 1.38 to 1.40.
constexpr int kTcRows = 128, kTcK = 16, kTcThreads = 192, kTcStages = 2, kTcSub = 256;
constexpr long long kTcBicgPolls = 1LL << 26;  // poll budget of each wait (about 1 s is the other bound)
constexpr int kTcAPlane = kTcRows * 32;             // 4 KB: 128 rows of 16 FP16 values
constexpr int kTcRaw = kTcRows * kTcK * int(sizeof(float2));  // 16 KB of A as stored
static_assert(kVecRows % kTcSub == 0 && kBicgTcSliceCols % kTcSub == 0, "one scale of X per accumulation");

// k3M: the three-product form P1 = Ar Xr, P2 = Ai Xi, P3 = (Ar + Ai)(Xr + Xi),
// Yr = P1 - P2, Yi = P3 - P1 - P2 (six A planes, 6 MMAs of 2N or N columns,
// large and small accumulators of three products); otherwise the four products
// above.
template <int N, bool k3M = false> struct TcMv {
  static constexpr int kAPlanes = k3M ? 6 : 4;
  static constexpr int kA = kAPlanes * kTcAPlane;
  static constexpr int kBPlane = N * 32;
  static constexpr int kB = tc_x_slots(k3M) * kBPlane;
  static constexpr int kRing = kTcRaw + kB;
  static constexpr int kDepth = N == 16 && !k3M ? 4 : 3;  // two CTAs an SM but for the three products with N = 32
  static constexpr int kBars = 256;        // barriers, TMEM slot, abort flag
  static constexpr int kSmem = kDepth * kRing + kTcStages * kA + kBars + 256;
  // TMEM columns (a power of two >= 32): [Yr Yi | yr yi], or three of [P | p]
  static constexpr uint32_t kCols = k3M ? 8u * N : 4u * N;
};
// kind::f16, D = F32, A = B = FP16, both K-major, M = 128
__device__ __forceinline__ constexpr uint32_t tc_idesc(int n) {
  return (1u << 4) | (uint32_t(n >> 3) << 17) | (uint32_t(kTcRows >> 4) << 24);
}

__device__ __forceinline__ uint32_t tc_smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// start >> 4, LBO 1 (unused when swizzled), SBO = 8 rows x 32 B, version 1, 32-byte swizzle (layout 6)
__device__ __forceinline__ uint64_t tc_desc32(uint32_t saddr) {
  return uint64_t((saddr >> 4) & 0x3FFFu) | (uint64_t(1) << 16) | (uint64_t(256 >> 4) << 32) | (uint64_t(1) << 46) |
         (uint64_t(6) << 61);
}
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void tc_bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void tc_bar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// bytes (a multiple of 16) from global to shared memory, both 16-byte aligned; completes on `bar`
__device__ __forceinline__ void tc_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint64_t tc_now() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool tc_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// Bounded wait (poll budget, or 1 s); a timeout raises the CTA's abort flag and *err.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err,
                                        long long polls) {
  uint64_t t0 = 0;  // the clock is read only by a wait that is already long
  for (long long it = 0; it < polls; ++it) {
    if (tc_try(bar, parity)) return true;
    if ((it & 63) == 63) {
      if (*abort_flag) return false;
      const uint64_t t = tc_now();
      if (t0 == 0) t0 = t;
      if (t - t0 > 1000000000ull) break;
    }
  }
  *abort_flag = 1;
  atomicExch(err, 1);
  return false;
}
// Bounded wait of a warp or thread that is about to leave, for what it has started.
__device__ __forceinline__ void tc_drain(uint32_t bar, uint32_t parity, long long polls) {
  const uint64_t t0 = tc_now();
  for (long long it = 0; it < polls; ++it)
    if (tc_try(bar, parity) || ((it & 1023) == 1023 && tc_now() - t0 > 1000000000ull)) break;
}

// amax[b lda + r] = bits of row r's largest |component| over A's columns (zeroed before; grid z: column slices).  Once
// a batch of matrices, one read of A: 0.26 ms for 12 matrices of n = 4112, beside the products of some 300 iterations.
constexpr int kScaleCols = 512;
__global__ void __launch_bounds__(128) bicg_row_max_kernel(View w, const float2* __restrict__ M32, size_t stride,
                                                           const int* skip) {
  const int b = blockIdx.y, r = blockIdx.x * 128 + threadIdx.x;
  if ((skip && skip[b]) || r >= w.n) return;
  const int c0 = blockIdx.z * kScaleCols, c1 = min(w.n, c0 + kScaleCols);
  const float2* A = M32 + size_t(b) * stride + r;
  unsigned m = 0;
#pragma unroll 16
  for (int c = c0; c < c1; ++c) m = max(m, abs_bits(__ldcs(A + size_t(w.lda) * c)));
  atomicMax(w.amax + size_t(b) * w.lda + r, m);
}

template <int N, bool k3M>
__global__ void __launch_bounds__(kTcThreads, 2) bicg_tc_matvec_kernel(View w, const float2* __restrict__ M32,
                                                                     size_t stride, int dst, int kchunk,
                                                                     const int* skip, int* err, long long polls) {
  using L = TcMv<N, k3M>;
  constexpr int kMaxSubs = kBicgTcSliceCols / kTcSub;
  const int b = w.matrix();
  // decided once for the whole CTA (another CTA may raise the error flag meanwhile), before any tensor
  // memory is taken; a raised error skips the product
  __shared__ int go;
  __shared__ int xexp[kMaxSubs][N];  // the scale exponents of X's columns
  if (threadIdx.x == 0) go = !(b < 0 || (skip && skip[b]) || w.done[b] || *reinterpret_cast<volatile int*>(err));
  __syncthreads();
  if (!go) return;
  extern __shared__ uint8_t tsm[];
  const uint32_t raw = tc_smem_u32(tsm);
  const uint32_t sbase = (raw + 255u) & ~255u;  // the swizzle repeats after 256 bytes
  uint8_t* const gbase = tsm + (sbase - raw);  // [kTcStages] planes, [kTcRing] (A as stored, X operand)
  constexpr int kTcRing = L::kDepth, kRingBase = kTcStages * L::kA;
  uint8_t* const meta = gbase + kRingBase + kTcRing * L::kRing;
  // barriers: planes full[2] (4 warps) and empty[2] (commit); X full[] (copy) and empty[] (commit);
  // accumulators (commit); drain (commit)
  auto bar = [&](int i) { return tc_smem_u32(meta + 8 * i); };
  constexpr int kFull = 0, kEmpty = kTcStages, kRFull = 2 * kTcStages, kREmpty = kRFull + kTcRing,
                kAcc = kREmpty + kTcRing, kDrain = kAcc + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(meta + 192);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(meta + 196);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slice = blockIdx.z;
  const int n = w.n, r0 = blockIdx.x * kTcRows;
  const int kbeg = slice * kchunk, kend = min(n, kbeg + kchunk);
  const int slabs = (kend - kbeg + kTcK - 1) / kTcK;  // >= 1: slices start below n
  constexpr int kSubSlabs = kTcSub / kTcK;

  if (tid == 0) {
    for (int i = 0; i < kTcStages; ++i) {
      tc_bar_init(bar(kFull + i), 4);
      tc_bar_init(bar(kEmpty + i), 1);
    }
    for (int i = 0; i < kTcRing; ++i) {
      tc_bar_init(bar(kRFull + i), 1);
      tc_bar_init(bar(kREmpty + i), 1);
    }
    tc_bar_init(bar(kAcc), 1);
    tc_bar_init(bar(kDrain), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();  // the copies start beside the rest of the preparation
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tmem_slot)),
                 "r"(L::kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  uint32_t tmem = 0;
  if (warp < 5) {
    for (int i = tid; i < kMaxSubs * N; i += 160) {
      const int sub = i / N, c = i % N, k = kbeg + sub * kTcSub;
      xexp[sub][c] = c < w.m && k < kend ? w.xexp[(size_t(b) * w.m + c) * w.xblocks + k / kVecRows] : 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.sync 1, 160;" ::: "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tmem = *tmem_slot;
  }

  if (warp < 4) {
    // ---- operand warps: row r0 + tid of A ----
    const int row = r0 + tid;
    const bool row_ok = row < n;
    const int aexp = scale_exponent(row_ok ? w.amax[size_t(b) * w.lda + row] : 0u, tc_top(k3M));
    const float as = pow2(aexp);
    float2 y[N];
#pragma unroll
    for (int c = 0; c < N; ++c) y[c] = make_float2(0.f, 0.f);
    // a slab of the warp's 32 rows: lanes 0-15 the row pairs of its even columns, 16-31 of its odd ones; zeros past the
    // matrix's columns and rows.  Only this warp reads them.
    const int prow = r0 + warp * 32 + 2 * (lane & 15), pcol = lane >> 4;
    const float2* const ap = M32 + size_t(b) * stride + (prow < w.lda ? prow : 0);
    auto fetch = [&](int sl) {
      if (sl < slabs) {
        const int k0 = kbeg + sl * kTcK;
        float2* to = reinterpret_cast<float2*>(gbase + kRingBase + (sl % kTcRing) * L::kRing) + (prow - r0);
#pragma unroll
        for (int q = 0; q < kTcK / 2; ++q) {
          const int col = 2 * q + pcol;
          const bool in = k0 + col < kend && prow < w.lda;
          cp_async16(to + col * kTcRows, in ? ap + size_t(w.lda) * (k0 + col) : ap, in ? 16 : 0);
        }
      }
      cp_async_commit();
    };
#pragma unroll
    for (int sl = 0; sl < kTcRing - 1; ++sl) fetch(sl);
    bool ok = true;
    int rs = 0;  // ring stage
    for (int sl = 0; sl < slabs; ++sl) {
      const int st = sl & 1;
      fetch(sl + kTcRing - 1);  // into the stage that slab sl - 1 has left
      cp_async_wait<kTcRing - 1>();
      __syncwarp();
      ok = tc_wait(bar(kEmpty + st), uint32_t((sl >> 1) & 1) ^ 1u, abort_flag, err, polls);  // the MMAs of slab sl - 2
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        break;
      }
      const float2* ra = reinterpret_cast<const float2*>(gbase + kRingBase + rs * L::kRing) + tid;
      float2 v[kTcK];
#pragma unroll
      for (int kk = 0; kk < kTcK; ++kk) v[kk] = ra[kk * kTcRows];
      uint8_t* const sA = gbase + st * L::kA;
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        uint32_t q[L::kAPlanes][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 a0 = v[8 * ch + 2 * i], a1 = v[8 * ch + 2 * i + 1];
          const float r0s = a0.x * as, r1s = a1.x * as, i0s = a0.y * as, i1s = a1.y * as;
          tc_split(r0s, r1s, q[0][i], q[1][i]);
          tc_split(i0s, i1s, q[2][i], q[3][i]);
          if constexpr (k3M) tc_split(r0s + i0s, r1s + i1s, q[4][i], q[5][i]);  // Ar + Ai
        }
        const int off = tc_sw32(tid, ch);
#pragma unroll
        for (int pl = 0; pl < L::kAPlanes; ++pl)
          *reinterpret_cast<uint4*>(sA + pl * kTcAPlane + off) = make_uint4(q[pl][0], q[pl][1], q[pl][2], q[pl][3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the planes are read by the tensor cores
      __syncwarp();
      if (lane == 0) tc_bar_arrive(bar(kFull + st));
      if (++rs == kTcRing) rs = 0;
      if ((sl + 1) % kSubSlabs == 0 || sl + 1 == slabs) {
        // ---- the accumulators of these columns ----
        const int sub = sl / kSubSlabs;
        ok = tc_wait(bar(kAcc), uint32_t(sub & 1), abort_flag, err, polls);
        if (!__all_sync(0xffffffffu, ok)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tr = tmem + (uint32_t(warp * 32) << 16);
        auto ld8 = [](uint32_t addr, uint32_t (&o)[8]) {
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                       : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3]), "=r"(o[4]), "=r"(o[5]), "=r"(o[6]), "=r"(o[7])
                       : "r"(addr));
        };
#pragma unroll
        for (int cb = 0; cb < N / 8; ++cb) {
          // accumulator groups of N columns: Yr, Yi, yr, yi, or P1, p1, P2, p2, P3, p3
          constexpr int kGroups = k3M ? 6 : 4;
          uint32_t g[kGroups][8];
#pragma unroll
          for (int i = 0; i < kGroups; ++i) ld8(tr + uint32_t(i * N + cb * 8), g[i]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int c = cb * 8 + j;
            auto sum = [&](int hi, int lo) { return __uint_as_float(g[hi][j]) + __uint_as_float(g[lo][j]); };
            float2 out;
            if constexpr (k3M) {  // Yr = P1 - P2, Yi = P3 - P1 - P2
              const float p1 = sum(0, 1), p2 = sum(2, 3), p3 = sum(4, 5);
              out = make_float2(p1 - p2, p3 - p1 - p2);
            } else {
              out = make_float2(sum(0, 2), sum(1, 3));
            }
            const int e = -(aexp + xexp[sub][c]), e1 = e >> 1;
            const float f1 = pow2(e1), f2 = pow2(e - e1);
            y[c] = cadd(y[c], make_float2(out.x * f1 * f2, out.y * f1 * f2));
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");  // the next slab's MMAs overwrite them
      }
    }
    cp_async_wait<0>();  // no copy outlives the CTA
    if (ok && row_ok) {
#pragma unroll
      for (int c = 0; c < N; ++c)
        if (c < w.m) (slice == 0 ? w.v(dst, b, c) : w.pv(slice, b, c))[row] = y[c];
    }
  } else if (warp == 4 && lane == 0) {
    // ---- MMA issuer ----
    bool issued = false, ok = true;
    int rs = 0;
    uint32_t rph = 0;
    for (int sl = 0; sl < slabs; ++sl) {
      const int st = sl & 1;
      ok = tc_wait(bar(kRFull + rs), rph, abort_flag, err, polls) &&                          // the slab of X
           tc_wait(bar(kFull + st), uint32_t((sl >> 1) & 1), abort_flag, err, polls);  // the planes
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sA = sbase + uint32_t(st * L::kA), sB = sbase + uint32_t(kRingBase + rs * L::kRing + kTcRaw);
      auto ad = [&](int pl) { return tc_desc32(sA + uint32_t(pl * kTcAPlane)); };
      auto bd = [&](int pl) { return tc_desc32(sB + uint32_t(pl * L::kBPlane)); };
      const uint32_t a0 = sl % kSubSlabs == 0 ? 0u : 1u;
      if constexpr (k3M) {
#pragma unroll
        for (int p = 0; p < 3; ++p) {  // [P | p] += hi [hi | lo], p += lo hi
          const uint32_t t = tmem + uint32_t(2 * N * p);
          tc_mma(t, ad(2 * p), bd(2 * p), tc_idesc(2 * N), a0);
          tc_mma(t + uint32_t(N), ad(2 * p + 1), bd(2 * p), tc_idesc(N), 1u);
        }
      } else {
        tc_mma(tmem, ad(0), bd(0), tc_idesc(4 * N), a0);
        tc_mma(tmem, ad(2), bd(4), tc_idesc(4 * N), 1u);
        tc_mma(tmem + uint32_t(2 * N), ad(1), bd(0), tc_idesc(2 * N), 1u);
        tc_mma(tmem + uint32_t(2 * N), ad(3), bd(4), tc_idesc(2 * N), 1u);
      }
      issued = true;
      tc_commit(bar(kEmpty + st));   // the planes and
      tc_commit(bar(kREmpty + rs));  // the ring stage are free once these MMAs have read them
      if ((sl + 1) % kSubSlabs == 0 || sl + 1 == slabs) tc_commit(bar(kAcc));
      if (++rs == kTcRing) {
        rs = 0;
        rph ^= 1u;
      }
    }
    if (issued) {
      // every MMA of this CTA has completed before the tensor memory is freed
      tc_commit(bar(kDrain));
      tc_drain(bar(kDrain), 0u, polls);
    }
  } else if (warp == 5) {
    // ---- copies of X's operand ----
    const uint8_t* X = w.image + (size_t(b) * ((n + kTcK - 1) / kTcK) + kbeg / kTcK) * L::kB;
    int rs = 0, sl = 0;
    uint32_t rph = 0;
    for (; sl < slabs && lane == 0; ++sl) {
      if (!tc_wait(bar(kREmpty + rs), rph ^ 1u, abort_flag, err, polls)) break;
      tc_bar_expect(bar(kRFull + rs), uint32_t(L::kB));
      tc_bulk(sbase + uint32_t(kRingBase + rs * L::kRing + kTcRaw), X + size_t(sl) * L::kB, uint32_t(L::kB),
              bar(kRFull + rs));
      if (++rs == kTcRing) {
        rs = 0;
        rph ^= 1u;
      }
    }
    // no copy outlives the CTA: the last ones started
    if (lane == 0)
      for (int q = max(0, sl - kTcRing); q < sl; ++q) tc_drain(bar(kRFull + q % kTcRing), uint32_t((q / kTcRing) & 1), polls);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 4) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::kCols));
}

// acc2 += (r~, v)
__global__ void bicg_dot_rv_kernel(View w, const int* skip) {
  const int b = w.matrix(), c = blockIdx.z;
  if (b < 0) return;
  if (column_idle(w, b, c, skip)) return;
  const float2* rh = w.v(kRh, b, c);
  float2* v = w.v(kV, b, c);
  double2 acc = make_double2(0.0, 0.0);
  for (int k = 0; k < kVecRowsPerThread; ++k) {
    const int i = blockIdx.x * kVecRows + k * kVecThreads + threadIdx.x;
    if (i >= w.n) break;
    acc = cdot_acc(acc, rh[i], w.gather(v, b, c, i));
  }
  double* sc = w.s(b, c);
  block_accumulate(sc + kAcc2, acc.x, sc + kAcc2 + 1, acc.y, nullptr, 0.0);
}

__device__ __forceinline__ bool czero(double2 z) { return z.x == 0.0 && z.y == 0.0; }

// alpha = rho_new / (r~, v); rho = rho_new.  One thread per (matrix, column).
__global__ void bicg_alpha_kernel(View w, const int* skip) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= w.batch * w.m) return;
  const int b = idx / w.m, c = idx % w.m;
  if (column_idle(w, b, c, skip)) return;
  double* sc = w.s(b, c);
  if (sc[kB2] == 0.0) {  // b = 0: x = 0 is exact
    w.state[idx] = 1;
    return;
  }
  const double2 rho_new = make_double2(sc[kAcc1], sc[kAcc1 + 1]);
  const double2 rv = make_double2(sc[kAcc2], sc[kAcc2 + 1]);
  sc[kAcc1] = sc[kAcc1 + 1] = sc[kAcc2] = sc[kAcc2 + 1] = 0.0;
  if (czero(rho_new) || czero(rv) || !isfinite(rv.x) || !isfinite(rv.y)) {
    w.state[idx] = 2;
    return;
  }
  const double2 alpha = cdiv(rho_new, rv);
  sc[kAlpha] = alpha.x;
  sc[kAlpha + 1] = alpha.y;
  sc[kRho] = rho_new.x;
  sc[kRho + 1] = rho_new.y;
}

// dst = Bblk src for every running column: the block-diagonal preconditioner,
// one C x C block per atom (Bblk[(b N + atom) C^2 + q C + q']), one thread
// per row.
__global__ void bicg_block_apply_kernel(View w, int src, int dst, const float2* __restrict__ Bblk,
                                        const int* __restrict__ state_atom, const int* __restrict__ atom_off, int N,
                                        int C, const int* skip) {
  const int b = w.matrix(), c = blockIdx.z;
  if (b < 0) return;
  if (column_idle(w, b, c, skip)) return;
  const float2* in = w.v(src, b, c);
  float2* out = w.v(dst, b, c);
  float2 xv[kVecRowsPerThread] = {};
#pragma unroll
  for (int k = 0; k < kVecRowsPerThread; ++k) {
    const int i = blockIdx.x * kVecRows + k * kVecThreads + threadIdx.x;
    if (i >= w.n) break;
    const int a = state_atom[i], s0 = atom_off[a], cnt = atom_off[a + 1] - s0, q = i - s0;
    const float2* row = Bblk + ((size_t(b) * N + a) * C + q) * C;
    float2 acc = make_float2(0.f, 0.f);
    for (int q2 = 0; q2 < cnt; ++q2) cfma(acc, row[q2], in[s0 + q2]);
    out[i] = acc;
    xv[k] = acc;
  }
  store_x_image(w, b, c, xv);
}

// s = r - alpha v (in r);  s^ = D s, which also goes to the product's operand
__global__ void bicg_s_kernel(View w, const float2* __restrict__ D, const int* skip) {
  const int b = w.matrix(), c = blockIdx.z;
  if (b < 0) return;
  if (column_idle(w, b, c, skip)) return;
  const double* sc = w.s(b, c);
  const float2 af = make_float2(float(sc[kAlpha]), float(sc[kAlpha + 1]));
  float2 *r = w.v(kR, b, c), *sh = w.v(kSh, b, c);
  const float2* v = w.v(kV, b, c);
  const float2* Db = D ? D + size_t(b) * w.lda : nullptr;
  float2 xv[kVecRowsPerThread] = {};
#pragma unroll
  for (int k = 0; k < kVecRowsPerThread; ++k) {
    const int i = blockIdx.x * kVecRows + k * kVecThreads + threadIdx.x;
    if (i >= w.n) break;
    const float2 si = csub(r[i], cmul(af, v[i]));
    r[i] = si;
    const float2 x = Db ? cmul(Db[i], si) : si;
    sh[i] = x;
    xv[k] = x;
  }
  store_x_image(w, b, c, xv);
}

// acc2 += (t, s), acc3 += |t|^2
__global__ void bicg_dot_ts_kernel(View w, const int* skip) {
  const int b = w.matrix(), c = blockIdx.z;
  if (b < 0) return;
  if (column_idle(w, b, c, skip)) return;
  float2* t = w.v(kT, b, c);
  const float2* sv = w.v(kR, b, c);
  double2 ts = make_double2(0.0, 0.0);
  double tt = 0.0;
  for (int k = 0; k < kVecRowsPerThread; ++k) {
    const int i = blockIdx.x * kVecRows + k * kVecThreads + threadIdx.x;
    if (i >= w.n) break;
    const float2 ti = w.gather(t, b, c, i);
    ts = cdot_acc(ts, ti, sv[i]);
    tt += double(ti.x) * ti.x + double(ti.y) * ti.y;
  }
  double* sc = w.s(b, c);
  block_accumulate(sc + kAcc2, ts.x, sc + kAcc2 + 1, ts.y, sc + kAcc3, tt);
}

// omega = (t, s) / (t, t)
__global__ void bicg_omega_kernel(View w, const int* skip) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= w.batch * w.m) return;
  const int b = idx / w.m, c = idx % w.m;
  if (column_idle(w, b, c, skip)) return;
  double* sc = w.s(b, c);
  const double2 ts = make_double2(sc[kAcc2], sc[kAcc2 + 1]);
  const double tt = sc[kAcc3];
  sc[kAcc2] = sc[kAcc2 + 1] = sc[kAcc3] = 0.0;
  if (!(tt > 0.0) || czero(ts) || !isfinite(ts.x) || !isfinite(ts.y)) {
    w.state[idx] = 2;
    return;
  }
  sc[kOmega] = ts.x / tt;
  sc[kOmega + 1] = ts.y / tt;
}

// x += alpha p^ + omega s^;  r = s - omega t;  acc4 += |r|^2, acc1 += (r~, r)
__global__ void bicg_xr_kernel(View w, const int* skip) {
  const int b = w.matrix(), c = blockIdx.z;
  if (b < 0) return;
  if (column_idle(w, b, c, skip)) return;
  const double* sc = w.s(b, c);
  const float2 af = make_float2(float(sc[kAlpha]), float(sc[kAlpha + 1]));
  const float2 of = make_float2(float(sc[kOmega]), float(sc[kOmega + 1]));
  float2 *x = w.v(kX, b, c), *r = w.v(kR, b, c);
  const float2 *ph = w.v(kPh, b, c), *sh = w.v(kSh, b, c), *t = w.v(kT, b, c), *rh = w.v(kRh, b, c);
  double rr = 0.0;
  double2 rho = make_double2(0.0, 0.0);
  for (int k = 0; k < kVecRowsPerThread; ++k) {
    const int i = blockIdx.x * kVecRows + k * kVecThreads + threadIdx.x;
    if (i >= w.n) break;
    x[i] = cadd(x[i], cadd(cmul(af, ph[i]), cmul(of, sh[i])));
    const float2 ri = csub(r[i], cmul(of, t[i]));
    r[i] = ri;
    rr += double(ri.x) * ri.x + double(ri.y) * ri.y;
    rho = cdot_acc(rho, rh[i], ri);
  }
  double* s2 = w.s(b, c);
  block_accumulate(s2 + kAcc4, rr, s2 + kAcc1, rho.x, s2 + kAcc1 + 1, rho.y);
}

// Convergence per column; per matrix done flag and iteration count; the
// number of running matrices for the host poll.
__global__ void bicg_check_kernel(View w, double tol2, int iter, int* iters, int* active, const int* skip) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= w.batch) return;
  if ((skip && skip[b]) || w.done[b]) return;
  bool all = true;
  for (int c = 0; c < w.m; ++c) {
    int& st = w.state[size_t(b) * w.m + c];
    double* sc = w.s(b, c);
    if (st == 0) {
      const double rr = sc[kAcc4];
      if (!isfinite(rr)) st = 2;
      else if (rr <= tol2 * sc[kB2]) st = 1;
    }
    sc[kAcc4] = 0.0;
    all = all && st != 0;
  }
  iters[b] = iter;
  if (all) w.done[b] = 1;
  else atomicAdd(active, 1);
}

// The compacted list of running matrices (one block, batch <= kCompactMax):
// act[0..count) the running ones in order, -1 after.
constexpr int kCompactMax = 1024;
__device__ __forceinline__ void compact_running(bool alive, int b, int batch, int* act) {
  __shared__ int warp_total[kCompactMax / 32];
  const unsigned bal = __ballot_sync(0xffffffffu, alive);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) warp_total[wid] = __popc(bal);
  __syncthreads();
  int base = 0, total = 0;
  for (int i = 0; i < int(blockDim.x >> 5); ++i) {
    if (i < wid) base += warp_total[i];
    total += warp_total[i];
  }
  if (alive) act[base + __popc(bal & ((1u << lane) - 1u))] = b;
  if (b >= total && b < batch) act[b] = -1;  // disjoint from the positions below total
}

__global__ void bicg_act_init_kernel(int batch, const int* skip, int* act) {
  const int b = threadIdx.x;
  compact_running(b < batch && !(skip && skip[b]), b, batch, act);
}

// bicg_check_kernel for one block over the whole batch, which also rebuilds
// the compacted list of running matrices for the next iteration's launches.
__global__ void bicg_check_compact_kernel(View w, double tol2, int iter, int* iters, int* active, const int* skip,
                                          int* act) {
  const int b = threadIdx.x;
  bool alive = false;
  if (b < w.batch && !(skip && skip[b]) && !w.done[b]) {
    bool all = true;
    for (int c = 0; c < w.m; ++c) {
      int& st = w.state[size_t(b) * w.m + c];
      double* sc = w.s(b, c);
      if (st == 0) {
        const double rr = sc[kAcc4];
        if (!isfinite(rr)) st = 2;
        else if (rr <= tol2 * sc[kB2]) st = 1;
      }
      sc[kAcc4] = 0.0;
      all = all && st != 0;
    }
    iters[b] = iter;
    if (all) {
      w.done[b] = 1;
    } else {
      alive = true;
      atomicAdd(active, 1);
    }
  }
  compact_running(alive, b, w.batch, act);
}

// Solution X -> RHS columns of M32; failed[b] = 2 when a column did not converge.
__global__ void bicg_finish_kernel(View w, float2* __restrict__ M32, size_t stride, int* failed, const int* skip,
                                   const int* tc_err) {
  const int b = blockIdx.y, c = blockIdx.z;
  if (skip && skip[b]) return;
  const float2* x = w.v(kX, b, c);
  float2* out = M32 + size_t(b) * stride + size_t(w.lda) * (w.n + c);
  for (int k = 0; k < kVecRowsPerThread; ++k) {
    const int i = blockIdx.x * kVecRows + k * kVecThreads + threadIdx.x;
    if (i >= w.n) break;
    out[i] = x[i];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && (w.state[size_t(b) * w.m + c] != 1 || (tc_err && *tc_err))) failed[b] = 2;
}

}  // namespace

int bicg_slices(int n, bool tensor, int* chunk) {
  int c = tensor ? kBicgTcSliceCols
                 : std::max(kMvSliceCols, ((n + kBicgMaxSplit - 1) / kBicgMaxSplit + kMvK - 1) / kMvK * kMvK);
  c = std::min(c, std::max(n, 1));
  if (chunk) *chunk = c;
  return (n + c - 1) / c;
}

size_t bicg_image_bytes(int n, int m, int batch) {
  return m > 32 ? 0 : size_t(batch) * size_t((n + kTcK - 1) / kTcK) * tc_x_slots(false) * (m <= 16 ? 16 : 32) * 32;
}
size_t bicg_exponents(int n, int m, int batch) { return size_t(batch) * m * size_t((n + kVecRows - 1) / kVecRows); }

cudaError_t bicg_row_scales(const BatchLayout& lay, int batch, const float2* M32, const BicgWork& w, const int* skip,
                            cudaStream_t s) {
  if (!w.tensor || !w.tc_err || lay.m > 32) return cudaSuccess;
  View v{lay.n, lay.m, lay.lda, batch, w.vec, w.sc, w.state, w.done, w.part, 1};
  v.amax = w.amax;
  cudaMemsetAsync(w.amax, 0, size_t(batch) * lay.lda * sizeof(unsigned), s);
  count_launch();
  const dim3 grid(unsigned((lay.n + 127) / 128), unsigned(batch), unsigned((lay.n + kScaleCols - 1) / kScaleCols));
  bicg_row_max_kernel<<<grid, 128, 0, s>>>(v, M32, lay.stride, skip);
  return cudaGetLastError();
}

cudaError_t bicgstab_solve(const BatchLayout& lay, int batch, float2* M32, const float2* D, const BlockPrecond* blk,
                           const BicgWork& w, double tol, int max_iter, int poll, const int* skip, int* failed,
                           cudaStream_t s) {
  View v{lay.n, lay.m, lay.lda, batch, w.vec, w.sc, w.state, w.done, w.part, 1};
  const dim3 vgrid(unsigned((lay.n + kVecRows - 1) / kVecRows), unsigned(batch), unsigned(lay.m));
  const int row_blocks = (lay.n + kMvRows - 1) / kMvRows, groups = (lay.m + kMvCols - 1) / kMvCols;
  {
    const cudaError_t e = cudaFuncSetAttribute(bicg_matvec_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(kMvSmem));
    if (e != cudaSuccess) return e;
  }
  // the tensor-core product for up to 32 right-hand sides (N = 16 or 32 accumulator columns)
  const bool tensor = w.tensor && w.tc_err && lay.m <= 32 && (w.part || lay.n <= kBicgTcSliceCols);
  const bool n16 = lay.m <= 16, three = w.tensor == 2;
  if (tensor) {
    v.amax = w.amax;
    v.xexp = w.xexp;
    v.image = w.image;
    v.xblocks = (lay.n + kVecRows - 1) / kVecRows;
    v.tc_n = n16 ? 16 : 32;
    v.tc_three = three;
  }
  // the four instantiations: N = 16 / 32 accumulator columns, four or three products
  auto tc_launch = [&](auto kN, auto k3, const dim3& grid, const View& view, int dst, int chunk) {
    constexpr int N = decltype(kN)::value;
    constexpr bool M3 = decltype(k3)::value;
    bicg_tc_matvec_kernel<N, M3><<<grid, kTcThreads, TcMv<N, M3>::kSmem, s>>>(view, M32, lay.stride, dst, chunk, skip,
                                                                              w.tc_err, kTcBicgPolls);
  };
  auto tc_attr = [&](auto kN, auto k3) {
    constexpr int N = decltype(kN)::value;
    constexpr bool M3 = decltype(k3)::value;
    return cudaFuncSetAttribute(bicg_tc_matvec_kernel<N, M3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                TcMv<N, M3>::kSmem);
  };
  using I16 = std::integral_constant<int, 16>;
  using I32 = std::integral_constant<int, 32>;
  using T3 = std::true_type;
  using T4 = std::false_type;
  if (tensor) {
    const cudaError_t e = n16 ? (three ? tc_attr(I16{}, T3{}) : tc_attr(I16{}, T4{}))
                              : (three ? tc_attr(I32{}, T3{}) : tc_attr(I32{}, T4{}));
    if (e != cudaSuccess) return e;
    cudaMemsetAsync(w.tc_err, 0, sizeof(int), s);
  }
  const unsigned tc_row_blocks = unsigned((lay.n + kTcRows - 1) / kTcRows);
  // Slices of A's columns (bicg_slices): the last running matrices still fill
  // the GPU with product CTAs.  The slicing depends on n (and the product's
  // kind) alone: a matrix's arithmetic does not depend on which others share
  // its batch.
  int chunk = lay.n, nsplit = 1;
  if (w.part) nsplit = bicg_slices(lay.n, tensor, &chunk);
  const int sthreads = 128, sblocks = (batch * lay.m + sthreads - 1) / sthreads;
  const int bblocks = (batch + sthreads - 1) / sthreads;
  cudaMemsetAsync(w.sc, 0, size_t(batch) * lay.m * kBicgScalars * sizeof(double), s);
  cudaMemsetAsync(w.state, 0, size_t(batch) * lay.m * sizeof(int), s);
  cudaMemsetAsync(w.done, 0, size_t(batch) * sizeof(int), s);
  cudaMemsetAsync(w.iters, 0, size_t(batch) * sizeof(int), s);
  // rho = alpha = omega = 1 (the first p = r)
  {
    std::vector<double> init(size_t(batch) * lay.m * kBicgScalars, 0.0);
    for (size_t i = 0; i < size_t(batch) * lay.m; ++i) {
      init[i * kBicgScalars + kRho] = 1.0;
      init[i * kBicgScalars + kAlpha] = 1.0;
      init[i * kBicgScalars + kOmega] = 1.0;
    }
    cudaMemcpyAsync(w.sc, init.data(), init.size() * sizeof(double), cudaMemcpyHostToDevice, s);
    count_launch();
    bicg_init_kernel<<<vgrid, kVecThreads, 0, s>>>(v, M32, lay.stride, skip);
    // the host vector must outlive the copy
    cudaStreamSynchronize(s);
  }
  // The iteration's launches cover only the running matrices: the check
  // kernel keeps a compacted list of them, and the grids are sized by the
  // count of the last host poll (an upper bound: matrices only finish).
  const bool compact = w.act && batch <= kCompactMax;
  const unsigned cthreads = unsigned((batch + 31) / 32 * 32);
  if (compact) {
    count_launch();
    bicg_act_init_kernel<<<1, cthreads, 0, s>>>(batch, skip, w.act);
  }
  View vr = v;  // the view of the iteration's launches
  vr.act = compact ? w.act : nullptr;
  // dst = A src over the running matrices: V = A P^ or T = A S^ (the tensor-core product's operand is w.image, written
  // with src)
  auto product = [&](unsigned rows_y, int src, int dst) {
    count_launch();
    if (tensor) {
      const dim3 tgrid(tc_row_blocks, rows_y, unsigned(nsplit));
      if (n16) {
        if (three) tc_launch(I16{}, T3{}, tgrid, vr, dst, chunk);
        else tc_launch(I16{}, T4{}, tgrid, vr, dst, chunk);
      } else {
        if (three) tc_launch(I32{}, T3{}, tgrid, vr, dst, chunk);
        else tc_launch(I32{}, T4{}, tgrid, vr, dst, chunk);
      }
    } else {
      const dim3 mgrid(unsigned(row_blocks), rows_y, unsigned(groups * nsplit));
      bicg_matvec_kernel<<<mgrid, kMvThreads, kMvSmem, s>>>(vr, M32, lay.stride, src, dst, groups, chunk, skip);
    }
  };
  int running = batch;
  for (int it = 1; it <= max_iter && running > 0; ++it) {
    vr.nsplit = nsplit;  // the dot kernels sum the slices
    const unsigned rows_y = unsigned(compact ? running : batch);
    const dim3 rgrid(vgrid.x, rows_y, vgrid.z);
    View vec = vr;
    if (blk) vec.image = nullptr;  // bicg_block_apply_kernel writes the operand
    count_launch();
    bicg_p_kernel<<<rgrid, kVecThreads, 0, s>>>(vec, blk ? nullptr : D, skip);
    if (blk) {
      count_launch();
      bicg_block_apply_kernel<<<rgrid, kVecThreads, 0, s>>>(vr, kP, kPh, blk->B, blk->state_atom, blk->atom_off,
                                                            blk->N, blk->C, skip);
    }
    product(rows_y, kPh, kV);
    count_launch();
    bicg_dot_rv_kernel<<<rgrid, kVecThreads, 0, s>>>(vr, skip);
    count_launch();
    bicg_alpha_kernel<<<sblocks, sthreads, 0, s>>>(v, skip);
    count_launch();
    bicg_s_kernel<<<rgrid, kVecThreads, 0, s>>>(vec, blk ? nullptr : D, skip);
    if (blk) {
      count_launch();
      bicg_block_apply_kernel<<<rgrid, kVecThreads, 0, s>>>(vr, kR, kSh, blk->B, blk->state_atom, blk->atom_off,
                                                            blk->N, blk->C, skip);
    }
    product(rows_y, kSh, kT);
    count_launch();
    bicg_dot_ts_kernel<<<rgrid, kVecThreads, 0, s>>>(vr, skip);
    count_launch();
    bicg_omega_kernel<<<sblocks, sthreads, 0, s>>>(v, skip);
    count_launch();
    bicg_xr_kernel<<<rgrid, kVecThreads, 0, s>>>(vr, skip);
    const bool poll_now = (it % std::max(poll, 1)) == 0 || it == max_iter;
    if (poll_now) cudaMemsetAsync(w.active, 0, sizeof(int), s);
    count_launch();
    if (compact)
      bicg_check_compact_kernel<<<1, cthreads, 0, s>>>(v, tol * tol, it, w.iters, w.active, skip, w.act);
    else
      bicg_check_kernel<<<bblocks, sthreads, 0, s>>>(v, tol * tol, it, w.iters, w.active, skip);
    if (poll_now) {
      cudaError_t e = cudaMemcpyAsync(&running, w.active, sizeof(int), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return e;
    }
  }
  count_launch();
  bicg_finish_kernel<<<vgrid, kVecThreads, 0, s>>>(v, M32, lay.stride, failed, skip, tensor ? w.tc_err : nullptr);
  return cudaGetLastError();
}

}  // namespace rfx
