// Split-precision complex GEMM on the int8 tensor cores (tcgen05.mma
// kind::i8), used by the BSE in its split mode and exported as a batched
// ZGEMM.  No counterpart in the reference (its BSE runs FP64 ZGEMMs,
// SRC/parquet_BSE.f90:72-128).
//
// Error-free splitting after Ozaki, Ogita, Oishi & Rump (Numer. Algorithms
// 59, 2012), with integer slices:
//   C = A B (complex, M x K times K x N) is the real product C' = A' B' with
//   A' = [Re A | Im A] (M x 2K) and B' whose column 2j is [Re B_j ; -Im B_j]
//   and column 2j+1 is [Im B_j ; Re B_j].  Every row of A' is scaled by 2^-e
//   (max |row| < 2^e) and cut into s int8 slices of 7 bits; every column of
//   B' likewise.  Slice products with i + j = d < s are summed exactly in
//   int32 on the tensor cores (|sum| <= s K' 127^2 < 2^31) and combined in
//   FP64: C' = 2^(e+f) sum_d 2^(-7(d+2)) D_d.
//
// Layout: slices of A' as rows of Kpad bytes (K-major), slices of B' as rows
// of Kpad bytes (one row per column of B'); Kpad = 2K rounded up to 128.
// The GEMM kernel reads 128-byte K chunks of both with TMA (128-byte
// swizzle), accumulates two diagonals at a time in TMEM (four buffers, so the
// FP64 drain of two diagonals overlaps the MMAs of the next two), and folds
// each diagonal into FP64 sums in registers; after the last one the scales and
// the caller's epilogue are applied.
#include <cuda.h>

#include <algorithm>
#include <cstdio>
#include <atomic>
#include <cstring>

#include "tups_device.cuh"

namespace tups {

constexpr int OZ_BM = 128;       // rows per tile (TMEM lanes)
constexpr int OZ_BK = 128;       // K bytes per pipeline stage
constexpr int OZ_STAGES = 7;     // 7 x (16 KB of A + <= 16 KB of B) in flight
constexpr uint32_t OZ_STAGE_BYTES = 2 * OZ_BM * OZ_BK;
constexpr int OZ_SLICE_BITS = 7;

// ---- splitting ---------------------------------------------------------------
// Operand: line = [X1 | X2] for rows of A, [Y1 ; Y2] for columns of B;
// part 2 may be absent (K2 = 0).  Instance b of a batch uses X1 + b*s1,
// X2 + b*s2, or, in BSE mode, the (q, r) vertex of the chunk.
__device__ __forceinline__ const cplx* oz_part(const OzOperand& o, int part, int inst) {
  const bool bse = part == 1 ? o.bse1 : o.bse2;
  if (bse) {
    const int q = o.q_begin + inst / 4, r = inst % 4;
    // constant indices keep the parameter struct out of local memory
    const cplx* Fr = r == 0 ? o.F[0] : r == 1 ? o.F[1] : r == 2 ? o.F[2] : o.F[3];
    return Fr + (size_t)o.Nz * o.Nz * q;
  }
  return part == 1 ? o.p1 + (size_t)o.s1 * inst : o.p2 + (size_t)o.s2 * inst;
}

// Per-instance view of an operand
struct OzLine {
  const cplx* p1;
  const cplx* p2;
  int ld1, ld2, K1;
};

__device__ __forceinline__ OzLine oz_view(const OzOperand& o, int inst) {
  OzLine v;
  v.ld1 = o.ld1;
  v.ld2 = o.ld2;
  v.K1 = o.K1;
  v.p1 = oz_part(o, 1, inst);
  v.p2 = o.K2 ? oz_part(o, 2, inst) : nullptr;
  return v;
}

// element (m, k) of a row operand (parts)
__device__ __forceinline__ const cplx& oz_a(const OzLine& v, int m, int k) {
  return k < v.K1 ? v.p1[m + (size_t)v.ld1 * k] : v.p2[m + (size_t)v.ld2 * (k - v.K1)];
}

// element (k, j) of a column operand (parts)
__device__ __forceinline__ const cplx& oz_b(const OzLine& v, int k, int j) {
  return k < v.K1 ? v.p1[k + (size_t)v.ld1 * j] : v.p2[(k - v.K1) + (size_t)v.ld2 * j];
}

__device__ __forceinline__ int oz_exponent(double maxabs) {
  int e = 0;
  if (maxabs > 0.0) frexp(maxabs, &e);
  return e;
}

// max(mx, |v.x|, |v.y|) that ignores NaN
__device__ __forceinline__ double oz_absmax(double mx, cplx v) {
  mx = fabs(v.x) > mx ? fabs(v.x) : mx;
  return fabs(v.y) > mx ? fabs(v.y) : mx;
}

// The s int8 slices of v 2^-e (|v 2^-e| < 1) are the base-128 digits, most
// significant first and carrying the sign of v, of t = trunc(|v| 2^(7s - e)):
// the same bytes as the repeated a = trunc(128 r), r = 128 r - a of the
// error-free splitting (all steps exact in FP64), with
// one scaling and one conversion instead of 4 s FP64 operations.  t <
// 2^(7s) <= 2^56, so t is an exact int64.  2^(7s - e) is the product of two
// normal doubles (e >= -1073: one of them is 1 except for lines below 2^-960).
struct OzScale {
  double f1, f2;
};
__device__ __forceinline__ OzScale oz_scale(int e, int s) {
  const int k = OZ_SLICE_BITS * s - e, k1 = min(k, 1023);
  return {__hiloint2double((k1 + 1023) << 20, 0), __hiloint2double((k - k1 + 1023) << 20, 0)};
}
// digit j (0 = least significant) of v in byte j & 3 of lo (j < 4) or hi: the
// 7-bit groups of t spread to bytes, then, for v < 0, each negated as
// (128 - d) ^ 128, which borrows from no neighbour.
__device__ __forceinline__ void oz_digits(double v, const OzScale& sc, uint32_t& lo, uint32_t& hi) {
  const unsigned long long u = (unsigned long long)__double2ll_rz(fabs(v) * sc.f1 * sc.f2);
  auto spread = [](uint32_t x) {  // 28 bits -> 4 bytes of 7
    x += 3u * (x & 0xfffc000u);
    return x + (x & 0x3f803f80u);
  };
  const int neg = __double2hiint(v) >> 31;
  const uint32_t bias = (uint32_t)neg & 0x80808080u, sg = (uint32_t)neg | 1u;
  lo = (spread((uint32_t)u & 0xfffffffu) * sg + bias) ^ bias;
  hi = (spread((uint32_t)(u >> 28) & 0xfffffffu) * sg + bias) ^ bias;
}
// bytes (column c, digit j) of four columns -> word j holds digit j of the four
__device__ __forceinline__ void oz_transpose4(uint32_t& w0, uint32_t& w1, uint32_t& w2, uint32_t& w3) {
  const uint32_t t0 = __byte_perm(w0, w1, 0x5140), t1 = __byte_perm(w2, w3, 0x5140);
  const uint32_t t2 = __byte_perm(w0, w1, 0x7362), t3 = __byte_perm(w2, w3, 0x7362);
  w0 = __byte_perm(t0, t1, 0x5410);
  w1 = __byte_perm(t0, t1, 0x7632);
  w2 = __byte_perm(t2, t3, 0x5410);
  w3 = __byte_perm(t2, t3, 0x7632);
}

__device__ __forceinline__ void oz_cp_async16(void* sdst, const void* gsrc, bool valid) {
  const unsigned sz = valid ? 16u : 0u;
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gsrc), "r"(sz));
}

constexpr size_t kOzLinesSmem = 74 * 1024;  // a CTA's whole rows or columns: three CTAs per SM

// the slices of row entries k .. k + 7 (at(c): entry k + c; beyond Kc unused):
// one 8-byte run per slice and part
template <class At>
__device__ __forceinline__ void oz_row_slices(At at, const OzScale& sc, int k, int Kc, int s, size_t slice_stride,
                                              int8_t* row) {
  double im[8];
  uint32_t lo[8], hi[8];
#pragma unroll
  for (int part = 0; part < 2; part++) {
#pragma unroll
    for (int c = 0; c < 8; c++) {
      double v;
      if (part == 0) {
        const cplx x = at(c);
        v = x.x;
        im[c] = x.y;
      } else {
        v = im[c];
      }
      oz_digits(v, sc, lo[c], hi[c]);
    }
#pragma unroll
    for (int c = 0; c < 8; c += 4) {
      oz_transpose4(lo[c], lo[c + 1], lo[c + 2], lo[c + 3]);
      oz_transpose4(hi[c], hi[c + 1], hi[c + 2], hi[c + 3]);
    }
    int8_t* dst = row + k + (part ? Kc : 0);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if (j >= s) continue;
      const uint32_t a = j < 4 ? lo[j & 3] : hi[j & 3], b = j < 4 ? lo[4 + (j & 3)] : hi[4 + (j & 3)];
      int8_t* o = dst + (size_t)(s - 1 - j) * slice_stride;
      if ((Kc & 7) == 0) {
        *reinterpret_cast<uint2*>(o) = make_uint2(a, b);
      } else {
        for (int c = 0; c < 8 && k + c < Kc; c++) o[c] = (int8_t)((c < 4 ? a : b) >> (8 * (c & 3)));
      }
    }
  }
}

// zero the K padding [2 Kc, Kpad) of rows m0 .. m0 + R - 1
template <int R>
__device__ __forceinline__ void oz_row_padding(int8_t* base, int m0, int M, int Kc, int s, int Kpad, size_t slice_stride) {
  const int pad = Kpad - 2 * Kc;
  for (int x = threadIdx.x; x < R * pad * s; x += 256) {
    const int b = x % pad, r = (x / pad) % R, i = x / (pad * R);
    if (m0 + r < M) base[(size_t)i * slice_stride + (size_t)(m0 + r) * Kpad + 2 * Kc + b] = 0;
  }
}

// Rows of A', whole rows staged: one CTA per R rows of one instance (out:
// [inst][s][M][Kpad]), brought
// into shared memory by cp.async, all of it in flight, and read there for the
// scales and for the slices, so that A crosses HBM once.  Entry (row r,
// column c) stands at oz_at<R>: the eight lanes of a quarter warp (one row,
// columns 8 apart) meet on no bank, and neither do the copies (rows fastest).
// Bound by HBM and by issue: 32 x 576 x 576 in six slices, 297 MB, takes 68 us
// (4.4 TB/s); the streamed form below read A twice and took 168 us, 93 with
// today's conversion.
template <int R>
__device__ __forceinline__ int oz_at(int r, int c) {
  return (R == 8 ? c : c ^ ((c >> 5) & 1)) * R + ((r + (c >> 3)) & (R - 1));
}
template <int R>
__global__ void __launch_bounds__(256) k_oz_split_rows_once(OzOperand A, int M, int s, int Kpad,
                                                            int8_t* __restrict__ out, double* __restrict__ rscale) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx* rows = reinterpret_cast<cplx*>(smraw);
  __shared__ double smax[8][R];
  __shared__ int sexp[R];
  const int inst = blockIdx.y;
  const int m0 = blockIdx.x * R;
  const int Kc = A.K1 + A.K2;
  const OzLine V = oz_view(A, inst);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  {
    const int r = threadIdx.x & (R - 1);
    const bool ok = m0 + r < M;
    for (int c = threadIdx.x / R; c < Kc; c += 256 / R)
      oz_cp_async16(rows + oz_at<R>(r, c), ok ? &oz_a(V, m0 + r, c) : V.p1, ok);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    double mx = 0.0;  // of the entries this thread copied
    for (int c = threadIdx.x / R; c < Kc; c += 256 / R) mx = oz_absmax(mx, rows[oz_at<R>(r, c)]);
#pragma unroll
    for (int o = 16; o >= R; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane < R) smax[w][lane] = mx;
  }
  __syncthreads();
  if (threadIdx.x < R) {
    double mx = 0.0;
    for (int i = 0; i < 8; i++) mx = fmax(mx, smax[i][threadIdx.x]);
    const int e = oz_exponent(mx);
    sexp[threadIdx.x] = e;
    const int m = m0 + threadIdx.x;
    if (m < M) rscale[(size_t)inst * M + m] = ldexp(1.0, e);
  }
  __syncthreads();
  const size_t slice_stride = (size_t)M * Kpad;
  int8_t* base = out + (size_t)inst * s * slice_stride;
  const int r = (threadIdx.x >> 3) & (R - 1), m = m0 + r;
  if (m < M) {
    const OzScale sc = oz_scale(sexp[r], s);
#pragma unroll 1
    for (int k = 8 * ((threadIdx.x & 7) + 8 * (threadIdx.x / (8 * R))); k < Kc; k += 8 * (256 / R))
      oz_row_slices([&](int c) { return rows[oz_at<R>(r, k + c)]; }, sc, k, Kc, s, slice_stride,
                    base + (size_t)m * Kpad);
  }
  oz_row_padding<R>(base, m0, M, Kc, s, Kpad, slice_stride);
}

// Rows of A' that are too long for that: one CTA per 32 rows of one instance.
// Pass 1 finds each row's scale (a warp per 8 columns at a time, eight loads
// in flight per thread); pass 2 brings 32 x 64 complex tiles into two
// shared-memory buffers by cp.async, two tiles ahead of the conversion, and
// writes each row's slices as 8-byte runs.  Element (row r, column c) of a tile
// stands at 32 c + ((r + c / 8) & 31), so that neither the copies (rows
// fastest) nor the eight lanes of a quarter warp (one row, columns 8 apart)
// meet on a bank.  Bound by HBM: A is read twice (the second read misses L2).
constexpr int OZ_RT = 64;  // columns per staged tile of the row slicer
constexpr size_t kOzRowsSmem = (size_t)2 * OZ_RT * 32 * sizeof(cplx);
__global__ void __launch_bounds__(256, 3) k_oz_split_rows(OzOperand A, int M, int s, int Kpad, int8_t* __restrict__ out,
                                                       double* __restrict__ rscale) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx* tiles = reinterpret_cast<cplx*>(smraw);
  const int inst = blockIdx.y;
  const int m0 = blockIdx.x * 32;
  const int Kc = A.K1 + A.K2;
  const OzLine V = oz_view(A, inst);
  __shared__ double smax[8][33];
  __shared__ int sexp[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  {
    const int m = m0 + lane;
    double mx[8] = {};
    if (m < M) {
      int k = w;
      for (; k + 56 < Kc; k += 64) {
        cplx v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = oz_a(V, m, k + 8 * j);
#pragma unroll
        for (int j = 0; j < 8; j++) mx[j] = oz_absmax(mx[j], v[j]);
      }
      for (; k < Kc; k += 8) {
        mx[0] = oz_absmax(mx[0], oz_a(V, m, k));
      }
    }
#pragma unroll
    for (int j = 4; j > 0; j >>= 1)
      for (int x = 0; x < j; x++) mx[x] = fmax(mx[x], mx[x + j]);
    smax[w][lane] = mx[0];
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double mx = 0.0;
    for (int i = 0; i < 8; i++) mx = fmax(mx, smax[i][threadIdx.x]);
    const int e = oz_exponent(mx);
    sexp[threadIdx.x] = e;
    const int m = m0 + threadIdx.x;
    if (m < M) rscale[(size_t)inst * M + m] = ldexp(1.0, e);
  }
  const int ntile = (Kc + OZ_RT - 1) / OZ_RT;
  auto load = [&](int t) {
    if (t < ntile) {
      cplx* d = tiles + (size_t)(t & 1) * OZ_RT * 32;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int c = w + 8 * j, k = t * OZ_RT + c;
        const bool ok = m0 + lane < M && k < Kc;
        oz_cp_async16(d + 32 * c + ((lane + (c >> 3)) & 31), ok ? &oz_a(V, m0 + lane, k) : V.p1, ok);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  load(0);
  load(1);
  __syncthreads();
  const size_t slice_stride = (size_t)M * Kpad;
  int8_t* base = out + (size_t)inst * s * slice_stride;
  // thread -> (row rr, 8 consecutive columns 8 cg .. 8 cg + 7): 8 groups x 32 rows
  const int cg = threadIdx.x & 7, rr = threadIdx.x >> 3;
  const int m = m0 + rr;
  const OzScale sc = oz_scale(sexp[rr], s);
  for (int t = 0; t < ntile; t++) {
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncthreads();
    const cplx* tile = tiles + (size_t)(t & 1) * OZ_RT * 32 + 256 * cg + ((rr + cg) & 31);
    const int k = t * OZ_RT + cg * 8;
    if (m < M && k < Kc) {
      oz_row_slices([&](int c) { return tile[32 * c]; }, sc, k, Kc, s, slice_stride, base + (size_t)m * Kpad);
    }
    __syncthreads();
    load(t + 2);
  }
  oz_row_padding<32>(base, m0, M, Kc, s, Kpad, slice_stride);
}

// Columns of B': one warp per complex column j of B (K1 + K2 long); writes
// rows 2j and 2j+1 of every slice.  out: [inst][s][2N][Kpad].  STAGED: the
// warp's column is brought into its own part of shared memory by cp.async, all
// of it in flight at once, and read there for the scale and for the slices;
// entry k stands at k ^ ((k >> 3) & 3), so that the eight lanes of a quarter
// warp (four entries each) meet on no bank.  Otherwise the column is read
// twice from global memory.  32 x 576 x 576 in six slices, 425 MB: 81 us
// (5.2 TB/s), 127 before with two reads from global memory and the digits taken
// one by one.
template <bool STAGED>
__global__ void __launch_bounds__(256) k_oz_split_cols(OzOperand B, int N, int s, int Kpad, int8_t* __restrict__ out,
                                                       double* __restrict__ cscale) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int inst = blockIdx.y;
  const int w = threadIdx.x >> 5;
  const int j = blockIdx.x * (blockDim.x >> 5) + w;
  const int lane = threadIdx.x & 31;
  if (j >= N) return;
  const int Kc = B.K1 + B.K2;
  const OzLine V = oz_view(B, inst);
  cplx* col = reinterpret_cast<cplx*>(smraw) + (size_t)w * ((Kc + 3) & ~3);
  double mx = 0.0;
  if constexpr (STAGED) {
    for (int k = lane; k < ((Kc + 3) & ~3); k += 32)
      oz_cp_async16(col + (k ^ ((k >> 3) & 3)), k < Kc ? &oz_b(V, k, j) : V.p1, k < Kc);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
    for (int k = lane; k < Kc; k += 32) mx = oz_absmax(mx, col[k ^ ((k >> 3) & 3)]);
  } else {
    for (int k = lane; k < Kc; k += 32) mx = oz_absmax(mx, oz_b(V, k, j));
  }
  mx = warp_max(mx);
  const int e = oz_exponent(mx);
  if (lane == 0) cscale[(size_t)inst * N + j] = ldexp(1.0, e);
  const OzScale sc = oz_scale(e, s);
  const size_t slice_stride = (size_t)2 * N * Kpad;
  int8_t* r0 = out + (size_t)inst * s * slice_stride + (size_t)(2 * j) * Kpad;
  int8_t* r1 = r0 + Kpad;
  const bool vec = (Kc & 3) == 0;
#pragma unroll 1
  for (int k = lane * 4; k < Kc; k += 128) {
    cplx v[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      if constexpr (STAGED)
        v[c] = col[(k + c) ^ ((k >> 3) & 3)];
      else
        v[c] = k + c < Kc ? oz_b(V, k + c, j) : cmk(0.0, 0.0);
    }
    uint32_t rl[4], rh[4], il[4], ih[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      oz_digits(v[c].x, sc, rl[c], rh[c]);
      oz_digits(v[c].y, sc, il[c], ih[c]);
    }
    oz_transpose4(rl[0], rl[1], rl[2], rl[3]);
    oz_transpose4(rh[0], rh[1], rh[2], rh[3]);
    oz_transpose4(il[0], il[1], il[2], il[3]);
    oz_transpose4(ih[0], ih[1], ih[2], ih[3]);
#pragma unroll
    for (int d = 0; d < 8; d++) {
      if (d >= s) continue;
      const uint32_t wre = d < 4 ? rl[d & 3] : rh[d & 3], wim = d < 4 ? il[d & 3] : ih[d & 3];
      int8_t* d0 = r0 + (size_t)(s - 1 - d) * slice_stride;
      int8_t* d1 = r1 + (size_t)(s - 1 - d) * slice_stride;
      // the slices of -Im are the negated slices of Im (truncation is odd):
      // a byte-wise negation of the packed digits
      const uint32_t wnim = __vneg4(wim);
      if (vec && k + 3 < Kc) {
        *reinterpret_cast<uint32_t*>(d0 + k) = wre;
        *reinterpret_cast<uint32_t*>(d0 + Kc + k) = wnim;
        *reinterpret_cast<uint32_t*>(d1 + k) = wim;
        *reinterpret_cast<uint32_t*>(d1 + Kc + k) = wre;
      } else {
        for (int c = 0; c < 4 && k + c < Kc; c++) {
          d0[k + c] = (int8_t)(wre >> (8 * c));
          d0[Kc + k + c] = (int8_t)(wnim >> (8 * c));
          d1[k + c] = (int8_t)(wim >> (8 * c));
          d1[Kc + k + c] = (int8_t)(wre >> (8 * c));
        }
      }
    }
  }
  // zero the K padding [2 Kc, Kpad) of rows 2j, 2j+1
  for (int i = 0; i < s; i++)
    for (int b = 2 * Kc + lane; b < Kpad; b += 32) {
      r0[(size_t)i * slice_stride + b] = 0;
      r1[(size_t)i * slice_stride + b] = 0;
    }
}

// ---- tcgen05 helpers ------------------------------------------------------------
__device__ __forceinline__ uint32_t oz_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(oz_smem(bar)), "r"(count));
}

__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(oz_smem(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// SM cycles a wait of the work loop may take before the CTA gives up
// (about 2 s at 1.965 GHz); the waits of the abort path itself, for copies
// and MMAs already in flight, always use this default
constexpr long long OZ_WAIT_CYCLES = 4000000000LL;

// bounded wait: false when the CTA's abort flag is set (honor_abort) or
// `limit` SM cycles pass, in which case the abort flag is set
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          bool honor_abort = true, long long limit = OZ_WAIT_CYCLES) {
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t it = 0;; it++) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255) == 255) {
      if (honor_abort && *abort_flag) return false;
      if (clock64() - t0 > limit) {
        *abort_flag = 1;
        return false;
      }
    }
  }
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(oz_smem(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(oz_smem(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(oz_smem(bar))
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(oz_smem(bar))
               : "memory");
}

__device__ __forceinline__ void tc_mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, int32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// K-major operand tile with 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t oz_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// one lane of a converged warp, and a value that every lane has, in the form
// that lets the compiler keep control flow and operands warp-uniform
__device__ __forceinline__ bool oz_elect() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ uint32_t oz_uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }

// ---- the GEMM ----------------------------------------------------------------------
// Persistent: each CTA walks tiles blockIdx.x, blockIdx.x + gridDim.x, ... of
// the list (instance, row tile, column tile), instance outermost.  Per tile
// the diagonals i + j = d of slice products go two at a time, d1 - 1 and d1 (d
// = 0 alone where s is odd), each into its own of OZ_NBUF TMEM buffers: a
// stage holds the K chunk of A_i and of B_(d1-i), i = 0 .. d1, and serves
// A_i B_(d1-i) and, with the A of the stage before it, A_(i-1) B_(d1-i), so
// that an operand tile is loaded for two products (but the first and the last).
// The eight drain warps (two per TMEM lane quarter, each owning half of the
// tile's columns) fold the finished buffers into FP64 registers, acc +=
// 2^(-7(d+2)) D_d, while the MMAs of the next diagonals proceed; after the last
// diagonal they apply the row and column scales and the epilogue, and the next
// tile starts.
//
// What bounds it: the instructions of the one issuing thread came first (a wait
// and a commit per product and descriptors in divergent code: 600 cycles per
// product of 128 x 128 x 128, of which the MMAs need 256), then the drain
// (tcgen05.ld latency under the MMAs, FP64 conversions, one column's reads
// waiting for the last one's writes).  32 x 576^3 in six slices (1.03 P int8
// operations, 576 rows in 640): 637 us with a stage per product; 650 with two
// diagonals per stage; 490 with one wait and one commit per two products; 430
// with a warp-uniform schedule and one elected lane; 397 with the drain in loads of
// 16 columns, FP64 conversions by addition and four columns' reads ahead (2.6
// POPS).  The tensor pipe is 75 % busy then, and the clock falls to 1.64 GHz under
// the power limit: 367 cycles per product (cycles elapsed, mean over the SMs, over
// the mean number of products of an SM).  The rest is the drain, four times slower
// under the MMAs than alone, and shared memory: 16 KB of copies per product beside
// operand reads of up to 32 KB, which at 128 bytes per cycle would be 384 cycles
// if each MMA fetched both of its operands anew.
enum { OZ_EPI_ZGEMM = 0, OZ_EPI_BSE = 1, OZ_EPI_SUB = 2 };

constexpr int OZ_NBUF = 4;            // TMEM accumulator buffers
constexpr int OZ_MAX_NT = 128;        // columns per tile
constexpr int OZ_HALF = OZ_MAX_NT / 2;
constexpr int OZ_DRAIN_WARPS = 8;
constexpr int OZ_THREADS2 = (OZ_DRAIN_WARPS + 2) * 32;  // + MMA warp + TMA warp

struct OzGemm {
  int M, N;            // complex output size; N' = 2N real columns
  int s;               // slices
  int kchunks;         // Kpad / 128
  int n_tile;          // real columns per tile (multiple of 16, <= 128)
  int m_tiles, n_tiles, tiles;
  const double* rscale;  // [inst][M]
  const double* cscale;  // [inst][N]
  double* status;        // set to status_code on a timed-out wait
  double status_code;
  int epi;
  cplx* C;               // OZ_EPI_ZGEMM: col-major M x N per instance; OZ_EPI_SUB: C -= A B
  int ldc;               // OZ_EPI_SUB: leading dimension and instance stride of C
  long long c_stride;
  cplx* F[4];            // OZ_EPI_BSE: Phi = scale[r] C + omf (F - G) over G
  cplx* G[4];
  double scale[4];
  double omf;
  int q_begin;
  long long wait_cycles;  // limit of the work loop's waits
  int stall_test;         // 1: the MMA warp first waits on a barrier nothing signals
};

// acc += w D of one TMEM lane's `half` columns at tb (up to 8 more of the 512
// columns are read and left unused).  Loads of 16 columns: under the MMAs a
// load's latency, several hundred cycles, and not its width is what counts; 32
// would take the registers that the sums need.  An int32 v becomes exact in FP64 as the low word of
// 2^52 + 2^31 + v, one addition at the full FP64 rate where the conversion
// instruction has a quarter of it.
__device__ __forceinline__ void oz_fold(uint32_t tb, int half, double w, double* acc) {
#pragma unroll
  for (int c = 0; c < OZ_HALF; c += 16) {
    if (c < half) {
      int32_t v[16];
      tc_ld16(tb + (uint32_t)c, v);
#pragma unroll
      for (int e = 0; e < 16; e++)
        acc[c + e] = fma(__hiloint2double(0x43300000, v[e] ^ (int)0x80000000) - 4503601774854144.0, w, acc[c + e]);
    }
  }
}

// where the epilogue of an instance reads and writes
struct OzOut {
  const cplx* in;  // F (BSE only)
  cplx* out;
  size_t ld;
  double scale;
};
template <int EPI>
__device__ __forceinline__ OzOut oz_out(const OzGemm& P, int inst) {
  OzOut o = {nullptr, nullptr, (size_t)P.M, 1.0};
  if constexpr (EPI == OZ_EPI_BSE) {
    const int r = inst & 3;
    const size_t at = (size_t)P.M * P.M * (P.q_begin + (inst >> 2));
    o.in = (r == 0 ? P.F[0] : r == 1 ? P.F[1] : r == 2 ? P.F[2] : P.F[3]) + at;
    o.out = (r == 0 ? P.G[0] : r == 1 ? P.G[1] : r == 2 ? P.G[2] : P.G[3]) + at;
    o.scale = r == 0 ? P.scale[0] : r == 1 ? P.scale[1] : r == 2 ? P.scale[2] : P.scale[3];
  } else if constexpr (EPI == OZ_EPI_SUB) {
    o.out = P.C + (size_t)inst * P.c_stride;
    o.ld = P.ldc;
  } else {
    o.out = P.C + (size_t)inst * P.M * P.N;
  }
  return o;
}

// scales and epilogue of one row m: acc[0 .. half) are the real columns np0 ..,
// lane l of the warp holds the column scale of complex column np0 / 2 + l.  The
// reads of four columns go out together, before writes that they could alias;
// rows and columns beyond the matrix read its last ones and write nothing.
template <int EPI>
__device__ __forceinline__ void oz_epilogue(const OzGemm& P, int inst, int m, int np0, int half, const double* acc,
                                            double rs, double cs) {
  const int jc0 = np0 >> 1, nj = min(half >> 1, P.N - jc0);
  const OzOut o = oz_out<EPI>(P, inst);
  const size_t ld = o.ld;
  cplx* out = o.out + ld * jc0;
  const cplx* in = EPI == OZ_EPI_BSE ? o.in + ld * jc0 : nullptr;
  const double sr = o.scale;
  const int mr = min(m, P.M - 1);
#pragma unroll
  for (int c0 = 0; c0 < OZ_HALF / 2; c0 += 4) {
    if (c0 >= nj) continue;
    cplx f[4], g[4];
    if constexpr (EPI != OZ_EPI_ZGEMM) {
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const size_t ix = mr + ld * min(c0 + c, nj - 1);
        if constexpr (EPI == OZ_EPI_BSE) f[c] = in[ix];
        g[c] = out[ix];
      }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const double sc = rs * __shfl_sync(0xffffffffu, cs, c0 + c);
      const double cre = acc[2 * (c0 + c)] * sc, cim = acc[2 * (c0 + c) + 1] * sc;
      cplx v;
      if constexpr (EPI == OZ_EPI_ZGEMM)
        v = cmk(cre, cim);
      else if constexpr (EPI == OZ_EPI_SUB)
        v = cmk(g[c].x - cre, g[c].y - cim);
      else
        v = cmk(__dadd_rn(__dmul_rn(sr, cre), __dmul_rn(P.omf, __dsub_rn(f[c].x, g[c].x))),
                __dadd_rn(__dmul_rn(sr, cim), __dmul_rn(P.omf, __dsub_rn(f[c].y, g[c].y))));
      if (m < P.M && c0 + c < nj) out[m + ld * (c0 + c)] = v;
    }
  }
}

template <int EPI>
__global__ void __launch_bounds__(OZ_THREADS2, 1)
    k_oz_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, OzGemm P) {
  extern __shared__ uint8_t oz_dyn[];
  __shared__ uint64_t full_bar[OZ_STAGES], empty_bar[OZ_STAGES], accf_bar[OZ_NBUF], acce_bar[OZ_NBUF], done_bar;
  __shared__ uint64_t never_bar;  // initialised, never arrived on: the stall test waits here
  __shared__ uint32_t tmem_base_sh;
  __shared__ volatile int abort_sh;
  __shared__ int issued_sh, consumed_sh;

  const int warp = (int)oz_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int Np = 2 * P.N;
  const uint32_t a_bytes = OZ_BM * OZ_BK, b_bytes = (uint32_t)P.n_tile * OZ_BK;
  const uint32_t dyn = (oz_smem(oz_dyn) + 1023u) & ~1023u;
  auto slot_a = [&](int st) { return dyn + (uint32_t)st * OZ_STAGE_BYTES; };
  auto slot_b = [&](int st) { return dyn + (uint32_t)st * OZ_STAGE_BYTES + OZ_BM * OZ_BK; };
  const int per_inst = P.m_tiles * P.n_tiles;

  if (threadIdx.x == 0) {
    for (int i = 0; i < OZ_STAGES; i++) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < OZ_NBUF; i++) {
      mbar_init(&accf_bar[i], 1);
      mbar_init(&acce_bar[i], OZ_DRAIN_WARPS * 32);
    }
    mbar_init(&done_bar, 1);
    mbar_init(&never_bar, 1);
    abort_sh = 0;
    issued_sh = 0;
    consumed_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == OZ_DRAIN_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(oz_smem(&tmem_base_sh)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = oz_uniform(tmem_base_sh);

  if (warp == OZ_DRAIN_WARPS + 1) {
    // ---- TMA producer ----
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int issued = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < P.tiles && ok; t += gridDim.x) {
        const int inst = t / per_inst, rem = t % per_inst;
        const int m0 = (rem % P.m_tiles) * OZ_BM, n0 = (rem / P.m_tiles) * P.n_tile;
        // steps (d1 - 1, d1): stages (A_i, B_(d1 - i)), i = 0 .. d1
        for (int d1 = (P.s & 1) ? 0 : 1; d1 < P.s && ok; d1 += 2)
          for (int kc = 0; kc < P.kchunks && ok; kc++)
            for (int i = 0; i <= d1; i++) {
              if (!mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_sh, true, P.wait_cycles)) {
                ok = false;
                break;
              }
              mbar_expect_tx(&full_bar[stage], a_bytes + b_bytes);
              tma_load_2d(slot_b(stage), &tmB, kc * OZ_BK, (inst * P.s + d1 - i) * Np + n0, &full_bar[stage]);
              tma_load_2d(slot_a(stage), &tmA, kc * OZ_BK, (inst * P.s + i) * P.M + m0, &full_bar[stage]);
              issued++;
              if (++stage == OZ_STAGES) {
                stage = 0;
                phase ^= 1u;
              }
            }
      }
      issued_sh = issued;
    }
  } else if (warp == OZ_DRAIN_WARPS) {
    // ---- MMA issuer ----
    // the whole warp walks the schedule, so that it is uniform; one lane issues
    {
      const bool el = oz_elect();
      auto wait = [&](uint64_t* bar, uint32_t ph) {
        return __all_sync(0xffffffffu, mbar_wait(bar, ph, &abort_sh, true, P.wait_cycles)) != 0;
      };
      const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(P.n_tile >> 3) << 17) |
                             ((uint32_t)(OZ_BM >> 4) << 24);
      const uint64_t desc0 = oz_desc(dyn);  // of stage 0's A; the address counts 16 bytes
      int stage = 0;
      uint32_t phase = 0;
      int consumed = 0;
      int nacc = 0;  // accumulations issued so far (one per tile and diagonal)
      bool ok = true;
      // failure-path test: a wait that can only run out, before any MMA
      if (P.stall_test) ok = wait(&never_bar, 0);
      for (int t = blockIdx.x; t < P.tiles && ok; t += gridDim.x)
        for (int d1 = (P.s & 1) ? 0 : 1; d1 < P.s && ok; d1 += 2) {
          const int nb = d1 > 0 ? 2 : 1;  // diagonals of this step
          for (int b = 0; b < nb && ok; b++) {
            const int n = nacc + b;
            if (n >= OZ_NBUF)
              ok = wait(&acce_bar[n % OZ_NBUF], (uint32_t)((n - OZ_NBUF) / OZ_NBUF) & 1u);
          }
          tc_fence_after();
          const uint32_t dt1 = tmem + (uint32_t)((nacc + nb - 1) % OZ_NBUF * OZ_MAX_NT);
          const uint32_t dt0 = tmem + (uint32_t)(nacc % OZ_NBUF * OZ_MAX_NT);
          for (int kc = 0; kc < P.kchunks && ok; kc++) {
            uint64_t da = 0;
            int prev = 0;
            for (int i = 0; i <= d1; i++) {
              if (!wait(&full_bar[stage], phase)) {
                ok = false;
                break;
              }
              consumed++;
              tc_fence_after();
              const uint64_t db = desc0 + (uint32_t)(stage * (int)(OZ_STAGE_BYTES >> 4)) + (OZ_BM * OZ_BK >> 4);
              if (i > 0 && el) {  // A_(i-1) B_(d1-i): diagonal d1 - 1
#pragma unroll
                for (int kk = 0; kk < OZ_BK / 32; kk++)
                  tc_mma_i8(dt0, da + 2 * kk, db + 2 * kk, idesc, kc > 0 || i > 1 || kk > 0);
                tc_commit(&empty_bar[prev]);
              }
              da = desc0 + (uint32_t)(stage * (int)(OZ_STAGE_BYTES >> 4));
              if (el) {
#pragma unroll
                for (int kk = 0; kk < OZ_BK / 32; kk++)
                  tc_mma_i8(dt1, da + 2 * kk, db + 2 * kk, idesc, kc > 0 || i > 0 || kk > 0);
              }
              prev = stage;
              if (++stage == OZ_STAGES) {
                stage = 0;
                phase ^= 1u;
              }
            }
            if (ok && el) tc_commit(&empty_bar[prev]);
          }
          for (int b = 0; b < nb && ok; b++, nacc++)
            if (el) tc_commit(&accf_bar[nacc % OZ_NBUF]);
        }
      if (el) {
        consumed_sh = consumed;
        tc_commit(&done_bar);
        mbar_wait(&done_bar, 0, &abort_sh, false);
      }
      __syncwarp();
    }
  } else {
    // ---- drain: warp w reads TMEM lanes 32 (w % 4) .. + 31 and columns
    //      [h n_tile/2, (h+1) n_tile/2), h = w / 4 ----
    const int quarter = warp & 3, h = warp >> 2;
    const int half = P.n_tile >> 1;
    const int row = quarter * 32 + lane;
    double acc[OZ_HALF];
    int nacc = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < P.tiles && ok; t += gridDim.x) {
      const int inst = t / per_inst, rem = t % per_inst;
      const int m0 = (rem % P.m_tiles) * OZ_BM, n0 = (rem / P.m_tiles) * P.n_tile;
      const int m = m0 + row;
      const int np0 = n0 + h * half;
      // the scales, long before their use
      const double rs = m < P.M ? __ldg(P.rscale + (size_t)inst * P.M + m) : 0.0;
      const double cs = 2 * lane < half && (np0 >> 1) + lane < P.N ? __ldg(P.cscale + (size_t)inst * P.N + (np0 >> 1) + lane) : 0.0;
#pragma unroll
      for (int c = 0; c < OZ_HALF; c++) acc[c] = 0.0;
      for (int d = 0; d < P.s; d++, nacc++) {
        const int buf = nacc % OZ_NBUF;
        if (!mbar_wait(&accf_bar[buf], (uint32_t)(nacc / OZ_NBUF) & 1u, &abort_sh, true, P.wait_cycles)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const double w = ldexp(1.0, -OZ_SLICE_BITS * (d + 2));
        const uint32_t tb = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * OZ_MAX_NT + h * half);
        oz_fold(tb, half, w, acc);
        tc_fence_before();
        mbar_arrive(&acce_bar[buf]);
      }
      if (!ok) break;
      oz_epilogue<EPI>(P, inst, m, np0, half, acc, rs, cs);
    }
  }

  __syncthreads();
  if (threadIdx.x == 0 && abort_sh) {
    *P.status = P.status_code;
    // wait for the TMA copies that were issued but never consumed
    int stage = consumed_sh % OZ_STAGES;
    uint32_t phase = (uint32_t)(consumed_sh / OZ_STAGES) & 1u;
    for (int k = consumed_sh; k < issued_sh; k++) {
      mbar_wait(&full_bar[stage], phase, &abort_sh, false);
      if (++stage == OZ_STAGES) {
        stage = 0;
        phase ^= 1u;
      }
    }
  }
  __syncthreads();
  if (warp == OZ_DRAIN_WARPS) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

// ---- the GEMM on CTA pairs (tcgen05 cta_group::2) ------------------------------
// The same tiles, diagonal schedule and FP64 folding as k_oz_gemm (so the
// same bits), but a cluster of two CTAs computes a 256 x n_tile tile with
// one M = 256 MMA per K step: CTA r stages rows 128 r .. 128 r + 127 of the
// pair's A rows and half of the tile's B columns (n_tile / 2 rows of B'), so
// each SM's tensor core reads 4 KB + n_tile x 16 B of operands per MMA
// instead of 4 KB + n_tile x 32 B.  The leader (cluster rank 0) issues the
// MMAs and owns the stage-full barriers (both CTAs' copies complete there);
// the MMA completions reach both CTAs' stage-empty and accumulator-full
// barriers by multicast commits; each CTA's drain warps read their own TMEM
// rows and arrive on the leader's accumulator-empty barrier.  Only the
// tensor maps of this GPU's own memory are read, and no copy multicasts.
constexpr int OZ2_STAGES = 9;  // 9 x (16 KB of A + <= 8 KB of B)
constexpr uint32_t OZ2_STAGE_BYTES = OZ_BM * OZ_BK + OZ_HALF * OZ_BK;

__device__ __forceinline__ uint32_t oz_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the shared::cluster address of `addr` (a shared::cta address) in CTA `rank`
__device__ __forceinline__ uint32_t oz_mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void oz_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_cl(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(oz_smem(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait with cluster-scope acquire (barriers that other CTAs signal)
__device__ __forceinline__ bool mbar_wait_cl(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                             bool honor_abort = true, long long limit = OZ_WAIT_CYCLES) {
  if (mbar_try_cl(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t it = 0;; it++) {
    if (mbar_try_cl(bar, parity)) return true;
    if ((it & 255) == 255) {
      if (honor_abort && *abort_flag) return false;
      if (clock64() - t0 > limit) {
        *abort_flag = 1;
        return false;
      }
    }
  }
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y,
                                                 uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
      "%3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar_cluster)
      : "memory");
}
// MMA completion to the barrier at this offset in the CTAs of `mask`
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          oz_smem(bar)),
      "h"(mask)
      : "memory");
}
__device__ __forceinline__ void tc_mma_i8_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8, %9, %10, %11, %12}, p;\n\t}" ::"r"(
          d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u),
      "r"(0u), "r"(0u));
}

// P.m_tiles counts 256-row pair tiles here
template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(OZ_THREADS2, 1)
    k_oz_gemm2(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, OzGemm P) {
  extern __shared__ uint8_t oz_dyn[];
  __shared__ uint64_t full_bar[OZ2_STAGES], empty_bar[OZ2_STAGES], accf_bar[OZ_NBUF], acce_bar[OZ_NBUF], done_bar;
  __shared__ uint64_t never_bar;
  __shared__ uint32_t tmem_base_sh;
  __shared__ volatile int abort_sh;
  __shared__ int issued_sh, consumed_sh;

  const int warp = (int)oz_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t crank = oz_cluster_rank();
  const bool leader = crank == 0;
  const int Np = 2 * P.N;
  const int NT = P.n_tile, HB = NT >> 1;  // B' rows staged by each CTA
  const uint32_t a_bytes = OZ_BM * OZ_BK, b_bytes = (uint32_t)HB * OZ_BK;
  const uint32_t dyn = (oz_smem(oz_dyn) + 1023u) & ~1023u;
  auto slot_a = [&](int st) { return dyn + (uint32_t)st * OZ2_STAGE_BYTES; };
  auto slot_b = [&](int st) { return dyn + (uint32_t)st * OZ2_STAGE_BYTES + OZ_BM * OZ_BK; };
  const int per_inst = P.m_tiles * P.n_tiles;
  const int cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int i = 0; i < OZ2_STAGES; i++) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < OZ_NBUF; i++) {
      mbar_init(&accf_bar[i], 1);
      mbar_init(&acce_bar[i], 2 * OZ_DRAIN_WARPS * 32);
    }
    mbar_init(&done_bar, 1);
    mbar_init(&never_bar, 1);
    abort_sh = 0;
    issued_sh = 0;
    consumed_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == OZ_DRAIN_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(oz_smem(&tmem_base_sh)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  // both CTAs' barriers exist before either CTA signals the other's
  oz_cluster_sync();
  tc_fence_after();
  const uint32_t tmem = oz_uniform(tmem_base_sh);

  if (warp == OZ_DRAIN_WARPS + 1) {
    // ---- TMA producer (both CTAs): own rows of A, own half of B' ----
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int issued = 0;
      bool ok = true;
      for (int t = cid; t < P.tiles && ok; t += ncl) {
        const int inst = t / per_inst, rem = t % per_inst;
        const int m0 = (rem % P.m_tiles) * (2 * OZ_BM) + (int)crank * OZ_BM;
        const int n0 = (rem / P.m_tiles) * NT + (int)crank * HB;
        for (int d1 = (P.s & 1) ? 0 : 1; d1 < P.s && ok; d1 += 2)
          for (int kc = 0; kc < P.kchunks && ok; kc++)
            for (int i = 0; i <= d1; i++) {
              if (!mbar_wait_cl(&empty_bar[stage], phase ^ 1u, &abort_sh, true, P.wait_cycles)) {
                ok = false;
                break;
              }
              // the leader's stage-full barrier counts both CTAs' bytes
              if (leader) mbar_expect_tx(&full_bar[stage], 2 * (a_bytes + b_bytes));
              const uint32_t fb = oz_mapa(oz_smem(&full_bar[stage]), 0);
              tma_load_2d_pair(slot_b(stage), &tmB, kc * OZ_BK, (inst * P.s + d1 - i) * Np + n0, fb);
              tma_load_2d_pair(slot_a(stage), &tmA, kc * OZ_BK, (inst * P.s + i) * P.M + m0, fb);
              issued++;
              if (++stage == OZ2_STAGES) {
                stage = 0;
                phase ^= 1u;
              }
            }
      }
      issued_sh = issued;
    }
  } else if (warp == OZ_DRAIN_WARPS) {
    // ---- MMA issuer: the leader only ----
    // the whole warp walks the schedule, so that it is uniform; one lane issues
    if (leader) {
      const bool el = oz_elect();
      auto wait = [&](uint64_t* bar, uint32_t ph) {
        return __all_sync(0xffffffffu, mbar_wait_cl(bar, ph, &abort_sh, true, P.wait_cycles)) != 0;
      };
      const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) |
                             ((uint32_t)((2 * OZ_BM) >> 4) << 24);
      const uint64_t desc0 = oz_desc(dyn);  // of stage 0's A; the address counts 16 bytes
      int stage = 0;
      uint32_t phase = 0;
      int consumed = 0;
      int nacc = 0;  // accumulations issued so far (one per tile and diagonal)
      bool ok = true;
      // failure-path test: a wait that can only run out, before any MMA
      if (P.stall_test) ok = wait(&never_bar, 0);
      for (int t = cid; t < P.tiles && ok; t += ncl)
        for (int d1 = (P.s & 1) ? 0 : 1; d1 < P.s && ok; d1 += 2) {
          const int nb = d1 > 0 ? 2 : 1;  // diagonals of this step
          for (int b = 0; b < nb && ok; b++) {
            const int n = nacc + b;
            if (n >= OZ_NBUF)
              ok = wait(&acce_bar[n % OZ_NBUF], (uint32_t)((n - OZ_NBUF) / OZ_NBUF) & 1u);
          }
          tc_fence_after();
          const uint32_t dt1 = tmem + (uint32_t)((nacc + nb - 1) % OZ_NBUF * OZ_MAX_NT);
          const uint32_t dt0 = tmem + (uint32_t)(nacc % OZ_NBUF * OZ_MAX_NT);
          for (int kc = 0; kc < P.kchunks && ok; kc++) {
            uint64_t da = 0;
            int prev = 0;
            for (int i = 0; i <= d1; i++) {
              if (!wait(&full_bar[stage], phase)) {
                ok = false;
                break;
              }
              consumed++;
              tc_fence_after();
              const uint64_t db = desc0 + (uint32_t)(stage * (int)(OZ2_STAGE_BYTES >> 4)) + (OZ_BM * OZ_BK >> 4);
              if (i > 0 && el) {  // A_(i-1) B_(d1-i): diagonal d1 - 1
#pragma unroll
                for (int kk = 0; kk < OZ_BK / 32; kk++)
                  tc_mma_i8_pair(dt0, da + 2 * kk, db + 2 * kk, idesc, kc > 0 || i > 1 || kk > 0);
                tc_commit_pair(&empty_bar[prev], 0x3);
              }
              da = desc0 + (uint32_t)(stage * (int)(OZ2_STAGE_BYTES >> 4));
              if (el) {
#pragma unroll
                for (int kk = 0; kk < OZ_BK / 32; kk++)
                  tc_mma_i8_pair(dt1, da + 2 * kk, db + 2 * kk, idesc, kc > 0 || i > 0 || kk > 0);
              }
              prev = stage;
              if (++stage == OZ2_STAGES) {
                stage = 0;
                phase ^= 1u;
              }
            }
            if (ok && el) tc_commit_pair(&empty_bar[prev], 0x3);
          }
          for (int b = 0; b < nb && ok; b++, nacc++)
            if (el) tc_commit_pair(&accf_bar[nacc % OZ_NBUF], 0x3);
        }
      if (el) {
        consumed_sh = consumed;
        tc_commit_pair(&done_bar, 0x1);
        mbar_wait_cl(&done_bar, 0, &abort_sh, false);
      }
      __syncwarp();
    }
  } else {
    // ---- drain (both CTAs): own TMEM lanes = own 128 rows of the pair tile ----
    const int quarter = warp & 3, h = warp >> 2;
    const int half = NT >> 1;
    const int row = quarter * 32 + lane;
    const uint32_t acce_leader0 = oz_mapa(oz_smem(&acce_bar[0]), 0);
    double acc[OZ_HALF];
    int nacc = 0;
    bool ok = true;
    for (int t = cid; t < P.tiles && ok; t += ncl) {
      const int inst = t / per_inst, rem = t % per_inst;
      const int m0 = (rem % P.m_tiles) * (2 * OZ_BM) + (int)crank * OZ_BM;
      const int n0 = (rem / P.m_tiles) * NT;
      const int m = m0 + row;
      const int np0 = n0 + h * half;
      // the scales, long before their use
      const double rs = m < P.M ? __ldg(P.rscale + (size_t)inst * P.M + m) : 0.0;
      const double cs = 2 * lane < half && (np0 >> 1) + lane < P.N ? __ldg(P.cscale + (size_t)inst * P.N + (np0 >> 1) + lane) : 0.0;
#pragma unroll
      for (int c = 0; c < OZ_HALF; c++) acc[c] = 0.0;
      for (int d = 0; d < P.s; d++, nacc++) {
        const int buf = nacc % OZ_NBUF;
        if (!mbar_wait_cl(&accf_bar[buf], (uint32_t)(nacc / OZ_NBUF) & 1u, &abort_sh, true, P.wait_cycles)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const double w = ldexp(1.0, -OZ_SLICE_BITS * (d + 2));
        const uint32_t tb = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * OZ_MAX_NT + h * half);
        oz_fold(tb, half, w, acc);
        tc_fence_before();
        mbar_arrive_remote(acce_leader0 + (uint32_t)(buf * sizeof(uint64_t)));
      }
      if (!ok) break;
      oz_epilogue<EPI>(P, inst, m, np0, half, acc, rs, cs);
    }
  }

  __syncthreads();
  if (threadIdx.x == 0 && abort_sh) {
    *P.status = P.status_code;
    if (leader) {
      // wait for the stages whose copies were issued but never consumed
      int stage = consumed_sh % OZ2_STAGES;
      uint32_t phase = (uint32_t)(consumed_sh / OZ2_STAGES) & 1u;
      for (int k = consumed_sh; k < issued_sh; k++) {
        mbar_wait_cl(&full_bar[stage], phase, &abort_sh, false);
        if (++stage == OZ2_STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  }
  __syncthreads();
  // neither CTA frees its shared or tensor memory while the other may still use it
  oz_cluster_sync();
  if (warp == OZ_DRAIN_WARPS) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

// ---- host side ----------------------------------------------------------------------
// the work loop's wait limit (0: OZ_WAIT_CYCLES) and a pending stall test,
// set by tups_set_split_wait; the stall test applies to the next launch only
static std::atomic<long long> g_oz_wait_cycles{0};
static std::atomic<int> g_oz_stall_test{0};
static std::atomic<int> g_oz_n_tile{0};  // 0: oz_n_tile
static std::atomic<int> g_oz_pairs{0};   // 1: k_oz_gemm2 (CTA pairs) for M >= 256

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 2-D byte tensor [rows][Kpad], boxes of 128 bytes x box_rows, 128-byte swizzle
static bool make_map(CUtensorMap* map, const int8_t* base, long long rows, int Kpad, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  if (((uintptr_t)base & 15) || (Kpad % OZ_BK) || box_rows < 1 || box_rows > 256) return false;
  cuuint64_t dims[2] = {(cuuint64_t)Kpad, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)Kpad};
  cuuint32_t box[2] = {(cuuint32_t)OZ_BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)base, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int oz_kpad(int K) { return (int)(((long long)2 * K + OZ_BK - 1) / OZ_BK * OZ_BK); }

// columns per tile: multiple of 16, <= 128; cost = tiles x (columns + 64),
// the 64 standing for the per-tile cost of streaming the A rows
int oz_n_tile(int N) {
  const int Np = 2 * N;
  int best = 16;
  long long best_cost = -1;
  for (int t = 16; t <= OZ_MAX_NT; t += 16) {
    const long long cost = (long long)((Np + t - 1) / t) * (t + 64);
    if (best_cost < 0 || cost < best_cost || (cost == best_cost && t > best)) {
      best = t;
      best_cost = cost;
    }
  }
  return best;
}

size_t oz_smem_bytes() {  // > half of the SM's: the CTA owns all 512 TMEM columns
  return (size_t)OZ_STAGES * OZ_STAGE_BYTES + 1024;
}

OzWork oz_work_layout(int batch, int M, int N, int K, int s) {
  OzWork w;
  w.Kpad = oz_kpad(K);
  w.a_bytes = (size_t)batch * s * M * w.Kpad;
  w.b_bytes = (size_t)batch * s * 2 * N * w.Kpad;
  w.rs_bytes = (size_t)batch * M * sizeof(double);
  w.cs_bytes = (size_t)batch * N * sizeof(double);
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  w.total = up(w.a_bytes) + up(w.b_bytes) + up(w.rs_bytes) + up(w.cs_bytes) + 256;
  return w;
}

void oz_bind_work(OzRun& R, const OzWork& w, void* base) {
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  uint8_t* p = (uint8_t*)(((uintptr_t)base + 255) & ~(uintptr_t)255);
  R.a_slices = (int8_t*)p;
  p += up(w.a_bytes);
  R.b_slices = (int8_t*)p;
  p += up(w.b_bytes);
  R.rscale = (double*)p;
  p += up(w.rs_bytes);
  R.cscale = (double*)p;
}

// a failed CUDA step of oz_run on stderr (the batched ZGEMM entry point has no
// context to keep a message in)
static int oz_fail(const char* step, cudaError_t e) {
  std::fprintf(stderr, "tups split GEMM: %s failed: %s\n", step, e == cudaSuccess ? "-" : cudaGetErrorString(e));
  return TUPS_ERR_CUDA;
}

int oz_run(OzRun& R, cudaStream_t stream, long long* launches) {
  const int M = R.M, N = R.N, s = R.s, batch = R.batch;
  if (s < 1 || s > 8) return TUPS_ERR_BADARG;
  if (R.A.K1 + R.A.K2 != R.B.K1 + R.B.K2) return TUPS_ERR_BADDIM;
  const int K = R.A.K1 + R.A.K2;
  // exactness of the int32 sums: s K' 127^2 < 2^31
  if ((long long)s * 2 * K * 127 * 127 >= (1LL << 31)) return TUPS_ERR_BADDIM;
  const int Kpad = oz_kpad(K);
  if ((long long)batch * s * std::max(M, 2 * N) >= (1LL << 31)) return TUPS_ERR_BADDIM;
  // rows of the split kernels
  {
    cudaError_t e;
    auto rows = [&](auto* kernel, int nr, size_t smem) {
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess)
        kernel<<<dim3((M + nr - 1) / nr, batch), 256, smem, stream>>>(R.A, M, s, Kpad, R.a_slices, R.rscale);
    };
    const size_t entry = (size_t)((K + 7) & ~7) * sizeof(cplx);
    // whole rows while three CTAs of them share an SM (K' = 576: 68 us against 93 for
    // the streamed rows, 4 of them at 1152: 131 against 179); longer ones are
    // streamed (2304: 182 against 219 for 4 rows of 147 KB, one CTA per SM)
    if (8 * entry <= kOzLinesSmem)
      rows(k_oz_split_rows_once<8>, 8, 8 * entry);
    else if (4 * entry <= kOzLinesSmem)
      rows(k_oz_split_rows_once<4>, 4, 4 * entry);
    else
      rows(k_oz_split_rows, 32, kOzRowsSmem);
    if (e != cudaSuccess) return oz_fail("slice kernel attribute", e);
    if (launches) (*launches)++;
    // as many columns per CTA as fit; a column beyond that is read twice
    const size_t line = (size_t)((K + 3) & ~3) * sizeof(cplx);
    const bool staged = line <= kOzLinesSmem;
    int cols = 8;
    while (staged && cols > 1 && cols * line > kOzLinesSmem) cols /= 2;
    dim3 gc((N + cols - 1) / cols, batch);
    if (staged) {
      e = cudaFuncSetAttribute(k_oz_split_cols<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOzLinesSmem);
      if (e != cudaSuccess) return oz_fail("slice kernel attribute", e);
      k_oz_split_cols<true><<<gc, 32 * cols, cols * line, stream>>>(R.B, N, s, Kpad, R.b_slices, R.cscale);
    } else {
      k_oz_split_cols<false><<<gc, 256, 0, stream>>>(R.B, N, s, Kpad, R.b_slices, R.cscale);
    }
    if (launches) (*launches)++;
    e = cudaGetLastError();
    if (e != cudaSuccess) return oz_fail("slice kernels launch", e);
  }
  OzGemm P;
  std::memset(&P, 0, sizeof(P));
  P.M = M;
  P.N = N;
  P.s = s;
  P.kchunks = Kpad / OZ_BK;
  const bool pairs = g_oz_pairs.load() != 0 && M >= 2 * OZ_BM;
  {
    const int nt = g_oz_n_tile.load();
    P.n_tile = nt > 0 ? nt : oz_n_tile(N);
    // CTA pairs: each CTA stages n_tile / 2 rows of B', a multiple of 16
    if (pairs) P.n_tile = std::min(OZ_MAX_NT, (P.n_tile + 31) / 32 * 32);
  }
  P.m_tiles = pairs ? (M + 2 * OZ_BM - 1) / (2 * OZ_BM) : (M + OZ_BM - 1) / OZ_BM;
  P.n_tiles = (2 * N + P.n_tile - 1) / P.n_tile;
  if ((long long)batch * P.m_tiles * P.n_tiles >= (1LL << 31)) return TUPS_ERR_BADDIM;
  P.tiles = batch * P.m_tiles * P.n_tiles;
  P.rscale = R.rscale;
  P.cscale = R.cscale;
  P.status = R.status;
  P.status_code = R.status_code;
  P.epi = R.epi;
  P.C = R.C;
  P.ldc = R.ldc;
  P.c_stride = R.c_stride;
  for (int r = 0; r < 4; r++) {
    P.F[r] = R.F[r];
    P.G[r] = R.G[r];
    P.scale[r] = R.scale[r];
  }
  P.omf = R.omf;
  P.q_begin = R.q_begin;
  {
    const long long lim = g_oz_wait_cycles.load();
    P.wait_cycles = lim > 0 ? lim : OZ_WAIT_CYCLES;
    P.stall_test = g_oz_stall_test.exchange(0);
  }
  CUtensorMap ta, tb;
  if (!make_map(&ta, R.a_slices, (long long)batch * s * M, Kpad, OZ_BM))
    return oz_fail("tensor map of the A slices", cudaSuccess);
  if (!make_map(&tb, R.b_slices, (long long)batch * s * 2 * N, Kpad, pairs ? P.n_tile / 2 : P.n_tile))
    return oz_fail("tensor map of the B slices", cudaSuccess);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e;
  if (pairs) {
    const size_t smem = (size_t)OZ2_STAGES * OZ2_STAGE_BYTES + 1024;
    auto* kernel = P.epi == OZ_EPI_BSE ? k_oz_gemm2<OZ_EPI_BSE> : P.epi == OZ_EPI_SUB ? k_oz_gemm2<OZ_EPI_SUB> : k_oz_gemm2<OZ_EPI_ZGEMM>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return oz_fail("k_oz_gemm2 shared memory attribute", e);
    const int grid = 2 * std::max(1, std::min(P.tiles, sms / 2));
    kernel<<<grid, OZ_THREADS2, smem, stream>>>(ta, tb, P);
    if (launches) (*launches)++;
    e = cudaGetLastError();
    return e == cudaSuccess ? TUPS_OK : oz_fail("k_oz_gemm2 launch", e);
  }
  const size_t smem = oz_smem_bytes();
  auto* kernel = P.epi == OZ_EPI_BSE ? k_oz_gemm<OZ_EPI_BSE> : P.epi == OZ_EPI_SUB ? k_oz_gemm<OZ_EPI_SUB> : k_oz_gemm<OZ_EPI_ZGEMM>;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return oz_fail("k_oz_gemm shared memory attribute", e);
  const int grid = std::max(1, std::min(P.tiles, sms));
  kernel<<<grid, OZ_THREADS2, smem, stream>>>(ta, tb, P);
  if (launches) (*launches)++;
  e = cudaGetLastError();
  return e == cudaSuccess ? TUPS_OK : oz_fail("k_oz_gemm launch", e);
}

}  // namespace tups

// ---- C-ABI: batched split-precision ZGEMM ---------------------------------------------
extern "C" size_t tups_zgemm_split_workspace(int batch, int M, int N, int K, int slices) {
  if (batch < 1 || M < 1 || N < 1 || K < 1 || slices < 1 || slices > 8) return 0;
  return tups::oz_work_layout(batch, M, N, K, slices).total + 256;
}

extern "C" int tups_zgemm_split(int batch, int M, int N, int K, const double* A, const double* B, double* C,
                                int slices, void* work, size_t work_bytes, void* stream) {
  using namespace tups;
  if (batch < 1 || M < 1 || N < 1 || K < 1 || !A || !B || !C || !work) return TUPS_ERR_BADARG;
  if (slices < 1 || slices > 8) return TUPS_ERR_BADARG;
  const OzWork w = oz_work_layout(batch, M, N, K, slices);
  if (work_bytes < w.total + 256) return TUPS_ERR_BADARG;
  cudaStream_t st = (cudaStream_t)stream;
  OzRun R;
  R.batch = batch;
  R.M = M;
  R.N = N;
  R.s = slices;
  R.A.p1 = (const cplx*)A;
  R.A.s1 = (long long)M * K;
  R.A.ld1 = M;
  R.A.K1 = K;
  R.B.p1 = (const cplx*)B;
  R.B.s1 = (long long)K * N;
  R.B.ld1 = K;
  R.B.K1 = K;
  oz_bind_work(R, w, work);
  // the status slot sits after the carved buffers
  double* status = (double*)((uint8_t*)work + w.total);
  status = (double*)(((uintptr_t)status + 7) & ~(uintptr_t)7);
  if ((uint8_t*)(status + 1) > (uint8_t*)work + work_bytes) return TUPS_ERR_BADARG;
  if (cudaMemsetAsync(status, 0, sizeof(double), st) != cudaSuccess) return TUPS_ERR_CUDA;
  R.status = status;
  R.status_code = 1.0;
  R.epi = 0;
  R.C = (cplx*)C;
  int rc = oz_run(R, st, nullptr);
  if (rc) return rc;
  double flag = 0.0;
  cudaError_t e = cudaMemcpyAsync(&flag, status, sizeof(double), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return oz_fail("split ZGEMM completion", e);
  return flag != 0.0 ? TUPS_ERR_TIMEOUT : TUPS_OK;
}

// Failure detection of the split GEMM's bounded device waits.  cycles > 0
// sets how many SM cycles a wait of the work loop may take (0 restores the
// default, about 2 s); stall_test = 1 makes the next split GEMM launch wait
// first on a barrier that nothing signals, so its bounded wait runs out: the
// kernel then drains its copies in flight, frees its tensor memory, returns,
// and the call reports TUPS_ERR_TIMEOUT; the launch after it runs normally.
extern "C" int tups_set_split_wait(long long cycles, int stall_test) {
  if (cycles < 0) return TUPS_ERR_BADARG;
  tups::g_oz_wait_cycles.store(cycles);
  tups::g_oz_stall_test.store(stall_test ? 1 : 0);
  return TUPS_OK;
}

extern "C" int tups_set_split_tile(int n_tile) {
  if (n_tile < 0 || n_tile > tups::OZ_MAX_NT || n_tile % 16) return TUPS_ERR_BADARG;
  tups::g_oz_n_tile.store(n_tile);
  return TUPS_OK;
}

// The split GEMM on CTA pairs (tcgen05 cta_group::2, M = 256 over two SMs)
// for row counts >= 256: 1 enables, 0 restores one CTA per 128-row tile.
// Both forms give the same bits.  Process-wide; no counterpart in the
// reference.
extern "C" int tups_set_split_cta_pairs(int enable) {
  tups::g_oz_pairs.store(enable ? 1 : 0);
  return TUPS_OK;
}
