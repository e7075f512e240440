// Device pieces shared by the batched LU kernels (lu.cu, lu_split.cu):
// the factorisation of a block of 64 columns by one CTA as two 32-column
// panels, and the inversion of its 64 x 64 triangles.
#pragma once

#include "tups_device.cuh"

namespace tups {
namespace lud {

static __device__ __forceinline__ double cabs1(cplx a) { return fabs(a.x) + fabs(a.y); }

static __device__ __forceinline__ void dmma8(double* c, const double* a, const double* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// ---- factorisation of one panel of up to 32 columns by one CTA -----------------
//
// Partial pivoting (largest |re| + |im|, lowest row on ties, a column of NaNs
// keeps its own row) in sub-panels of kPanelSub columns.  A thread owns the
// sub-panel's entries of its rows in registers, so a column costs one block
// argmax, one exchange of two rows through shared memory and register FMAs:
// two barriers and no pass over the column in global memory.  The sub-panels
// left of it are applied when a sub-panel is loaded (left-looking: L is read,
// nothing but the sub-panel itself is written).
constexpr int kPanelThreads = 512;
constexpr int kPanelCols = 32;
constexpr int kPanelSub = 8;
constexpr int kPanelRows = 2 * kPanelThreads;  // rows that fit the registers

struct PanelShared {
  cplx l[kPanelCols][kPanelCols + 1];  // [column][row] of the unit lower factor of the rows above
  cplx u[kPanelCols][kPanelSub];   // U rows of the sub-panel's columns above it
  cplx prow[kPanelSub], crow[kPanelSub];
  cplx inv;
  unsigned hi[kPanelThreads / 32], lo[kPanelThreads / 32];
  int row[kPanelThreads / 32];
  int piv[kPanelSub];
  int loc[kPanelRows];             // where a row's content stood before the sub-panel
};

// acc - a b, two dependent FMAs per part
static __device__ __forceinline__ cplx cfnma(cplx a, cplx b, cplx acc) {
  acc.x = fma(-a.x, b.x, acc.x);
  acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(-a.x, b.y, acc.y);
  acc.y = fma(-a.y, b.x, acc.y);
  return acc;
}

// 1/z with one reciprocal
static __device__ __forceinline__ cplx crecip1(cplx z) {
  const double q = __drcp_rn(z.x * z.x + z.y * z.y);
  return cmk(z.x * q, -z.y * q);
}

// larger |re| + |im| <=> larger key; NaN below every number
static __device__ __forceinline__ unsigned long long pivot_key(cplx a) {
  const double v = cabs1(a);
  return v >= 0.0 ? (unsigned long long)__double_as_longlong(v) + 1ull : 0ull;
}

// argmax over the warp of (key, lowest row); row = INT_MAX where a lane has none
static __device__ __forceinline__ void warp_argmax(unsigned& hi, unsigned& lo, int& row) {
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const bool a = hi == mh;
  const unsigned ml = __reduce_max_sync(0xffffffffu, a ? lo : 0u);
  row = __reduce_min_sync(0xffffffffu, a && lo == ml ? row : 0x7fffffff);
  hi = mh;
  lo = ml;
}

// Rows [h0, n), columns [h0, h0 + kb), kb <= 32; ipiv[c] = pivot row of column
// c.  Interchanges are applied to the columns [ca, cb) of the enclosing block
// and, through track(c, p), recorded by the caller.  n - h0 <= RPT * 512.
// `loc` holds the identity on entry and on return.
template <int RPT, int COLS, class Track>
static __device__ void panel_factor(cplx* __restrict__ A, int n, int h0, int kb, int ca, int cb, int* __restrict__ ipiv,
                                    int* __restrict__ status, PanelShared& S, Track track) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int p0 = 0; p0 < kb; p0 += kPanelSub) {
    const int jj = h0 + p0, w = min(kPanelSub, kb - p0);
    cplx a[RPT][kPanelSub];
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      const int r = h0 + tid + i * kPanelThreads;
#pragma unroll
      for (int k = 0; k < kPanelSub; k++)
        a[i][k] = (r < n && k < w) ? A[r + (size_t)n * (jj + k)] : cmk(0.0, 0.0);
    }
    if (p0 > 0) {
      // U rows above the sub-panel (rows h0 .. jj-1, held by warp 0): a warp
      // per column, lanes over rows, L from shared memory
      for (int e = tid; e < p0 * kPanelCols; e += kPanelThreads) {
        const int r = e % kPanelCols, t = e / kPanelCols;
        S.l[t][r] = r < p0 ? A[h0 + r + (size_t)n * (h0 + t)] : cmk(0.0, 0.0);
      }
      if (tid < p0)
#pragma unroll
        for (int k = 0; k < kPanelSub; k++) S.u[tid][k] = a[0][k];
      __syncthreads();
      if (warp < kPanelSub) {
        cplx x = S.u[lane][warp];
        for (int t = 0; t < p0 - 1; t++) {
          const cplx xt = cmk(__shfl_sync(0xffffffffu, x.x, t), __shfl_sync(0xffffffffu, x.y, t));
          if (lane > t && lane < p0) x = cfnma(S.l[t][lane], xt, x);
        }
        if (lane < p0) S.u[lane][warp] = x;
      }
      __syncthreads();
      if (tid < p0)
#pragma unroll
        for (int k = 0; k < kPanelSub; k++) a[0][k] = S.u[tid][k];
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        const int r = h0 + tid + i * kPanelThreads;
        if (r >= jj && r < n) {
          cplx l[kPanelSub], m[kPanelSub];
#pragma unroll
          for (int x = 0; x < kPanelSub; x++) l[x] = A[r + (size_t)n * (h0 + x)];
          for (int t = 0; t < p0; t += kPanelSub) {
            if (t + kPanelSub < p0)
#pragma unroll
              for (int x = 0; x < kPanelSub; x++) m[x] = A[r + (size_t)n * (h0 + t + kPanelSub + x)];
#pragma unroll
            for (int x = 0; x < kPanelSub; x++)
#pragma unroll
              for (int k = 0; k < kPanelSub; k++) a[i][k] = cfnma(l[x], S.u[t + x][k], a[i][k]);
#pragma unroll
            for (int x = 0; x < kPanelSub; x++) l[x] = m[x];
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < kPanelSub; c++) {
      if (c >= w) break;
      const int col = jj + c;
      unsigned long long key = 0;
      int row = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        const int r = h0 + tid + i * kPanelThreads;
        if (r >= col && r < n) {
          const unsigned long long v = pivot_key(a[i][c]);
          if (row == 0x7fffffff || v > key) {
            key = v;
            row = r;
          }
        }
      }
      unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
      warp_argmax(hi, lo, row);
      if (lane == 0) {
        S.hi[warp] = hi;
        S.lo[warp] = lo;
        S.row[warp] = row;
      }
      __syncthreads();
      const bool has = lane < kPanelThreads / 32;
      hi = has ? S.hi[lane] : 0u;
      lo = has ? S.lo[lane] : 0u;
      row = has ? S.row[lane] : 0x7fffffff;
      warp_argmax(hi, lo, row);
      const int p = row;
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        const int r = h0 + tid + i * kPanelThreads;
        if (r == p) {
#pragma unroll
          for (int k = 0; k < kPanelSub; k++) S.prow[k] = a[i][k];
          const bool zero = hi == 0u && lo == 1u;  // the key of 0.0
          S.inv = zero ? cmk(0.0, 0.0) : crecip1(a[i][c]);
          if (zero && *status == 0) *status = col + 1;
          S.piv[c] = p;
          ipiv[col] = p;
        }
        if (r == col) {
#pragma unroll
          for (int k = 0; k < kPanelSub; k++) S.crow[k] = a[i][k];
        }
      }
      if (tid == kPanelThreads - 1 && p != col) {
        const int x = S.loc[col - h0];
        S.loc[col - h0] = S.loc[p - h0];
        S.loc[p - h0] = x;
        track(col, p);
      }
      __syncthreads();
      const cplx inv = S.inv;
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        const int r = h0 + tid + i * kPanelThreads;
        if (p != col) {
          if (r == p)
#pragma unroll
            for (int k = 0; k < kPanelSub; k++) a[i][k] = S.crow[k];
          if (r == col)
#pragma unroll
            for (int k = 0; k < kPanelSub; k++) a[i][k] = S.prow[k];
        }
        if (r > col) {
          const cplx l = cmul(a[i][c], inv);
          a[i][c] = l;
#pragma unroll
          for (int k = c + 1; k < kPanelSub; k++) a[i][k] = cfnma(l, S.prow[k], a[i][k]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      const int r = h0 + tid + i * kPanelThreads;
#pragma unroll
      for (int k = 0; k < kPanelSub; k++)
        if (r < n && k < w) A[r + (size_t)n * (jj + k)] = a[i][k];
    }
    __syncthreads();
    // the sub-panel's interchanges on the block's other columns: its w rows
    // and their pivots, each from where its content stood (a row named twice
    // gets the same value twice)
    const int ncol = cb - ca - w;
    constexpr int kMove = 2 * kPanelSub, kMaxMove = (kMove * COLS + kPanelThreads - 1) / kPanelThreads;
    cplx v[kMaxMove];
    const int ms = tid % kMove, mk = ms % kPanelSub;  // this thread's row of the exchange
    const int mdst = mk >= w ? h0 : ms < kPanelSub ? jj + mk : S.piv[mk];
    const int msrc = h0 + S.loc[mdst - h0];
#pragma unroll
    for (int m = 0; m < kMaxMove; m++) {
      const int x = (tid + m * kPanelThreads) / kMove, col = ca + x < jj ? ca + x : ca + x + w;
      if (mk < w && x < ncol) v[m] = A[msrc + (size_t)n * col];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < kMaxMove; m++) {
      const int x = (tid + m * kPanelThreads) / kMove, col = ca + x < jj ? ca + x : ca + x + w;
      if (mk < w && x < ncol) A[mdst + (size_t)n * col] = v[m];
    }
    __syncthreads();
    if (tid < kMove && mk < w) S.loc[mdst - h0] = mdst - h0;
    __syncthreads();
  }
}

// Columns [h0, h0 + kb) after the 32 columns [j0, h0) left of them are
// factored: rows j0 .. h0-1 by forward substitution (a warp per column pair,
// lanes over rows), then the rows below, 16 x 32 warp tiles on the FP64 tensor
// cores with the substituted rows in shared memory.
struct HalfShared {
  cplx l[kPanelCols][kPanelCols + 1];  // [column][row]
  cplx b[kPanelCols][kPanelCols + 4];  // [column][k]
};

static __device__ void panel_half(cplx* __restrict__ A, int n, int j0, int kb, HalfShared& S) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h0 = j0 + kPanelCols;
  const int gid = lane >> 2, tig = lane & 3;
  for (int e = tid; e < kPanelCols * kPanelCols; e += kPanelThreads) {
    const int r = e % kPanelCols, t = e / kPanelCols;
    S.l[t][r] = A[j0 + r + (size_t)n * (j0 + t)];
  }
  constexpr int kWarps = kPanelThreads / 32, kPer = kPanelCols / kWarps;
  cplx x[kPer];
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const int c = warp + i * kWarps;
    x[i] = c < kb ? A[j0 + lane + (size_t)n * (h0 + c)] : cmk(0.0, 0.0);
  }
  __syncthreads();
  for (int t = 0; t < kPanelCols - 1; t++) {
    const cplx l = S.l[t][lane];
#pragma unroll
    for (int i = 0; i < kPer; i++) {
      const cplx xt = cmk(__shfl_sync(0xffffffffu, x[i].x, t), __shfl_sync(0xffffffffu, x[i].y, t));
      if (lane > t) x[i] = cfnma(l, xt, x[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const int c = warp + i * kWarps;
    S.b[c][lane] = x[i];
    if (c < kb) A[j0 + lane + (size_t)n * (h0 + c)] = x[i];
  }
  __syncthreads();
  for (int r0 = h0 + warp * 16; r0 < n; r0 += kWarps * 16) {
    const int ra = r0 + gid, rb = ra + 8;
    double cre[4][4], cim[4][4];
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int r = e >= 2 ? rb : ra, c = j * 8 + 2 * tig + (e & 1);
        const cplx v = r < n && c < kb ? A[r + (size_t)n * (h0 + c)] : cmk(0.0, 0.0);
        cre[j][e] = v.x;
        cim[j][e] = v.y;
      }
    const cplx z = cmk(0.0, 0.0);
    cplx f[4], g[4];
    auto load = [&](cplx* d, int k8) {
      const size_t ca = (size_t)n * (j0 + k8 + tig), cb = ca + 4 * (size_t)n;
      d[0] = ra < n ? A[ra + ca] : z;
      d[1] = rb < n ? A[rb + ca] : z;
      d[2] = ra < n ? A[ra + cb] : z;
      d[3] = rb < n ? A[rb + cb] : z;
    };
    load(f, 0);
#pragma unroll
    for (int k8 = 0; k8 < kPanelCols; k8 += 8) {
      if (k8 + 8 < kPanelCols) load(g, k8 + 8);
      double are[4], aim[4], apos[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        are[e] = -f[e].x;  // C -= A B
        aim[e] = -f[e].y;
        apos[e] = f[e].y;
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const cplx w0 = S.b[j * 8 + gid][k8 + tig], w1 = S.b[j * 8 + gid][k8 + tig + 4];
        const double bre[2] = {w0.x, w1.x}, bim[2] = {w0.y, w1.y};
        dmma8(cre[j], are, bre);
        dmma8(cre[j], apos, bim);
        dmma8(cim[j], are, bim);
        dmma8(cim[j], aim, bre);
      }
#pragma unroll
      for (int e = 0; e < 4; e++) f[e] = g[e];
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int r = e >= 2 ? rb : ra, c = j * 8 + 2 * tig + (e & 1);
        if (r < n && c < kb) A[r + (size_t)n * (h0 + c)] = cmk(cre[j][e], cim[j][e]);
      }
  }
  __syncthreads();
}

// The same panel with its columns in global memory, for more rows than the
// registers hold (n - h0 > kPanelRows): a pass over the columns per step.
template <class Track>
static __device__ void panel_factor_global(cplx* __restrict__ A, int n, int h0, int kb, int ca, int cb,
                                           int* __restrict__ ipiv, int* __restrict__ status, PanelShared& S,
                                           Track track) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = kPanelThreads;
  for (int c = h0; c < h0 + kb; c++) {
    unsigned long long key = 0;
    int row = 0x7fffffff;
    for (int r = c + tid; r < n; r += nt) {
      const unsigned long long v = pivot_key(A[r + (size_t)n * c]);
      if (row == 0x7fffffff || v > key) {
        key = v;
        row = r;
      }
    }
    unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    warp_argmax(hi, lo, row);
    if (lane == 0) {
      S.hi[warp] = hi;
      S.lo[warp] = lo;
      S.row[warp] = row;
    }
    __syncthreads();
    const bool has = lane < kPanelThreads / 32;
    hi = has ? S.hi[lane] : 0u;
    lo = has ? S.lo[lane] : 0u;
    row = has ? S.row[lane] : 0x7fffffff;
    warp_argmax(hi, lo, row);
    const int p = row;
    const bool zero = hi == 0u && lo == 1u;
    const cplx inv = zero ? cmk(0.0, 0.0) : crecip1(A[p + (size_t)n * c]);
    __syncthreads();
    if (tid == 0) {
      ipiv[c] = p;
      if (zero && *status == 0) *status = c + 1;
      if (p != c) track(c, p);
    }
    if (p != c)
      for (int col = ca + tid; col < cb; col += nt) {
        const cplx t = A[c + (size_t)n * col];
        A[c + (size_t)n * col] = A[p + (size_t)n * col];
        A[p + (size_t)n * col] = t;
      }
    __syncthreads();
    for (int r = c + 1 + tid; r < n; r += nt) {
      const cplx l = cmul(A[r + (size_t)n * c], inv);
      A[r + (size_t)n * c] = l;
      for (int k = c + 1; k < h0 + kb; k++)
        A[r + (size_t)n * k] = cfnma(l, A[c + (size_t)n * k], A[r + (size_t)n * k]);
    }
    __syncthreads();
  }
}

// ---- one block of 64 columns by one CTA ------------------------------------------
constexpr int kBlock = 2 * kPanelCols, kInvLd = kBlock + 1;

struct BlockShared {
  PanelShared p;
  int orig[kPanelRows];  // where a row's content stood before the block
  union {
    HalfShared half;
    struct {
      cplx M[kBlock * kInvLd], T[kPanelCols * kPanelCols];  // [col][row]
    };
  };
};

// M <- M^{-1}, a 64 x 64 triangle (unit lower, or UP: upper) in shared memory
// with the pitch kInvLd: 16 x 16 diagonal blocks by substitution, one thread
// per column, then merged pairwise, inv([X 0; Y Z]) = [X' 0; -Z' Y X' Z'] and
// its mirror.  A zero pivot divides by one (its instance is reported
// singular).  T: 1024 complex of scratch.  At least 64 threads.
template <bool UP>
static __device__ void invert_triangle(cplx* __restrict__ M, cplx* __restrict__ T) {
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid < 64) {
    const int b = tid & 48, c = tid & 15;
    const cplx* D = M + b * kInvLd + b;
    cplx x[16];
#pragma unroll
    for (int r = 0; r < 16; r++) x[r] = cmk(r == c ? 1.0 : 0.0, 0.0);
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const int k = UP ? 15 - i : i;
      if (UP) {
        const cplx u = D[k * kInvLd + k];
        if (u.x != 0.0 || u.y != 0.0) x[k] = cmul(x[k], crecip1(u));
      }
#pragma unroll
      for (int r = 0; r < 16; r++)
        if (UP ? r < k : r > k) x[r] = cfnma(D[k * kInvLd + r], x[k], x[r]);
    }
    __syncwarp();  // a 16-column block belongs to half a warp
#pragma unroll
    for (int r = 0; r < 16; r++) M[(b + c) * kInvLd + b + r] = x[r];
  }
  __syncthreads();
  // Y is s x s; a warp per 16 x 8 tile of a product
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5, gid = lane >> 2, tig = lane & 3;
  auto product = [&](const cplx* L, int ldl, const cplx* R, int ldr, int s, int m0, int c0, double* re, double* im) {
    for (int k8 = 0; k8 < s; k8 += 8) {
      const cplx* l = L + (k8 + tig) * ldl + m0 + gid;
      const cplx* r = R + (c0 + gid) * ldr + k8 + tig;
      const cplx a0 = l[0], a1 = l[8], a2 = l[4 * ldl], a3 = l[4 * ldl + 8], b0 = r[0], b1 = r[4];
      const double ar[4] = {a0.x, a1.x, a2.x, a3.x}, ai[4] = {a0.y, a1.y, a2.y, a3.y};
      const double an[4] = {-a0.y, -a1.y, -a2.y, -a3.y}, br[2] = {b0.x, b1.x}, bi[2] = {b0.y, b1.y};
      dmma8(re, ar, br);
      dmma8(im, ar, bi);
      dmma8(re, an, bi);
      dmma8(im, ai, br);
    }
  };
  for (int s = 16; s < kBlock; s *= 2) {
    const int per = s / 16 * (s / 8), tiles = kBlock / (2 * s) * per;
    for (int pass = 0; pass < 2; pass++) {
      // pass 0: T = Y X' (lower) or Y Z' (upper); pass 1: Y = -Z' T or -X' T
      for (int t = warp; t < tiles; t += nw) {
        const int b = t / per * 2 * s, m0 = t % per % (s / 16) * 16, c0 = t % per / (s / 16) * 8;
        const int y0 = UP ? b : b + s, x0 = UP ? b + s : b;  // first row and column of Y
        cplx* Y = M + x0 * kInvLd + y0;
        cplx* Tp = T + t / per * s * s;  // [c][r]
        double re[4] = {}, im[4] = {};
        if (pass == 0) product(Y, kInvLd, M + x0 * kInvLd + x0, kInvLd, s, m0, c0, re, im);
        else product(M + y0 * kInvLd + y0, kInvLd, Tp, s, s, m0, c0, re, im);
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int r = m0 + gid + (e >= 2 ? 8 : 0), c = c0 + 2 * tig + (e & 1);
          if (pass == 0) Tp[c * s + r] = cmk(re[e], im[e]);
          else Y[c * kInvLd + r] = cmk(-re[e], -im[e]);
        }
      }
      __syncthreads();
    }
  }
}

// the triangle of the diagonal block at (j0, j0), identity past jb, into M
template <bool UP>
static __device__ void load_triangle(const cplx* __restrict__ A, int n, int j0, int jb, cplx* __restrict__ M) {
  for (int e = threadIdx.x; e < kBlock * kBlock; e += blockDim.x) {
    const int r = e % kBlock, c = e / kBlock;
    const bool in = r < jb && c < jb && (UP ? r <= c : r > c);
    M[c * kInvLd + r] = in ? A[j0 + r + (size_t)n * (j0 + c)] : cmk(r == c ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
}

template <bool UP>
static __device__ void store_triangle(cplx* __restrict__ A, int n, int j0, int jb, const cplx* __restrict__ M) {
  for (int e = threadIdx.x; e < kBlock * kBlock; e += blockDim.x) {
    const int r = e % kBlock, c = e / kBlock;
    if (r < jb && c < jb && (UP ? r <= c : r > c)) A[j0 + r + (size_t)n * (j0 + c)] = M[c * kInvLd + r];
  }
}


// Columns [j0, j0 + jb), jb <= 64, rows j0 .. n-1: two 32-column panels with a
// 32-wide update between them, then the unit lower diagonal factor replaced by
// its inverse (nothing later needs the factor).  RPT: rows per thread in
// registers, 0 = columns in global memory.  Interchanges as panel_factor's.
// Ends with a barrier.
template <int RPT, int COLS, class Track>
static __device__ void block_factor(cplx* __restrict__ A, int n, int j0, int jb, int ca, int cb, int* __restrict__ ipiv,
                                    int* __restrict__ status, BlockShared& S, Track track) {
  const int je = j0 + jb;
  for (int i = threadIdx.x; i < kPanelRows; i += kPanelThreads) S.p.loc[i] = i;
  __syncthreads();
  for (int h0 = j0; h0 < je; h0 += kPanelCols) {
    const int kb = min(kPanelCols, je - h0);
    if (h0 > j0) panel_half(A, n, j0, kb, S.half);
    if constexpr (RPT > 0) panel_factor<RPT, COLS>(A, n, h0, kb, ca, cb, ipiv, status, S.p, track);
    else panel_factor_global(A, n, h0, kb, ca, cb, ipiv, status, S.p, track);
  }
  load_triangle<false>(A, n, j0, jb, S.M);
  invert_triangle<false>(S.M, S.T);
  store_triangle<false>(A, n, j0, jb, S.M);
  __syncthreads();
}

}  // namespace lud
}  // namespace tups
