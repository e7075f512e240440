// Device pieces shared by the batched LU kernels (lu.cu, lu_split.cu):
// the factorisation of a block of 64 columns by one CTA as two 32-column
// panels, and the solves with its 64 x 64 triangles.
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

// 1/z with one reciprocal.  Where |z|^2 would leave the normal range, z is
// scaled by the power of two of its larger part first.
static __device__ __forceinline__ cplx crecip1(cplx z) {
  const double d = z.x * z.x + z.y * z.y;
  if (d > 1e-290 && d < 1e290) {
    const double q = __drcp_rn(d);
    return cmk(z.x * q, -z.y * q);
  }
  const int e = min(max(max(__double2hiint(fabs(z.x)), __double2hiint(fabs(z.y))) >> 20, 1), 2045);
  const double s = __hiloint2double((2046 - e) << 20, 0), x = z.x * s, y = z.y * s;
  const double q = __drcp_rn(x * x + y * y);
  return cmk(x * q * s, -y * q * s);
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
constexpr int kBlock = 2 * kPanelCols;

struct BlockShared {
  PanelShared p;
  int orig[kPanelRows];  // where a row's content stood before the block
  HalfShared half;
};

// Columns [j0, j0 + jb), jb <= 64, rows j0 .. n-1: two 32-column panels with a
// 32-wide update between them.  RPT: rows per thread in registers, 0 = columns
// in global memory.  Interchanges as panel_factor's.  Ends with a barrier.
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
}

// ---- solves with a 64 x 64 triangle ------------------------------------------------
//
// X <- T^{-1} X for one warp's 8 columns, `rows` <= 64 rows each in shared
// memory (column c at X + c ldx; the rest of the last 16 rows is zero): T, [column][row] with the pitch ldt, is unit lower
// (entries above and on the diagonal are not read) or, UP, upper with the
// reciprocals of its diagonal in inv.  Blocks of 16 rows: what the rows solved
// before contribute goes through the FP64 tensor cores (four real products per
// complex one), the block itself by substitution, four lanes per column with
// the rows interleaved over them.
//
// Products with explicit inverses of the triangles instead were faster (with
// three real products per complex one in the updates besides, 96 instances of
// n = 64..832 9.3 ms against 10.4), but their error grows with the triangle's
// condition: the residuals of well-conditioned systems were three to ten times
// those of substitution, a thousand units of |L| |U| |X| against eleven for rows
// that spread over twelve decades.
template <bool UP>
static __device__ __forceinline__ void solve_triangle(const cplx* __restrict__ T, int ldt, const cplx* __restrict__ inv,
                                                      cplx* X, int ldx, int rows) {
  const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3, nb = (rows + 15) / 16;
#pragma unroll 1
  for (int b = 0; b < nb; b++) {
    const int r0 = 16 * (UP ? nb - 1 - b : b);
    if (b > 0) {
      double re[4], im[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const cplx v = X[(2 * tig + (e & 1)) * ldx + r0 + gid + (e >= 2 ? 8 : 0)];
        re[e] = v.x;
        im[e] = v.y;
      }
      for (int k8 = UP ? r0 + 16 : 0; k8 < (UP ? 16 * nb : r0); k8 += 8) {
        const cplx* l = T + (k8 + tig) * ldt + r0 + gid;
        const cplx a0 = l[0], a1 = l[8], a2 = l[4 * ldt], a3 = l[4 * ldt + 8];
        const double ar[4] = {-a0.x, -a1.x, -a2.x, -a3.x}, an[4] = {-a0.y, -a1.y, -a2.y, -a3.y};
        const double ai[4] = {a0.y, a1.y, a2.y, a3.y};
        const cplx b0 = X[gid * ldx + k8 + tig], b1 = X[gid * ldx + k8 + tig + 4];
        const double br[2] = {b0.x, b1.x}, bi[2] = {b0.y, b1.y};
        dmma8(re, ar, br);
        dmma8(re, ai, bi);
        dmma8(im, ar, bi);
        dmma8(im, an, br);
      }
#pragma unroll
      for (int e = 0; e < 4; e++)
        X[(2 * tig + (e & 1)) * ldx + r0 + gid + (e >= 2 ? 8 : 0)] = cmk(re[e], im[e]);
      __syncwarp();
    }
    cplx x[4];
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = X[gid * ldx + r0 + tig + 4 * i];
#pragma unroll
    for (int c = 0; c < 16; c++) {
      const int k = UP ? 15 - c : c;
      cplx xk = cmk(__shfl_sync(0xffffffffu, x[k >> 2].x, (lane & ~3) | (k & 3)),
                    __shfl_sync(0xffffffffu, x[k >> 2].y, (lane & ~3) | (k & 3)));
      if (UP) {
        xk = cmul(xk, inv[r0 + k]);
        if (tig == (k & 3)) x[k >> 2] = xk;
      }
      const cplx* l = T + (r0 + k) * ldt + r0 + tig;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (UP ? i > k >> 2 : i < k >> 2) continue;
        const bool mine = i != k >> 2 || (UP ? tig < (k & 3) : tig > (k & 3));
        const cplx y = cfnma(l[4 * i], xk, x[i]);
        if (mine) x[i] = y;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) X[gid * ldx + r0 + tig + 4 * i] = x[i];
    __syncwarp();
  }
}

// ---- whole instances of up to 32 rows ------------------------------------------------
//
// X = A^{-1} Y by one CTA: [A | Y] in shared memory, columns with a lane per
// row, so a column step is one search by every warp on its own, one barrier,
// and a rank-1 update of the columns right of it that takes the interchange
// along; L is not kept.  Pivots, status and zero pivots as in panel_factor.
// X may be Y.  16384 instances of n = 5, 16, 32 (with the forming of A): 0.97,
// 2.7, 7.9 ms with one CTA per instance on global memory, 2.2, 3.2, 6.0 by blocks
// of 64 columns, 0.42, 0.95, 2.7 here.
constexpr int kSmall = 32, kSmallThreads = 128;

struct SmallShared {
  cplx m[2 * kSmall][kSmall + 1];  // [column][row]
  cplx inv[kSmall];                // reciprocals of U's diagonal, one for a zero
};

static __device__ void small_solve(const cplx* __restrict__ A, const cplx* Y, cplx* X, int n, int* __restrict__ ipiv,
                                   int* __restrict__ status, SmallShared& S) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarps = kSmallThreads / 32;
  for (int j = warp; j < 2 * n; j += kWarps)
    if (lane < n) S.m[j][lane] = j < n ? A[lane + (size_t)n * j] : Y[lane + (size_t)n * (j - n)];
  __syncthreads();
  const cplx zero = cmk(0.0, 0.0);
  for (int c = 0; c < n; c++) {
    cplx a = lane < n ? S.m[c][lane] : zero;
    const bool in = lane >= c && lane < n;
    const unsigned long long key = in ? pivot_key(a) : 0ull;
    unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    int p = in ? lane : 0x7fffffff;
    warp_argmax(hi, lo, p);
    const bool singular = hi == 0u && lo == 1u;  // the key of 0.0
    auto exchanged = [&](cplx v) {
      const int from = lane == c ? p : lane == p ? c : lane;
      return cmk(__shfl_sync(0xffffffffu, v.x, from), __shfl_sync(0xffffffffu, v.y, from));
    };
    a = exchanged(a);
    const cplx pv = cmk(__shfl_sync(0xffffffffu, a.x, c), __shfl_sync(0xffffffffu, a.y, c));
    const cplx inv = singular ? zero : crecip1(pv);
    const cplx l = lane > c ? cmul(a, inv) : zero;
    for (int j = c + 1 + warp; j < 2 * n; j += kWarps) {
      cplx x = exchanged(lane < n ? S.m[j][lane] : zero);
      const cplx u = cmk(__shfl_sync(0xffffffffu, x.x, c), __shfl_sync(0xffffffffu, x.y, c));
      if (lane > c) x = cfnma(l, u, x);
      if (lane < n) S.m[j][lane] = x;
    }
    if (threadIdx.x == 0) {
      ipiv[c] = p;
      S.inv[c] = singular ? cmk(1.0, 0.0) : inv;
      if (singular && *status == 0) *status = c + 1;
    }
    __syncthreads();
  }
  for (int j = n + warp; j < 2 * n; j += kWarps) {
    cplx x = lane < n ? S.m[j][lane] : zero;
    for (int c = n - 1; c >= 0; c--) {
      const cplx v = cmul(cmk(__shfl_sync(0xffffffffu, x.x, c), __shfl_sync(0xffffffffu, x.y, c)), S.inv[c]);
      if (lane == c) x = v;
      if (lane < c) x = cfnma(S.m[c][lane], v, x);
    }
    if (lane < n) X[lane + (size_t)n * (j - n)] = x;
  }
}

// reciprocal of a diagonal entry of U; a zero pivot divides by one (its
// instance is reported singular)
static __device__ __forceinline__ cplx diagonal_reciprocal(cplx u) {
  return u.x == 0.0 && u.y == 0.0 ? cmk(1.0, 0.0) : crecip1(u);
}

}  // namespace lud
}  // namespace tups
