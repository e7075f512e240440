// LU form of the Bethe-Salpeter equation in split precision with FP64
// iterative refinement, batched over instances of uneven size (no
// counterpart in the reference, whose BSE is the damped update of
// SRC/parquet_BSE.f90:72-128; this mode agrees with it at the fixed point):
//   F = (1 - c Gamma chi)^{-1} Gamma,   Phi = F - Gamma.
//
// Instances are grouped by size n and each group is solved in group-
// contiguous buffers:
//  * A = I - c Gamma chi (chi block-diagonal in nu, n^2 Nl per instance).
//  * Blocked right-looking LU with partial pivoting, blocks of 128 columns.
//    The block is factored in FP64 as two panels of 64 columns, one CTA per
//    instance each (lu_device.cuh), with the second panel's update over 32 x 32
//    tiles between them; the trailing update A22 -= L21 U12 (K = 128) runs on
//    the int8 tensor cores as an Ozaki split GEMM with s slices (ozaki.cu),
//    so the factors are those of a matrix within about 10^(1.1-2s) of A.
//  * X = U^{-1} L^{-1} P Gamma: 128-row diagonal blocks in FP64 (their 64 x 64
//    triangles by blocked substitution), the off-diagonal updates on the int8
//    path.
//  * Refinement: R = Gamma - A X = Gamma - X + c Gamma (chi X) in FP64 (the
//    GEMM on the FP64 tensor cores, three real products per complex one);
//    stop when max|R| <= tol max|Gamma| for every instance of the group (or
//    after max_refine corrections), else D = U^{-1} L^{-1} P R as above and
//    X += D.  Each correction multiplies the error by about
//    kappa(A) 10^(1.1-2s).
//
// Caller-owned workspace only (tups_bse_lu_split_workspace bytes).
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <vector>

#include "lu_device.cuh"
#include "tups_device.cuh"
#include "zgemm_tile.cuh"

namespace tups {
namespace {

constexpr int LS_NB = 128;      // block of the split-precision updates
constexpr int LS_THREADS = 256;
constexpr int LS_EPI_SUB = 2;   // OzRun::epi: C -= A B

struct LsDesc {
  long long g_off;  // complex offset of Gamma_i / out_i in the caller's packed arrays
  long long c_off;  // complex offset of chi_i
  int nl;
  double scale;     // c
};

__device__ __forceinline__ void atomic_max_nonneg(unsigned long long* a, double v) {
  // non-negative doubles order like their bit patterns
  atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

__device__ double block_max(double v) {
  __shared__ double red[LS_THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double m = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) m = fmax(m, red[w]);
  __syncthreads();
  return m;
}

// Gg = Gamma_i, Ag = I - c Gamma_i chi_i (sums over l1 ascending, as the
// FP64 LU form in lu.cu)
__global__ void __launch_bounds__(LS_THREADS) k_ls_form(const LsDesc* __restrict__ desc, const cplx* __restrict__ gamma,
                                                        const cplx* __restrict__ chi_all, cplx* __restrict__ Gg,
                                                        cplx* __restrict__ Ag, unsigned long long* gmax, int n) {
  const int i = blockIdx.y;
  const LsDesc d = desc[i];
  const int nl = d.nl, nf = n / nl;
  const size_t n2 = (size_t)n * n;
  const cplx* G = gamma + d.g_off;
  const cplx* chi = chi_all + d.c_off;
  double mx = 0.0;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n2; e += (size_t)gridDim.x * blockDim.x) {
    const int row = (int)(e % n), col = (int)(e / n);
    const int l2 = col / nf, nu = col % nf;
    cplx acc = cmk(0.0, 0.0);
    for (int l1 = 0; l1 < nl; l1++) acc = cfma(G[row + (size_t)n * (l1 * nf + nu)], chi[l1 + nl * (l2 + (size_t)nl * nu)], acc);
    const cplx g = G[e];
    Gg[n2 * i + e] = g;
    Ag[n2 * i + e] = cmk((row == col ? 1.0 : 0.0) - d.scale * acc.x, -d.scale * acc.y);
    mx = fmax(mx, fmax(fabs(g.x), fabs(g.y)));
  }
  mx = block_max(mx);
  if (threadIdx.x == 0) atomic_max_nonneg(&gmax[i], mx);
}

// ---- 128-column block ------------------------------------------------------------
using lud::BlockShared;
using lud::kBlock;
using lud::kPanelRows;
using lud::kPanelThreads;

constexpr int LS_LDT = kBlock + 2, LS_LDX = kBlock + 4;

struct LsPanelShared {
  BlockShared b;
  cplx t[kBlock * LS_LDT];  // [column][row] of L11
  cplx x[kBlock * LS_LDX];  // [column][row]: the block's columns right of the panel
};

// Columns [j0, j0 + 64) of the block [J0, JE), one CTA per instance: the panel
// with its interchanges on all the block's columns and for the first panel U12
// = L11^{-1} A12 of the block's other columns, a warp per 8 of them.
// worig[r]: the row whose content, as it stood before the block, row r now
// holds.  With the block's last panel the instance's whole permutation
// follows: perm'[r] = perm[worig[r]].  RPT as in block_factor.
template <int RPT>
__global__ void __launch_bounds__(kPanelThreads, 1) k_ls_panel(cplx* __restrict__ Ag, int* __restrict__ ipiv_all,
                                                               int* __restrict__ worig_all, int* __restrict__ wtmp_all,
                                                               int* __restrict__ perm_all, int* __restrict__ status,
                                                               int n, int j0, int J0, int JE) {
  extern __shared__ __align__(16) unsigned char smraw[];
  LsPanelShared& S = *reinterpret_cast<LsPanelShared*>(smraw);
  const int i = blockIdx.x, tid = threadIdx.x;
  const int jb = min(kBlock, JE - j0), je = j0 + jb;
  cplx* A = Ag + (size_t)n * n * i;
  int* worig = worig_all + (size_t)n * i;
  for (int r = j0 + tid; r < n; r += kPanelThreads) {
    const int o = j0 == J0 ? r : worig[r];
    if (RPT > 0) S.b.orig[r - j0] = o;
    else worig[r] = o;
  }
  __syncthreads();
  auto track = [&](int c, int p) {
    int* o = RPT > 0 ? S.b.orig - j0 : worig;
    const int x = o[c];
    o[c] = o[p];
    o[p] = x;
  };
  lud::block_factor<RPT, LS_NB>(A, n, j0, jb, J0, JE, ipiv_all + (size_t)n * i, &status[i], S.b, track);
  if (RPT > 0)
    for (int r = j0 + tid; r < n; r += kPanelThreads) worig[r] = S.b.orig[r - j0];
  if (je == JE) {
    int *perm = perm_all + (size_t)n * i, *tmp = wtmp_all + (size_t)n * i;
    __syncthreads();
    for (int r = J0 + tid; r < n; r += kPanelThreads) tmp[r] = J0 == 0 ? worig[r] : perm[worig[r]];
    __syncthreads();
    for (int r = J0 + tid; r < n; r += kPanelThreads) perm[r] = tmp[r];
    return;
  }
  const int warp = tid >> 5;
  for (int e = tid; e < kBlock * kBlock; e += kPanelThreads) {
    const int r = e % kBlock, c = e / kBlock;
    S.t[c * LS_LDT + r] = A[j0 + r + (size_t)n * (j0 + c)];
    S.x[c * LS_LDX + r] = je + c < JE ? A[j0 + r + (size_t)n * (je + c)] : cmk(0.0, 0.0);
  }
  __syncthreads();
  if (8 * warp < JE - je) lud::solve_triangle<false>(S.t, LS_LDT, nullptr, S.x + 8 * warp * LS_LDX, LS_LDX, kBlock);
  __syncthreads();
  for (int e = tid; e < kBlock * (JE - je); e += kPanelThreads) {
    const int r = e % kBlock, c = e / kBlock;
    A[j0 + r + (size_t)n * (je + c)] = S.x[c * LS_LDX + r];
  }
}

// A[j1.., j1..JE) -= A[j1.., J0..j1) A[J0..j1, j1..JE): the block's second panel;
// four real products per complex one, as the FP64 form's update (lu.cu)
using LsTile = ZgemmTile<1, 2, 2, 2, 16, 2, false, false>;

struct LsSource {
  static constexpr bool kGather = false;
  const cplx *l, *r;
  int n, K, n0;
  __device__ int ktiles() const { return (K + 15) / 16; }
  __device__ int depth(int kt) const { return min(16, K - 16 * kt); }
  __device__ size_t ldl() const { return (size_t)n; }
  __device__ const cplx* left(int kt) const { return l + (size_t)n * 16 * kt; }
  __device__ const cplx* right(int kt) const { return r + 16 * kt; }
  __device__ size_t roff(int c) const { return (size_t)n * (n0 + c); }
};

__global__ void __launch_bounds__(LsTile::NT, 5) k_ls_mid(cplx* __restrict__ Ag, int n, int J0, int j1, int JE) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx* A = Ag + (size_t)n * n * blockIdx.z;
  const int m0 = blockIdx.x * LsTile::BM, n0 = blockIdx.y * LsTile::BN, rows = n - j1 - m0, cols = JE - j1 - n0;
  LsTile t;
  t.run(LsSource{A + j1 + m0 + (size_t)n * J0, A + J0 + (size_t)n * j1, n, j1 - J0, n0}, reinterpret_cast<cplx*>(smraw),
        rows, cols);
  cplx* C = A + (j1 + m0) + (size_t)n * (j1 + n0);
  t.each(
      rows, cols, [&](int row, int col) { return C[row + (size_t)n * col]; },
      [&](int row, int col, cplx v, cplx c) { C[row + (size_t)n * col] = csub(c, v); });
}

// ---- solves with a 128-row diagonal block [j0, j0 + jb) on LT_COLS columns per CTA ----
// T is the block's unit lower (or, BACK, upper) triangle, in 64 x 64 parts: X =
// T^{-1} X is, lower, X1 = L11^{-1} X1, X2 -= L21 X1, X2 = L22^{-1} X2.  A warp
// takes 8 columns through all of it.
// ROWS: the columns of A outside the block first take the block's interchanges
// (worig), all reads of a tile before its first write; those left of the
// block take nothing else.
constexpr int LT_COLS = 32, LT_LDX = LS_NB + 4;
constexpr size_t kTriSmem = ((size_t)kBlock * LS_LDT + LT_COLS * LT_LDX + kBlock) * sizeof(cplx);
enum { TRI_ROWS = 0, TRI_FWD = 1, TRI_BACK = 2 };

__device__ __forceinline__ void ls_cp_async16(void* sdst, const void* gsrc, bool valid) {
  unsigned sz = valid ? 16u : 0u;
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gsrc), "r"(sz));
}

// one 64 x 64 part, A's rows row.. (nr of them) and columns col.. (nk): KIND 0
// unit lower, 1 upper: the tile's rows r0.. become T^{-1} of themselves; 2: minus
// the part times the tile's rows k0..
template <int KIND>
__device__ __forceinline__ void tri_stage(const cplx* __restrict__ A, int n, int row, int col, int nr, int nk, cplx* sL,
                                          cplx* sI, cplx* sX, int r0, int k0) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gid = lane >> 2, tig = lane & 3;
  __syncthreads();  // every warp is done with the part before
#pragma unroll 8
  for (int i = 0; i < kBlock * kBlock / 128; i++) {
    const int m = tid % kBlock, k = tid / kBlock + 2 * i;
    const bool in = m < nr && k < nk;
    ls_cp_async16(sL + k * LS_LDT + m, in ? A + row + m + (size_t)n * (col + k) : A, in);
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  cplx* X = sX + warp * 8 * LT_LDX;
  if (KIND == 1) {
    if (tid < kBlock) sI[tid] = lud::diagonal_reciprocal(sL[tid * LS_LDT + tid]);
    __syncthreads();
  }
  if (KIND < 2) {
    lud::solve_triangle<KIND == 1>(sL, LS_LDT, sI, X + r0, LT_LDX, nr);
    return;
  }
  double re[4][4], im[4][4];
  auto at = [&](int t, int e) { return X + (2 * tig + (e & 1)) * LT_LDX + r0 + 16 * t + gid + (e >= 2 ? 8 : 0); };
#pragma unroll
  for (int t = 0; t < 4; t++)
#pragma unroll
    for (int e = 0; e < 4; e++) {
      re[t][e] = at(t, e)->x;
      im[t][e] = at(t, e)->y;
    }
  const cplx* x = X + gid * LT_LDX + k0 + tig;
#pragma unroll 2
  for (int k8 = 0; k8 < kBlock; k8 += 8) {
    const double br[2] = {x[k8].x, x[k8 + 4].x}, bi[2] = {x[k8].y, x[k8 + 4].y};
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const cplx* l = sL + (k8 + tig) * LS_LDT + 16 * t + gid;
      const cplx a0 = l[0], a1 = l[8], a2 = l[4 * LS_LDT], a3 = l[4 * LS_LDT + 8];
      const double ar[4] = {-a0.x, -a1.x, -a2.x, -a3.x}, an[4] = {-a0.y, -a1.y, -a2.y, -a3.y};
      const double ai[4] = {a0.y, a1.y, a2.y, a3.y};
      lud::dmma8(re[t], ar, br);
      lud::dmma8(re[t], ai, bi);
      lud::dmma8(im[t], ar, bi);
      lud::dmma8(im[t], an, br);
    }
  }
#pragma unroll
  for (int t = 0; t < 4; t++)
#pragma unroll
    for (int e = 0; e < 4; e++) *at(t, e) = cmk(re[t][e], im[t][e]);
  __syncwarp();
}

template <int MODE>
__global__ void __launch_bounds__(128, 1) k_ls_tri(const cplx* __restrict__ Ag, cplx* Xg, const int* __restrict__ worig_all,
                                                   int n, int j0, int jb) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int s_moved[LS_NB];
  __shared__ int s_cnt;
  cplx* sL = reinterpret_cast<cplx*>(smraw);  // [k][m]
  cplx* sX = sL + kBlock * LS_LDT;            // [column][row]
  cplx* sI = sX + LT_COLS * LT_LDX;
  const int i = blockIdx.y, tid = threadIdx.x, je = j0 + jb;
  const cplx* A = Ag + (size_t)n * n * i;
  cplx* X = Xg + (size_t)n * n * i;
  // ROWS: the columns are those of A outside the block, left ones first
  const int ncol = MODE == TRI_ROWS ? n - jb : n, c0 = blockIdx.x * LT_COLS;
  auto column = [&](int c) {
    return X + (size_t)n * (MODE == TRI_ROWS && c0 + c >= j0 ? c0 + c + jb : c0 + c);
  };
  const int nc = min(LT_COLS, ncol - c0);
  int src = j0 + tid;
  if (MODE == TRI_ROWS) {
    const int* worig = worig_all + (size_t)n * i;
    if (tid == 0) s_cnt = 0;
    __syncthreads();
    if (tid < jb) src = worig[j0 + tid];
    for (int r = je + tid; r < n; r += 128)
      if (worig[r] != r) s_moved[atomicAdd(&s_cnt, 1)] = r;
  }
#pragma unroll
  for (int c = 0; c < LT_COLS; c++) {
    const bool in = tid < jb && c < nc;
    ls_cp_async16(sX + c * LT_LDX + tid, in ? column(c) + src : X, in);
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  if (MODE == TRI_ROWS) {
    // rows below the block that take a block row: each interchange moves one
    const int cnt = s_cnt;
    cplx v[LT_COLS];
    const int dst = tid < cnt ? s_moved[tid] : 0;
    const int from = tid < cnt ? worig_all[(size_t)n * i + dst] : 0;
#pragma unroll
    for (int c = 0; c < LT_COLS; c++)
      if (tid < cnt && c < nc) v[c] = column(c)[from];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < LT_COLS; c++)
      if (tid < cnt && c < nc) column(c)[dst] = v[c];
  }
  // a tile of left columns only is done with the interchanges; a mixed one
  // solves all its columns and stores the right ones
  const bool solve = MODE != TRI_ROWS || c0 + nc > j0;
  const int b1 = min(jb, kBlock), b2 = jb - b1;
  if (MODE == TRI_ROWS && c0 < j0) {
#pragma unroll
    for (int c = 0; c < LT_COLS; c++)
      if (tid < jb && c < nc && c0 + c < j0) column(c)[j0 + tid] = sX[c * LT_LDX + tid];
  }
  if (!solve) return;
  if (MODE == TRI_BACK) {
    if (b2 > 0) {
      tri_stage<1>(A, n, j0 + kBlock, j0 + kBlock, b2, b2, sL, sI, sX, kBlock, kBlock);
      tri_stage<2>(A, n, j0, j0 + kBlock, b1, b2, sL, sI, sX, 0, kBlock);
    }
    tri_stage<1>(A, n, j0, j0, b1, b1, sL, sI, sX, 0, 0);
  } else {
    tri_stage<0>(A, n, j0, j0, b1, b1, sL, sI, sX, 0, 0);
    if (b2 > 0) {
      tri_stage<2>(A, n, j0 + kBlock, j0, b2, b1, sL, sI, sX, kBlock, 0);
      tri_stage<0>(A, n, j0 + kBlock, j0 + kBlock, b2, b2, sL, sI, sX, kBlock, kBlock);
    }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < LT_COLS; c++)
    if (tid < jb && c < nc && (MODE != TRI_ROWS || c0 + c >= j0)) column(c)[j0 + tid] = sX[c * LT_LDX + tid];
}

// X = A^{-1} Y for instances of up to lud::kSmall rows, a CTA each, factors and all
__global__ void __launch_bounds__(lud::kSmallThreads) k_ls_small(const cplx* __restrict__ Ag, const cplx* __restrict__ Yg,
                                                                 cplx* __restrict__ Xg, int* __restrict__ ipiv_all,
                                                                 int* __restrict__ status, int n) {
  __shared__ lud::SmallShared S;
  const size_t i = blockIdx.x, n2 = (size_t)n * n;
  lud::small_solve(Ag + n2 * i, Yg + n2 * i, Xg + n2 * i, n, ipiv_all + n * i, &status[i], S);
}

// X = P Y: row r from row perm[r]
__global__ void __launch_bounds__(LS_THREADS) k_ls_gather(const cplx* __restrict__ Yg, const int* __restrict__ perm_all,
                                                          cplx* __restrict__ Xg, int n) {
  const int i = blockIdx.y;
  const size_t n2 = (size_t)n * n;
  const int* perm = perm_all + (size_t)n * i;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n2; e += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(e % n);
    Xg[n2 * i + e] = Yg[n2 * i + (e - r) + perm[r]];
  }
}

// Y = chi X (chi block-diagonal in nu, sums over l2 ascending)
__global__ void __launch_bounds__(LS_THREADS) k_ls_chimul(const LsDesc* __restrict__ desc, const cplx* __restrict__ chi_all,
                                                          const cplx* __restrict__ Xg, cplx* __restrict__ Yg, int n) {
  const int i = blockIdx.y;
  const LsDesc d = desc[i];
  const int nl = d.nl, nf = n / nl;
  const size_t n2 = (size_t)n * n;
  const cplx* chi = chi_all + d.c_off;
  const cplx* X = Xg + n2 * i;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n2; e += (size_t)gridDim.x * blockDim.x) {
    const int row = (int)(e % n), col = (int)(e / n);
    const int l1 = row / nf, nu = row % nf;
    cplx acc = cmk(0.0, 0.0);
    for (int l2 = 0; l2 < nl; l2++) acc = cfma(chi[l1 + nl * (l2 + (size_t)nl * nu)], X[(l2 * nf + nu) + (size_t)n * col], acc);
    Yg[n2 * i + e] = acc;
  }
}

// R = Gamma - X + c Gamma Y on the FP64 tensor cores (the BSE GEMM's tile)
using RsTile = ZgemmTile<1, 2, 2, 2, 16, 3, true>;

__global__ void __launch_bounds__(RsTile::NT, 3) k_ls_resid(const LsDesc* __restrict__ desc, const cplx* __restrict__ Gg,
                                                            const cplx* __restrict__ Yg, const cplx* __restrict__ Xg,
                                                            cplx* __restrict__ Rg, unsigned long long* rmax, int n) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int i = blockIdx.y;
  const size_t n2 = (size_t)n * n;
  const cplx *G = Gg + n2 * i, *X = Xg + n2 * i;
  cplx* R = Rg + n2 * i;
  const int tiles_m = (n + RsTile::BM - 1) / RsTile::BM;
  const int m0 = (int)(blockIdx.x % tiles_m) * RsTile::BM, n0 = (int)(blockIdx.x / tiles_m) * RsTile::BN;
  RsTile t;
  t.run(LsSource{G + m0, Yg + n2 * i, n, n, n0}, reinterpret_cast<cplx*>(smraw), n - m0, n - n0);
  const double s = desc[i].scale;
  double mx = 0.0;
  const auto at = [&](int row, int col) { return (m0 + row) + (size_t)n * (n0 + col); };
  t.each(
      n - m0, n - n0, [&](int row, int col) { return ZgPair{G[at(row, col)], X[at(row, col)]}; },
      [&](int row, int col, cplx c, const ZgPair& in) {
        const cplx v = cmk((in.a.x - in.b.x) + s * c.x, (in.a.y - in.b.y) + s * c.y);
        R[at(row, col)] = v;
        mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
      });
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(&rmax[i], mx);
}

// X += D
__global__ void __launch_bounds__(LS_THREADS) k_ls_update(cplx* __restrict__ Xg, const cplx* __restrict__ Dg, int n) {
  const int i = blockIdx.y;
  const size_t n2 = (size_t)n * n;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n2; e += (size_t)gridDim.x * blockDim.x)
    Xg[n2 * i + e] = cadd(Xg[n2 * i + e], Dg[n2 * i + e]);
}

// out_i = X_i (want_phi: X_i - Gamma_i) at the instance's place in the caller's layout
__global__ void __launch_bounds__(LS_THREADS) k_ls_scatter(const LsDesc* __restrict__ desc, const cplx* __restrict__ Xg,
                                                           const cplx* __restrict__ Gg, cplx* __restrict__ out, int n,
                                                           int want_phi) {
  const int i = blockIdx.y;
  const size_t n2 = (size_t)n * n;
  cplx* o = out + desc[i].g_off;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n2; e += (size_t)gridDim.x * blockDim.x) {
    cplx v = Xg[n2 * i + e];
    if (want_phi) v = csub(v, Gg[n2 * i + e]);
    o[e] = v;
  }
}

// ---- host side ------------------------------------------------------------------------
size_t up256(size_t x) { return (x + 255) / 256 * 256; }

struct LsLayout {
  size_t mat, ipiv, desc, norms, status, oz, total;
};

LsLayout ls_layout(int b, int n, int slices) {
  LsLayout L;
  L.mat = up256((size_t)b * n * n * sizeof(cplx));
  L.ipiv = up256((size_t)4 * b * n * sizeof(int));  // pivots, block map, scratch, permutation
  L.desc = up256((size_t)b * sizeof(LsDesc));
  L.norms = up256((size_t)2 * b * sizeof(unsigned long long));  // max|R_i|, max|Gamma_i|
  L.status = up256((size_t)b * sizeof(int) + sizeof(double));
  L.oz = up256(oz_work_layout(b, n, n, std::min(LS_NB, n), slices).total + 256);
  L.total = 5 * L.mat + L.ipiv + L.desc + L.norms + L.status + L.oz + 256;
  return L;
}

// instances by size, largest first
std::map<int, std::vector<int>, std::greater<int>> ls_groups(int n_inst, const int* n) {
  std::map<int, std::vector<int>, std::greater<int>> g;
  for (int i = 0; i < n_inst; i++) g[n[i]].push_back(i);
  return g;
}

int ls_gemm_sub(cudaStream_t st, void* ozw, int b, int M, int N, int K, const cplx* A, int lda, const cplx* B,
                int ldb, cplx* C, int ldc, long long stride, int s, double* ozstat, long long* launches) {
  OzRun R;
  R.batch = b;
  R.M = M;
  R.N = N;
  R.s = s;
  R.A.p1 = A;
  R.A.s1 = stride;
  R.A.ld1 = lda;
  R.A.K1 = K;
  R.B.p1 = B;
  R.B.s1 = stride;
  R.B.ld1 = ldb;
  R.B.K1 = K;
  oz_bind_work(R, oz_work_layout(b, M, N, K, s), ozw);
  R.status = ozstat;
  R.status_code = 1.0;
  R.epi = LS_EPI_SUB;
  R.C = C;
  R.ldc = ldc;
  R.c_stride = stride;
  return oz_run(R, st, launches);
}

// X = U^{-1} L^{-1} P Y for every instance of the group
int ls_solve(cudaStream_t st, const cplx* Ag, const cplx* Yg, cplx* Xg, const int* perm, void* ozw, int b, int n, int s,
             double* ozstat, long long* launches) {
  const long long n2 = (long long)n * n;
  const dim3 eg((unsigned)std::min<size_t>(((size_t)n * n + LS_THREADS - 1) / LS_THREADS, 512), b);
  const dim3 tg((n + LT_COLS - 1) / LT_COLS, b);
  k_ls_gather<<<eg, LS_THREADS, 0, st>>>(Yg, perm, Xg, n);
  (*launches)++;
  for (int j0 = 0; j0 < n; j0 += LS_NB) {
    const int jb = std::min(LS_NB, n - j0), je = j0 + jb;
    k_ls_tri<TRI_FWD><<<tg, 128, kTriSmem, st>>>(Ag, Xg, nullptr, n, j0, jb);
    (*launches)++;
    if (je < n) {
      int rc = ls_gemm_sub(st, ozw, b, n - je, n, jb, Ag + je + (size_t)n * j0, n, Xg + j0, n, Xg + je, n, n2, s,
                           ozstat, launches);
      if (rc) return rc;
    }
  }
  const int nblk = (n + LS_NB - 1) / LS_NB;
  for (int bk = nblk - 1; bk >= 0; bk--) {
    const int j0 = bk * LS_NB, jb = std::min(LS_NB, n - j0);
    k_ls_tri<TRI_BACK><<<tg, 128, kTriSmem, st>>>(Ag, Xg, nullptr, n, j0, jb);
    (*launches)++;
    if (j0 > 0) {
      int rc = ls_gemm_sub(st, ozw, b, j0, n, jb, Ag + (size_t)n * j0, n, Xg + j0, n, Xg, n, n2, s, ozstat, launches);
      if (rc) return rc;
    }
  }
  return cudaGetLastError() == cudaSuccess ? TUPS_OK : TUPS_ERR_CUDA;
}

// opt-in shared-memory sizes
bool ls_prepare() {
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  const int ps = (int)sizeof(LsPanelShared), ts = (int)kTriSmem;
  return cudaFuncSetAttribute(k_ls_panel<0>, attr, ps) == cudaSuccess &&
         cudaFuncSetAttribute(k_ls_panel<1>, attr, ps) == cudaSuccess &&
         cudaFuncSetAttribute(k_ls_panel<2>, attr, ps) == cudaSuccess &&
         cudaFuncSetAttribute(k_ls_tri<TRI_ROWS>, attr, ts) == cudaSuccess &&
         cudaFuncSetAttribute(k_ls_tri<TRI_FWD>, attr, ts) == cudaSuccess &&
         cudaFuncSetAttribute(k_ls_tri<TRI_BACK>, attr, ts) == cudaSuccess &&
         cudaFuncSetAttribute(k_ls_mid, attr, (int)LsTile::kSmem) == cudaSuccess &&
         cudaFuncSetAttribute(k_ls_resid, attr, (int)RsTile::kSmem) == cudaSuccess;
}

}  // namespace
}  // namespace tups

extern "C" size_t tups_bse_lu_split_workspace(int n_inst, const int* n, int slices) {
  using namespace tups;
  if (n_inst < 1 || !n || slices < 2 || slices > 8) return 0;
  size_t best = 0;
  for (const auto& kv : ls_groups(n_inst, n)) {
    if (kv.first < 1) return 0;
    best = std::max(best, ls_layout((int)kv.second.size(), kv.first, slices).total);
  }
  return best;
}

extern "C" int tups_bse_lu_split_batched(int n_inst, const int* n, const int* nl, const double* scale,
                                         const double* gamma, const double* chi, double* out, int want_phi,
                                         int slices, double tol, int max_refine, void* work, size_t work_bytes,
                                         int* refinements, double* residual, int* status, void* stream) {
  using namespace tups;
  if (n_inst < 1 || !n || !nl || !scale || !gamma || !chi || !out || !work) return TUPS_ERR_BADARG;
  if (slices < 2 || slices > 8 || max_refine < 0 || !(tol > 0.0)) return TUPS_ERR_BADARG;
  if (work_bytes < tups_bse_lu_split_workspace(n_inst, n, slices)) return TUPS_ERR_BADARG;
  std::vector<long long> goff(n_inst), coff(n_inst);
  long long go = 0, co = 0;
  for (int i = 0; i < n_inst; i++) {
    if (n[i] < 1 || nl[i] < 1 || n[i] % nl[i]) return TUPS_ERR_BADDIM;
    goff[i] = go;
    coff[i] = co;
    go += (long long)n[i] * n[i];
    co += (long long)nl[i] * nl[i] * (n[i] / nl[i]);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  (void)cudaGetLastError();
  if (!ls_prepare()) {
    (void)cudaGetLastError();
    return TUPS_ERR_CUDA;
  }
  long long launches = 0;
  const cplx* G = reinterpret_cast<const cplx*>(gamma);
  const cplx* CH = reinterpret_cast<const cplx*>(chi);
  cplx* OUT = reinterpret_cast<cplx*>(out);
  for (const auto& kv : ls_groups(n_inst, n)) {
    const int nn = kv.first;
    const std::vector<int>& idx = kv.second;
    const int b = (int)idx.size();
    const LsLayout L = ls_layout(b, nn, slices);
    uint8_t* p = (uint8_t*)(((uintptr_t)work + 255) & ~(uintptr_t)255);
    cplx* Gg = (cplx*)p;
    cplx* Ag = (cplx*)(p + L.mat);
    cplx* Xg = (cplx*)(p + 2 * L.mat);
    cplx* Rg = (cplx*)(p + 3 * L.mat);
    cplx* Yg = (cplx*)(p + 4 * L.mat);
    p += 5 * L.mat;
    int* ipiv = (int*)p;
    int *worig = ipiv + (size_t)b * nn, *wtmp = worig + (size_t)b * nn, *perm = wtmp + (size_t)b * nn;
    p += L.ipiv;
    LsDesc* desc = (LsDesc*)p;
    p += L.desc;
    unsigned long long* norms = (unsigned long long*)p;  // max|R_i| [b], max|Gamma_i| [b]
    p += L.norms;
    int* stat = (int*)p;
    double* ozstat = (double*)(((uintptr_t)(stat + b) + 7) & ~(uintptr_t)7);
    p += L.status;
    void* ozw = p;
    std::vector<LsDesc> hd(b);
    for (int k = 0; k < b; k++) hd[k] = {goff[idx[k]], coff[idx[k]], nl[idx[k]], scale[idx[k]]};
    if (cudaMemcpyAsync(desc, hd.data(), b * sizeof(LsDesc), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemsetAsync(stat, 0, L.status, st) != cudaSuccess) {
      cudaGetLastError();
      return TUPS_ERR_CUDA;
    }
    const size_t n2 = (size_t)nn * nn;
    const dim3 eg((unsigned)std::min<size_t>((n2 + LS_THREADS - 1) / LS_THREADS, 512), b);
    if (cudaMemsetAsync(norms, 0, 2 * b * sizeof(unsigned long long), st) != cudaSuccess) return TUPS_ERR_CUDA;
    k_ls_form<<<eg, LS_THREADS, 0, st>>>(desc, G, CH, Gg, Ag, norms + b, nn);
    // X = A^{-1} Y; small instances factor A in the same kernel each time
    const bool small = nn <= lud::kSmall;
    const auto solve = [&](const cplx* Y, cplx* X) {
      if (!small) return ls_solve(st, Ag, Y, X, perm, ozw, b, nn, slices, ozstat, &launches);
      k_ls_small<<<b, lud::kSmallThreads, 0, st>>>(Ag, Y, X, ipiv, stat, nn);
      return cudaGetLastError() == cudaSuccess ? TUPS_OK : TUPS_ERR_CUDA;
    };
    // P A = L U
    for (int j0 = 0; !small && j0 < nn; j0 += LS_NB) {
      const int jb = std::min(LS_NB, nn - j0), je = j0 + jb;
      for (int h0 = j0; h0 < je; h0 += kBlock) {
        const int rows = nn - h0;
        if (h0 > j0)
          k_ls_mid<<<dim3((rows + LsTile::BM - 1) / LsTile::BM, (je - h0 + LsTile::BN - 1) / LsTile::BN, b), LsTile::NT,
                     LsTile::kSmem, st>>>(Ag, nn, j0, h0, je);
        const auto panel = rows <= kPanelThreads ? k_ls_panel<1> : rows <= kPanelRows ? k_ls_panel<2> : k_ls_panel<0>;
        panel<<<b, kPanelThreads, sizeof(LsPanelShared), st>>>(Ag, ipiv, worig, wtmp, perm, stat, nn, h0, j0, je);
      }
      if (jb < nn)
        k_ls_tri<TRI_ROWS><<<dim3((nn - jb + LT_COLS - 1) / LT_COLS, b), 128, kTriSmem, st>>>(Ag, Ag, worig, nn, j0, jb);
      if (je < nn) {
        int rc = ls_gemm_sub(st, ozw, b, nn - je, nn - je, jb, Ag + je + (size_t)nn * j0, nn, Ag + j0 + (size_t)nn * je,
                             nn, Ag + je + (size_t)nn * je, nn, (long long)n2, slices, ozstat, &launches);
        if (rc) return rc;
      }
    }
    if (cudaGetLastError() != cudaSuccess) return TUPS_ERR_CUDA;
    int rc = solve(Gg, Xg);
    if (rc) return rc;
    // refinement: residual in FP64; stop once max|R_i| <= tol max|Gamma_i| for
    // every instance of the group, else correct with the split-precision factors
    int steps = 0;
    const int tiles = ((nn + RsTile::BM - 1) / RsTile::BM) * ((nn + RsTile::BN - 1) / RsTile::BN);
    std::vector<unsigned long long> hn(2 * b);
    std::vector<double> rel(b, 0.0);
    for (;;) {
      if (cudaMemsetAsync(norms, 0, b * sizeof(unsigned long long), st) != cudaSuccess) return TUPS_ERR_CUDA;
      k_ls_chimul<<<eg, LS_THREADS, 0, st>>>(desc, CH, Xg, Yg, nn);
      k_ls_resid<<<dim3(tiles, b), RsTile::NT, RsTile::kSmem, st>>>(desc, Gg, Yg, Xg, Rg, norms, nn);
      if (cudaGetLastError() != cudaSuccess) return TUPS_ERR_CUDA;
      if (cudaMemcpyAsync(hn.data(), norms, 2 * b * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st) !=
              cudaSuccess ||
          cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return TUPS_ERR_CUDA;
      }
      double worst = 0.0;
      for (int k = 0; k < b; k++) {
        double rm, gm;
        std::memcpy(&rm, &hn[k], sizeof(double));
        std::memcpy(&gm, &hn[b + k], sizeof(double));
        rel[k] = gm > 0.0 ? rm / gm : rm;
        worst = std::max(worst, rel[k]);
      }
      if (worst <= tol || steps >= max_refine) break;
      rc = solve(Rg, Yg);
      if (rc) return rc;
      k_ls_update<<<eg, LS_THREADS, 0, st>>>(Xg, Yg, nn);
      steps++;
    }
    k_ls_scatter<<<eg, LS_THREADS, 0, st>>>(desc, Xg, Gg, OUT, nn, want_phi);
    std::vector<int> hs(b);
    double ozflag = 0.0;
    if (cudaMemcpyAsync(hs.data(), stat, b * sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(&ozflag, ozstat, sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      cudaGetLastError();
      return TUPS_ERR_CUDA;
    }
    for (int k = 0; k < b; k++) {
      if (status) status[idx[k]] = hs[k];
      if (refinements) refinements[idx[k]] = steps;
      if (residual) residual[idx[k]] = rel[k];
    }
    if (ozflag != 0.0) return TUPS_ERR_TIMEOUT;
  }
  return TUPS_OK;
}
