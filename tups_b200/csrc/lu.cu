// LU form of the Bethe-Salpeter equation, batched over instances of uneven
// size (no counterpart in the reference, whose BSE is the damped update of
// SRC/parquet_BSE.f90:72-128; this mode agrees with it at the fixed point):
//   F = (1 - c Gamma chi)^{-1} Gamma,   Phi = F - Gamma,
// per (q, channel) instance with n = Nl*Nnu and chi block-diagonal in nu.
//
// Right-looking LU with partial pivoting of [A | Gamma], A = I - c Gamma chi,
// in blocks of 64 columns, every step one launch over all instances that
// still have a block:
//   k_lu_panel   one CTA per instance factors the block's columns,
//   k_lu_rows    column tiles: the block's row interchanges, then
//                U12 = L11^{-1} P A12 (and the same of the right-hand sides),
//   k_lu_update  32 x 32 tiles of [A22 | F2] -= L21 U12,
// then back substitution from each instance's last block:
//   k_lu_rows    X_b = U_bb^{-1} F_b,      k_lu_update   F_above -= U_above,b X_b.
// The forward substitution of the right-hand sides is part of the update, so
// rows of L left of the block are never interchanged.  The products run on the
// FP64 tensor cores.  One CTA per instance for the whole solve, which this
// replaces, left most SMs idle and its largest instance alone at the end.
// Instances of up to 32 rows take one kernel for all of it (k_lu_small).
//
// Caller-owned buffers only; the instance table and the interchange maps live
// in static device arrays.
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <vector>

#include "tups_device.cuh"
#include "lu_device.cuh"

namespace {

using tups::cplx;
using tups::cmk;
using tups::lud::dmma8;
using tups::lud::kPanelCols;
using tups::lud::kPanelRows;
using tups::lud::kPanelThreads;

constexpr int kLuMaxInst = 16384;
constexpr int NB = 2 * kPanelCols;  // 64

struct LuDesc {
  long long g_off;  // complex offset of Gamma_i / F_i / A_i (n^2 each)
  long long c_off;  // complex offset of chi_i (Nl*Nl*Nnu)
  long long p_off;  // int offset of the pivots (n)
  int n, nl;
  double scale;     // c
};

// the interchanges of one block as a gather: block row k takes row src[k];
// rows below the block that changed, (row << 6 | block row it takes)
struct LuMap {
  int src[NB];
  int moved[NB];
  int count;
};

__device__ LuDesc g_lu_desc[kLuMaxInst];
__device__ LuMap g_lu_map[kLuMaxInst];
__device__ int g_lu_status[kLuMaxInst];

// ---- A = I - c Gamma chi, F = Gamma ---------------------------------------------
// One thread per (row, nu) line: the line's nl entries of Gamma are loaded once
// (LMAX registers) and give its nl entries of A; the lanes run over rows at
// one nu, so a chi entry is one address per warp.  Sums over l1 ascending.
// LMAX = 0: any nl, the line re-read for every l2.
template <int LMAX>
__device__ void form_lines(const LuDesc& d, const cplx* __restrict__ G, const cplx* __restrict__ chi,
                           cplx* __restrict__ A, cplx* __restrict__ F) {
  const int n = d.n, nl = d.nl, nf = n / nl;
  const size_t lines = (size_t)n * nf;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < lines; t += (size_t)gridDim.x * blockDim.x) {
    const int row = (int)(t % n), nu = (int)(t / n);
    cplx g[LMAX > 0 ? LMAX : 1];
    if constexpr (LMAX > 0) {
#pragma unroll
      for (int l = 0; l < LMAX; l++)
        if (l < nl) g[l] = G[row + (size_t)n * (l * nf + nu)];
    }
    for (int l2 = 0; l2 < nl; l2++) {
      const int col = l2 * nf + nu;
      const size_t e = row + (size_t)n * col;
      cplx acc = cmk(0.0, 0.0);
      if constexpr (LMAX > 0) {
#pragma unroll
        for (int l1 = 0; l1 < LMAX; l1++)
          if (l1 < nl) acc = tups::cfma(g[l1], chi[l1 + nl * (l2 + (size_t)nl * nu)], acc);
      } else {
        for (int l1 = 0; l1 < nl; l1++)
          acc = tups::cfma(G[row + (size_t)n * (l1 * nf + nu)], chi[l1 + nl * (l2 + (size_t)nl * nu)], acc);
      }
      A[e] = cmk((row == col ? 1.0 : 0.0) - d.scale * acc.x, -d.scale * acc.y);
      F[e] = G[e];
    }
  }
}

__global__ void __launch_bounds__(256) k_lu_form(const cplx* __restrict__ Gam, const cplx* __restrict__ chi_all,
                                                 cplx* __restrict__ Fout, cplx* __restrict__ Aw) {
  const LuDesc d = g_lu_desc[blockIdx.y];
  if (blockIdx.x == 0 && threadIdx.x == 0) g_lu_status[blockIdx.y] = 0;
  const cplx* G = Gam + d.g_off;
  const cplx* chi = chi_all + d.c_off;
  cplx* A = Aw + d.g_off;
  cplx* F = Fout + d.g_off;
  if (d.nl <= 1) form_lines<1>(d, G, chi, A, F);
  else if (d.nl <= 5) form_lines<5>(d, G, chi, A, F);
  else if (d.nl <= 9) form_lines<9>(d, G, chi, A, F);
  else if (d.nl <= 13) form_lines<13>(d, G, chi, A, F);
  else form_lines<0>(d, G, chi, A, F);
}

// ---- one block of 64 columns ------------------------------------------------------
struct LuPanelShared {
  tups::lud::BlockShared b;
  int moved;
  int row[2 * NB], cur[2 * NB];  // replay of the interchanges (tall blocks)
};

// Columns [j0, j0 + 64) of every instance (one CTA each): two 32-column panels
// with a 32-wide update between them, and the interchange map.
// RPT: rows per thread in registers, 0 = columns in global memory.
// A serial chain of column steps: bound by barrier and FP64 latency, not by
// bandwidth; its SMs' FP64 pipes idle between the steps.
template <int RPT>
__global__ void __launch_bounds__(kPanelThreads, 1) k_lu_panel(cplx* __restrict__ Aw, int* __restrict__ piv_all,
                                                               int step) {
  extern __shared__ __align__(16) unsigned char smraw[];
  LuPanelShared& S = *reinterpret_cast<LuPanelShared*>(smraw);
  const int inst = blockIdx.x, tid = threadIdx.x;
  const LuDesc d = g_lu_desc[inst];
  const int n = d.n, j0 = step * NB, jb = min(NB, n - j0), je = j0 + jb;
  cplx* A = Aw + d.g_off;
  int* ipiv = piv_all + d.p_off;
  LuMap& map = g_lu_map[inst];
  for (int i = tid; i < kPanelRows; i += kPanelThreads) S.b.orig[i] = i;
  if (tid == 0) S.moved = 0;
  __syncthreads();
  auto track = [&](int c, int p) {
    if (RPT > 0) {
      const int x = S.b.orig[c - j0];
      S.b.orig[c - j0] = S.b.orig[p - j0];
      S.b.orig[p - j0] = x;
    }
  };
  tups::lud::block_factor<RPT, NB>(A, n, j0, jb, j0, je, ipiv, &g_lu_status[inst], S.b, track);
  // the interchange map: block rows take src, the rows below that changed take
  // a block row (an interchange always involves the block)
  if (RPT > 0) {
    if (tid < NB) map.src[tid] = tid < jb ? j0 + S.b.orig[tid] : 0;
    for (int i = jb + tid; i < n - j0; i += kPanelThreads)
      if (S.b.orig[i] != i) map.moved[atomicAdd(&S.moved, 1)] = (j0 + i) << 6 | S.b.orig[i];
  } else if (tid == 0) {
    int cnt = jb;
    for (int k = 0; k < jb; k++) {
      S.row[k] = j0 + k;
      S.cur[k] = k;
    }
    for (int k = 0; k < jb; k++) {
      const int p = ipiv[j0 + k];
      int x = p < je ? p - j0 : jb;
      if (p >= je) {
        while (x < cnt && S.row[x] != p) x++;
        if (x == cnt) {
          S.row[cnt] = p;
          S.cur[cnt++] = x;
        }
      }
      const int t = S.cur[k];
      S.cur[k] = S.cur[x];
      S.cur[x] = t;
    }
    for (int k = 0; k < NB; k++) map.src[k] = k < jb ? S.row[S.cur[k]] : 0;
    for (int x = jb; x < cnt; x++) map.moved[x - jb] = S.row[x] << 6 | S.cur[x];
    S.moved = cnt - jb;
  }
  __syncthreads();
  if (tid == 0) map.count = S.moved;
}

// column c of [A right of the block | F] (forward) or of F (backward)
__device__ __forceinline__ cplx* rhs_column(cplx* A, cplx* F, int n, int right, int c) {
  return c < right ? A + (size_t)n * (n - right + c) : F + (size_t)n * (c - right);
}

// first row of the block of launch `step`: the step-th from the top, or from
// the bottom (BACK)
template <bool BACK>
__device__ __forceinline__ int block_start(int n, int step) {
  return BACK ? ((n + NB - 1) / NB - 1 - step) * NB : step * NB;
}

// ---- block row: X[block, tile] = T^{-1} (P X)[block, tile], T = L11 or U_bb -------
// 32 columns per CTA, a warp per 8 of them and all 64 rows, so the triangle's
// shape shortens every warp alike.  The interchanges are a gather: all reads of
// the tile end before its first write.
constexpr int RW_BN = 32, RW_THREADS = 4 * RW_BN, RW_LDL = NB + 2, RW_LDB = NB + 4;
constexpr size_t kRowsSmem = ((size_t)NB * RW_LDL + RW_BN * RW_LDB + NB) * sizeof(cplx);

__device__ __forceinline__ void lu_cp_async16(void* sdst, const void* gsrc, bool valid) {
  unsigned sz = valid ? 16u : 0u;
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gsrc), "r"(sz));
}

template <bool BACK>
__global__ void __launch_bounds__(RW_THREADS, 2) k_lu_rows(cplx* __restrict__ Aw, cplx* __restrict__ Fout, int step) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx* sL = reinterpret_cast<cplx*>(smraw);  // [k][m]
  cplx* sB = sL + NB * RW_LDL;                // [col][k]
  cplx* sI = sB + RW_BN * RW_LDB;             // reciprocals of U_bb's diagonal
  const int inst = blockIdx.y;
  const LuDesc d = g_lu_desc[inst];
  const int n = d.n, j0 = block_start<BACK>(n, step), jb = min(NB, n - j0), je = j0 + jb;
  const int right = BACK ? 0 : n - je, width = right + n, c0 = blockIdx.x * RW_BN;
  if (c0 >= width) return;
  cplx* A = Aw + d.g_off;
  cplx* F = Fout + d.g_off;
  const LuMap& map = g_lu_map[inst];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kStep = RW_THREADS / NB;
  const int tm = tid % NB, tc = tid / NB;  // this thread's row and first column of both operands
  const int srow = BACK ? j0 + tm : map.src[tm];
#pragma unroll
  for (int i = 0; i < RW_BN / kStep; i++) {
    const int c = c0 + tc + kStep * i;
    const bool in = tm < jb && c < width;
    lu_cp_async16(&sB[(tc + kStep * i) * RW_LDB + tm], in ? rhs_column(A, F, n, right, c) + srow : A, in);
  }
#pragma unroll
  for (int i = 0; i < NB / kStep; i++) {
    const int k = tc + kStep * i;
    const bool in = tm < jb && k < jb && (BACK ? tm <= k : tm > k);
    lu_cp_async16(&sL[k * RW_LDL + tm], in ? A + j0 + tm + (size_t)n * (j0 + k) : A, in);
  }
  asm volatile("cp.async.commit_group;\n" ::);
  // the rows below the block that take a block row
  cplx v[RW_BN / kStep];
  const int cnt = BACK ? 0 : map.count, mv = tm < cnt ? map.moved[tm] : 0;
  if (!BACK && tm < cnt) {
#pragma unroll
    for (int i = 0; i < RW_BN / kStep; i++) {
      const int c = c0 + tc + kStep * i;
      if (c < width) v[i] = rhs_column(A, F, n, right, c)[j0 + (mv & 63)];
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  if (BACK) {
    if (tid < NB) sI[tid] = tups::lud::diagonal_reciprocal(sL[tid * RW_LDL + tid]);
    __syncthreads();
  } else if (tm < cnt) {
#pragma unroll
    for (int i = 0; i < RW_BN / kStep; i++) {
      const int c = c0 + tc + kStep * i;
      if (c < width) rhs_column(A, F, n, right, c)[mv >> 6] = v[i];
    }
  }
  cplx* x = sB + warp * 8 * RW_LDB;
  tups::lud::solve_triangle<BACK>(sL, RW_LDL, sI, x, RW_LDB, jb);
#pragma unroll
  for (int i = 0; i < NB / 4; i++) {
    const int m = lane + 32 * (i & 1), j = i >> 1, c = c0 + warp * 8 + j;
    if (m < jb && c < width) rhs_column(A, F, n, right, c)[j0 + m] = x[j * RW_LDB + m];
  }
}

// ---- update: C -= L21 U12 (forward), F_above -= U_above,b X_b (backward) -----------
// 32 x 32 complex tiles, 4 warps of 16 x 16, K = 64 in two cp.async stages of
// 16, four real tensor-core products per complex one: with three the error of
// an imaginary part is that of the real parts' products, 1e-7 of it where the
// matrix is real to 1e-8.
constexpr int UP_BM = 32, UP_BN = 32, UP_BK = 16, UP_LDL = UP_BM + 2, UP_LDR = UP_BK + 4;

template <bool BACK>
__global__ void __launch_bounds__(128, 5) k_lu_update(cplx* __restrict__ Aw, cplx* __restrict__ Fout, int step) {
  __shared__ __align__(16) cplx sL[2][UP_BK][UP_LDL];
  __shared__ __align__(16) cplx sR[2][UP_BN][UP_LDR];
  const LuDesc& d = g_lu_desc[blockIdx.y];
  const int n = d.n, j0 = block_start<BACK>(n, step), je = min(j0 + NB, n);
  const int first = BACK ? 0 : je, rows = BACK ? j0 : n - je;  // rows of C
  const int right = BACK ? 0 : n - je, width = right + n;
  const int tiles_m = (rows + UP_BM - 1) / UP_BM;
  if (tiles_m == 0) return;
  const int m0 = (int)(blockIdx.x % tiles_m) * UP_BM, n0 = (int)(blockIdx.x / tiles_m) * UP_BN;
  if (n0 >= width) return;
  cplx* A = Aw + d.g_off;
  cplx* F = Fout + d.g_off;
  const int K = je - j0, ktiles = (K + UP_BK - 1) / UP_BK;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm0 = (warp % 2) * 16, wn0 = (warp / 2) * 16;
  const int gid = lane >> 2, tig = lane & 3;
  // this thread's fixed row of A, column of B and their k offsets
  const int am = tid % UP_BM, ak = tid / UP_BM, bk = tid % UP_BK, bc = tid / UP_BK;
  const cplx* pa = A + first + min(m0 + am, rows - 1) + (size_t)n * j0;
  const bool okm = m0 + am < rows;
  const cplx* pb[4];
  bool okc[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int c = n0 + bc + 8 * i;
    okc[i] = c < width;
    pb[i] = rhs_column(A, F, n, right, min(c, width - 1)) + j0;
  }
  auto load = [&](int st, int kt) {
    const int k0 = kt * UP_BK;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int k = k0 + ak + 4 * i;
      lu_cp_async16(&sL[st][ak + 4 * i][am], k < K ? pa + (size_t)n * k : pa, okm && k < K);
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
      lu_cp_async16(&sR[st][bc + 8 * i][bk], k0 + bk < K ? pb[i] + k0 + bk : pb[i], okc[i] && k0 + bk < K);
    asm volatile("cp.async.commit_group;\n" ::);
  };
  double re[2][4] = {}, im[2][4] = {};
  load(0, 0);
  for (int kt = 0; kt < ktiles; kt++) {
    const int cur = kt & 1;
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    if (kt + 1 < ktiles) load(cur ^ 1, kt + 1);
#pragma unroll
    for (int k8 = 0; k8 < UP_BK; k8 += 8) {
      const int mb = wm0 + gid;
      const cplx v0 = sL[cur][k8 + tig][mb], v1 = sL[cur][k8 + tig][mb + 8];
      const cplx v2 = sL[cur][k8 + tig + 4][mb], v3 = sL[cur][k8 + tig + 4][mb + 8];
      const double are[4] = {v0.x, v1.x, v2.x, v3.x}, aim[4] = {v0.y, v1.y, v2.y, v3.y};
      const double aneg[4] = {-v0.y, -v1.y, -v2.y, -v3.y};
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int nb = wn0 + j * 8 + gid;
        const cplx w0 = sR[cur][nb][k8 + tig], w1 = sR[cur][nb][k8 + tig + 4];
        const double bre[2] = {w0.x, w1.x}, bim[2] = {w0.y, w1.y};
        dmma8(re[j], are, bre);
        dmma8(re[j], aneg, bim);
        dmma8(im[j], are, bim);
        dmma8(im[j], aim, bre);
      }
    }
  }
  // the old entries all go out before the first write, which could alias them
  // (one after another they kept the kernel waiting: 0.9 ms over 96 instances of n = 64..832)
  cplx old[2][4];
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int x = 0; x < 4; x++) {
      const int row = m0 + wm0 + gid + (x >= 2 ? 8 : 0), col = n0 + wn0 + j * 8 + 2 * tig + (x & 1);
      old[j][x] = rhs_column(A, F, n, right, min(col, width - 1))[first + min(row, rows - 1)];
    }
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int x = 0; x < 4; x++) {
      const int row = m0 + wm0 + gid + (x >= 2 ? 8 : 0), col = n0 + wn0 + j * 8 + 2 * tig + (x & 1);
      const cplx v = old[j][x];
      if (row < rows && col < width)
        rhs_column(A, F, n, right, col)[first + row] =
            cmk(v.x - re[j][x], v.y - im[j][x]);
    }
}

// the instances of up to kSmall rows (the last of the queue, from `first` on): a CTA each
__global__ void __launch_bounds__(tups::lud::kSmallThreads) k_lu_small(cplx* __restrict__ Aw, cplx* __restrict__ Fout,
                                                                       int* __restrict__ piv_all, int first) {
  __shared__ tups::lud::SmallShared S;
  const int inst = first + blockIdx.x;
  const LuDesc& d = g_lu_desc[inst];
  cplx* F = Fout + d.g_off;
  tups::lud::small_solve(Aw + d.g_off, F, F, d.n, piv_all + d.p_off, &g_lu_status[inst], S);
}

// F -= Gamma
__global__ void __launch_bounds__(256) k_lu_phi(const cplx* __restrict__ Gam, cplx* __restrict__ Fout) {
  const LuDesc& d = g_lu_desc[blockIdx.y];
  const size_t n2 = (size_t)d.n * d.n;
  const cplx* G = Gam + d.g_off;
  cplx* F = Fout + d.g_off;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n2; e += (size_t)gridDim.x * blockDim.x)
    F[e] = tups::csub(F[e], G[e]);
}

// opt-in shared-memory sizes on the current device
bool lu_prepare() {
  const int ps = (int)sizeof(LuPanelShared), rs = (int)kRowsSmem;
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  return cudaFuncSetAttribute(k_lu_panel<0>, attr, ps) == cudaSuccess &&
         cudaFuncSetAttribute(k_lu_panel<1>, attr, ps) == cudaSuccess &&
         cudaFuncSetAttribute(k_lu_panel<2>, attr, ps) == cudaSuccess &&
         cudaFuncSetAttribute(k_lu_rows<false>, attr, rs) == cudaSuccess &&
         cudaFuncSetAttribute(k_lu_rows<true>, attr, rs) == cudaSuccess;
}

}  // namespace

extern "C" int tups_bse_lu_batched(int n_inst, const int* n, const int* nl, const double* scale, const double* gamma,
                                   const double* chi, double* out, double* work, int* ipiv, int want_phi,
                                   int* status, void* stream) {
  if (n_inst < 1 || n_inst > kLuMaxInst || !n || !nl || !scale || !gamma || !chi || !out || !work || !ipiv)
    return TUPS_ERR_BADARG;
  std::vector<LuDesc> desc(n_inst);
  long long go = 0, co = 0, po = 0;
  for (int i = 0; i < n_inst; i++) {
    if (n[i] < 1 || nl[i] < 1 || n[i] % nl[i]) return TUPS_ERR_BADDIM;
    desc[i] = {go, co, po, n[i], nl[i], scale[i]};
    go += (long long)n[i] * n[i];
    co += (long long)nl[i] * nl[i] * (n[i] / nl[i]);
    po += n[i];
  }
  // largest first: the instances that still have a block are the first ones
  std::vector<int> order(n_inst);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return n[a] > n[b]; });
  std::vector<LuDesc> queued(n_inst);
  for (int i = 0; i < n_inst; i++) queued[i] = desc[order[i]];
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (!lu_prepare() ||
      cudaMemcpyToSymbolAsync(g_lu_desc, queued.data(), n_inst * sizeof(LuDesc), 0, cudaMemcpyHostToDevice, st) !=
          cudaSuccess) {
    cudaGetLastError();
    return TUPS_ERR_CUDA;
  }
  const cplx* G = reinterpret_cast<const cplx*>(gamma);
  cplx* A = reinterpret_cast<cplx*>(work);
  cplx* F = reinterpret_cast<cplx*>(out);
  const int nmax = queued[0].n;
  const unsigned eg = (unsigned)std::min<long long>(((long long)nmax * nmax + 255) / 256, 512);
  const auto tiles = [](long long rows, long long cols) {
    return (unsigned)((rows + UP_BM - 1) / UP_BM * ((cols + UP_BN - 1) / UP_BN));
  };
  // grid rows of at most 65535 instances (n_inst <= 16384)
  k_lu_form<<<dim3(eg, n_inst), 256, 0, st>>>(G, reinterpret_cast<const cplx*>(chi), F, A);
  // instances of up to 32 rows, the last of the queue, whole; the others by blocks
  int large = n_inst;
  while (large > 0 && queued[large - 1].n <= tups::lud::kSmall) large--;
  if (large < n_inst) k_lu_small<<<n_inst - large, tups::lud::kSmallThreads, 0, st>>>(A, F, ipiv, large);
  int live = large;
  for (int step = 0; large > 0 && step * NB < nmax; step++) {
    const int j0 = step * NB;
    while (queued[live - 1].n <= j0) live--;
    const int rows = nmax - j0, below = std::max(0, rows - NB);
    const size_t ps = sizeof(LuPanelShared);
    const auto panel = rows <= kPanelThreads ? k_lu_panel<1> : rows <= kPanelRows ? k_lu_panel<2> : k_lu_panel<0>;
    panel<<<live, kPanelThreads, ps, st>>>(A, ipiv, step);
    const long long width = (long long)below + nmax;
    k_lu_rows<false><<<dim3((unsigned)((width + RW_BN - 1) / RW_BN), live), RW_THREADS, kRowsSmem, st>>>(A, F, step);
    if (below > 0) k_lu_update<false><<<dim3(tiles(below, width), live), 128, 0, st>>>(A, F, step);
  }
  live = large;
  for (int step = 0; large > 0 && step * NB < nmax; step++) {
    while (queued[live - 1].n <= step * NB) live--;
    const int above = ((nmax + NB - 1) / NB - 1 - step) * NB;
    k_lu_rows<true><<<dim3((unsigned)((nmax + RW_BN - 1) / RW_BN), live), RW_THREADS, kRowsSmem, st>>>(A, F, step);
    if (above > 0) k_lu_update<true><<<dim3(tiles(above, nmax), live), 128, 0, st>>>(A, F, step);
  }
  if (want_phi) k_lu_phi<<<dim3(eg, n_inst), 256, 0, st>>>(G, F);
  if (cudaGetLastError() != cudaSuccess) return TUPS_ERR_CUDA;
  if (status) {
    std::vector<int> st_q(n_inst);
    if (cudaMemcpyFromSymbolAsync(st_q.data(), g_lu_status, n_inst * sizeof(int), 0, cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      cudaGetLastError();
      return TUPS_ERR_CUDA;
    }
    for (int i = 0; i < n_inst; i++) status[order[i]] = st_q[i];
  }
  return TUPS_OK;
}
