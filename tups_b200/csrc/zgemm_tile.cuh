// One CTA tile of a complex GEMM on the FP64 tensor cores (mma.sync m16n8k8
// f64), shared by the BSE GEMM, its no-allocation form, the crossing and, in the
// split LU, the second panel's update and the residual.
//
// Operands arrive by cp.async into ST shared-memory stages of BK columns; the
// fragments of the next k8 step are read into a second register set before the
// current step's products, across the stage barrier too, so a warp's tensor
// products never wait for shared memory.  With M3 a complex product is three
// real ones (Gauss: P1 = Ar Br, P2 = Ai Bi, P3 = (Ar + Ai)(Br + Bi); Re = P1 -
// P2, Im = P3 - P1 - P2); the P1 and P2 products go out first and cover the
// latency of the sums.  What bounds it: the FP64 pipe, which the sums share
// with the products (a register-only loop with the same 8 sums per 6 products
// reaches 45 TFLOP/s, counted as four products per complex one, of 49).
// Fetching a stage's fragments only after its barrier and forming every source
// address by index, as before, the 160 x 160 BSE (K = 320, 960 matrices) ran at
// 35.2 TFLOP/s, this at 38.7; 576 x 576 (K = 1152): 36.8 -> 40.9.  TMA stages
// behind mbarriers with a producer warp measured no faster (40.0), nor did
// 16 x 32 or 32 x 16 warp tiles (32 and 27 at 160 x 160).
//
// Warps whose rows or columns all lie past the matrix only copy and keep the
// barriers.  The warp number comes through a shuffle so that this test is known
// to be uniform: as a plain function of threadIdx every product after it is
// compiled for a diverged warp, which costs 10 %.
#pragma once

#include "tups_device.cuh"

namespace tups {

__device__ __forceinline__ void zg_cp_async16(void* sdst, const void* gsrc, bool valid) {
  const unsigned sz = valid ? 16u : 0u;
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gsrc), "r"(sz));
}

__device__ __forceinline__ void zg_dmma(double* c, const double* a, const double* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// what an epilogue reads per entry: two matrices
struct ZgPair {
  cplx a, b;
};

// WM x WN warps of 16 TM x 8 TN.  Without AHEAD the fragments of a step are read
// when it starts: fewer registers, so more CTAs per SM, and the padding of a last
// stage is skipped, which is the better side for short sums (the crossing at K =
// 100: 5 CTAs per SM 1.03 ms, 3 with AHEAD 1.30).
template <int TM, int TN, int WM, int WN, int BK, int ST, bool M3, bool AHEAD = true>
struct ZgemmTile {
  static constexpr int BM = 16 * TM * WM, BN = 8 * TN * WN, NW = WM * WN, NT = 32 * NW;
  static constexpr int LDL = BM + 2, LDR = BK + 4;  // conflict-free 16-byte fragment reads
  static constexpr int KB = BK / 8;
  static constexpr size_t kSmem = (size_t)ST * (BK * LDL + BN * LDR) * sizeof(cplx);
  static_assert(ST >= 2 && KB >= 2 && KB % 2 == 0, "pipeline shape");

  double p1[TM][TN][4], p2[TM][TN][4], p3[M3 ? TM : 1][M3 ? TN : 1][4];
  int wm0, wn0, gid, tig;

  // The tile's sums.  src.ktiles() stages; stage kt holds src.depth(kt) <= BK
  // columns of the left operand, element (m, k) at src.left(kt)[m + ld k],
  // ld = src.ldl(), and as many rows of the right one, element (k, n) at
  // src.right(kt)[src.roff(n) + k].  rows, cols: extent of the matrix from the
  // tile on.  sm: kSmem bytes, 16-byte aligned.  With Src::kGather the source
  // forms the left operand itself: src.fetch(kt) reads what stage kt needs into
  // registers and src.put(stage) writes it, entry (m, k) at stage[k LDL + m],
  // after the products of the step between (only without AHEAD).
  template <class Src>
  __device__ __forceinline__ void run(Src src, cplx* sm, int rows, int cols) {
    static_assert(!(Src::kGather && AHEAD), "a gathering source has no read-ahead form");
    cplx* sL = sm;                         // [ST][BK][LDL]
    cplx* sR = sL + (size_t)ST * BK * LDL; // [ST][BN][LDR]
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    wm0 = (warp % WM) * (16 * TM);
    wn0 = (warp / WM) * (8 * TN);
    gid = lane >> 2;
    tig = lane & 3;
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          p1[i][j][e] = p2[i][j][e] = 0.0;
          if (M3) p3[M3 ? i : 0][M3 ? j : 0][e] = 0.0;
        }
    const int ktiles = src.ktiles();
    const size_t ld = src.ldl();
    auto load = [&](int st, int kt) {
      const int kv = src.depth(kt);
      const cplx *pl = src.left(kt), *pr = src.right(kt);
      cplx* dL = sL + (size_t)st * BK * LDL;
      cplx* dR = sR + (size_t)st * BN * LDR;
      if constexpr (!Src::kGather) {
#pragma unroll
        for (int i = 0; i < (BK * BM + NT - 1) / NT; i++) {
          const int e = tid + i * NT, m = e % BM, k = e / BM;
          if (BK * BM % NT == 0 || e < BK * BM) {
            const bool ok = m < rows && k < kv;
            zg_cp_async16(dL + k * LDL + m, ok ? pl + m + ld * k : pl, ok);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < (BK * BN + NT - 1) / NT; i++) {
        const int e = tid + i * NT, k = e % BK, n = e / BK;
        if (BK * BN % NT == 0 || e < BK * BN) {
          const bool ok = n < cols && k < kv;
          zg_cp_async16(dR + n * LDR + k, ok ? pr + src.roff(n) + k : pl, ok);
        }
      }
    };
    cplx fa[AHEAD ? 2 : 1][TM][4], fb[AHEAD ? 2 : 1][TN][2];
    auto fetch = [&](int buf, int st, int k8) {
      const cplx* cL = sL + (size_t)st * BK * LDL + (k8 + tig) * LDL + wm0 + gid;
      const cplx* cR = sR + (size_t)st * BN * LDR + (wn0 + gid) * LDR + k8 + tig;
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) fa[buf][i][e] = cL[(e >> 1) * 4 * LDL + 16 * i + (e & 1) * 8];
#pragma unroll
      for (int j = 0; j < TN; j++) {
        fb[buf][j][0] = cR[8 * j * LDR];
        fb[buf][j][1] = cR[8 * j * LDR + 4];
      }
    };
#pragma unroll
    for (int s = 0; s < ST - 1; s++) {
      if (s < ktiles) {
        load(s, s);
        if constexpr (Src::kGather) {
          src.fetch(s);
          src.put(sL + (size_t)s * BK * LDL);
        }
      }
      asm volatile("cp.async.commit_group;\n" ::);
    }
    // this thread's copies of the next stage, and every warp past its reads of
    // the stage before the current one
    auto land = [] {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2));
      asm volatile("bar.sync 0;\n" ::: "memory");  // working and idle warps meet here from different loops
    };
    int st = 0, ldst = ST - 1;
    cplx* filling = nullptr;  // kGather: the stage whose left operand is in registers
    auto refill = [&](int kt) {
      if (kt + ST - 1 < ktiles) {
        load(ldst, kt + ST - 1);
        if constexpr (Src::kGather) {
          src.fetch(kt + ST - 1);
          filling = sL + (size_t)ldst * BK * LDL;
        }
      }
      asm volatile("cp.async.commit_group;\n" ::);
      ldst = ldst + 1 == ST ? 0 : ldst + 1;
    };
    auto fill = [&] {
      if constexpr (Src::kGather) {
        if (filling) src.put(filling);
        filling = nullptr;
      }
    };
    if (AHEAD) land();
    if (wm0 >= rows || wn0 >= cols) {
      for (int kt = 0; kt < ktiles; kt++) {
        if (!AHEAD) land();
        refill(kt);
        fill();
        if (AHEAD) land();
      }
      return;
    }
    if (AHEAD) fetch(0, 0, 0);
    for (int kt = 0; kt < ktiles; kt++) {
      if (!AHEAD) {
        land();
        refill(kt);
      }
#pragma unroll
      for (int kk = 0; kk < KB; kk++) {
        const int cur = AHEAD ? kk & 1 : 0;
        if (!AHEAD) {
          fetch(0, st, 8 * kk);
          if (kk == KB - 1) st = st + 1 == ST ? 0 : st + 1;
        } else if (kk == KB - 1) {
          land();
          st = st + 1 == ST ? 0 : st + 1;
          fetch(cur ^ 1, st, 0);  // past the last stage: stale content, unused
        } else {
          fetch(cur ^ 1, st, 8 * (kk + 1));
        }
        if (AHEAD && kk == 0) refill(kt);
        if (!AHEAD && kk > 0 && 8 * kk >= src.depth(kt)) continue;  // a short last stage
        double ar[TM][4], ai[TM][4], as[TM][4];
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            ar[i][e] = fa[cur][i][e].x;
            ai[i][e] = fa[cur][i][e].y;
            as[i][e] = M3 ? ar[i][e] + ai[i][e] : -ai[i][e];
          }
        double bs[TN][2];
        if (M3) {
#pragma unroll
          for (int j = 0; j < TN; j++)
#pragma unroll
            for (int e = 0; e < 2; e++) bs[j][e] = fb[cur][j][e].x + fb[cur][j][e].y;
        }
#pragma unroll
        for (int j = 0; j < TN; j++) {
          const double br[2] = {fb[cur][j][0].x, fb[cur][j][1].x}, bi[2] = {fb[cur][j][0].y, fb[cur][j][1].y};
#pragma unroll
          for (int i = 0; i < TM; i++) {
            zg_dmma(p1[i][j], ar[i], br);
            zg_dmma(p2[i][j], ai[i], M3 ? bi : br);
            if (!M3) {
              zg_dmma(p1[i][j], as[i], bi);
              zg_dmma(p2[i][j], ar[i], bi);
            }
          }
        }
        if (M3) {
#pragma unroll
          for (int j = 0; j < TN; j++) {
  #pragma unroll
            for (int i = 0; i < TM; i++) zg_dmma(p3[M3 ? i : 0][M3 ? j : 0], as[i], bs[j]);
          }
        }
      }
      fill();
    }
  }

  // f(row, col, value) over this thread's entries inside the matrix
  template <class F>
  __device__ __forceinline__ void each(int rows, int cols, F f) const {
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int row = wm0 + 16 * i + gid + (e >= 2 ? 8 : 0), col = wn0 + 8 * j + 2 * tig + (e & 1);
          if (row < rows && col < cols)
            f(row, col, M3 ? cmk(p1[i][j][e] - p2[i][j][e], p3[M3 ? i : 0][M3 ? j : 0][e] - p1[i][j][e] - p2[i][j][e])
                           : cmk(p1[i][j][e], p2[i][j][e]));
        }
  }

  // the same with what f reads: get(row, col) of all of this thread's entries
  // goes out before the first f writes.  The writes could alias the reads, so
  // that otherwise each entry's reads wait for memory in turn.  Entries
  // outside the matrix get its last row or column and see no f.
  template <class G, class F>
  __device__ __forceinline__ void each(int rows, int cols, G get, F f) const {
    decltype(get(0, 0)) in[TM][TN][4];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++)
#pragma unroll
        for (int e = 0; e < 4; e++)
          in[i][j][e] = get(min(wm0 + 16 * i + gid + (e >= 2 ? 8 : 0), rows - 1),
                            min(wn0 + 8 * j + 2 * tig + (e & 1), cols - 1));
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int row = wm0 + 16 * i + gid + (e >= 2 ? 8 : 0), col = wn0 + 8 * j + 2 * tig + (e & 1);
          if (row < rows && col < cols)
            f(row, col, M3 ? cmk(p1[i][j][e] - p2[i][j][e], p3[M3 ? i : 0][M3 ? j : 0][e] - p1[i][j][e] - p2[i][j][e])
                           : cmk(p1[i][j][e], p2[i][j][e]), in[i][j][e]);
        }
  }
};

// [A | F] [F ; B]: the two halves of the BSE's K = 2 Nz, each padded to whole
// stages of its own.  a, f, b: (Nz, Nz) matrices of one instance
template <int BK>
struct BseSource {
  static constexpr bool kGather = false;
  const cplx *a, *f, *b;
  int Nz, m0, n0;
  __device__ int half() const { return (Nz + BK - 1) / BK; }
  __device__ int ktiles() const { return 2 * half(); }
  __device__ int k0(int kt) const { return (kt < half() ? kt : kt - half()) * BK; }
  __device__ int depth(int kt) const { return min(BK, Nz - k0(kt)); }
  __device__ size_t ldl() const { return (size_t)Nz; }
  __device__ const cplx* left(int kt) const { return (kt < half() ? a : f) + m0 + (size_t)Nz * k0(kt); }
  __device__ const cplx* right(int kt) const { return (kt < half() ? f : b) + k0(kt); }
  __device__ size_t roff(int n) const { return (size_t)Nz * (n0 + n); }
};

}  // namespace tups
