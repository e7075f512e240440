// Batched BSE update that allocates no device memory.
//
// The regular BSE path (bse.cu) keeps its Gamma*chi / chi*Gamma scratch in a
// buffer that tups_ctx_create obtains with cudaMalloc.  Some callers cannot
// allocate device memory when they call into this library: a Fortran/MPI
// host that hands the whole device memory to its own arena at start-up, or
// an embedding whose driver loop must not trigger the implicit device-wide
// synchronisation and possible failure of cudaMalloc/cudaFree.  This entry
// point takes only caller-owned inputs and outputs and keeps its scratch in
// a fixed-size array in the library's own static device memory.
//
// The scratch is a file-scope __device__ array of kScratchComplex complex128
// (32 MiB), present on every GPU that loads the library until the process
// exits.  Host code cannot use the array's name as a device address; the
// address is looked up once per device with cudaGetSymbolAddress (with that
// device current) on the first call made on the device, so that first call
// should come before any stream capture.  The address is kept for the life
// of the process: after a cudaDeviceReset the device's module, and with it
// the array, is loaded anew, so a process that resets a device must not call
// this entry point on that device again.  All calls share the array and it
// keeps the last call's contents; every element a call reads is written by
// that call first.  Calls whose kernels overlap on the GPU (different
// streams, or different host threads) race on the array.
#include <algorithm>
#include <cstdio>
#include <mutex>

#include "tups_device.cuh"
#include "zgemm_tile.cuh"

namespace {

using tups::cplx;

constexpr size_t kScratchComplex = (size_t)2 << 20;  // 2 Mi complex128 = 32 MiB
constexpr int kMaxDevices = 64;

static __device__ __align__(256) double2 g_bse_scratch[kScratchComplex];

std::mutex g_mu;
cplx* g_scratch_ptr[kMaxDevices] = {};

// device address of g_bse_scratch on the current device, looked up once
int scratch_address(int dev, cplx** out) {
  if (dev < 0 || dev >= kMaxDevices) return TUPS_ERR_BADARG;
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_bse_scratch);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      return TUPS_ERR_CUDA;
    }
    g_scratch_ptr[dev] = static_cast<cplx*>(p);
  }
  *out = g_scratch_ptr[dev];
  return TUPS_OK;
}

// A = Gamma chi, B = chi Gamma for instances [i0, i0+n) into the scratch, sums
// over the form factor ascending.  The first nA CTAs of an instance form A: a
// thread per (row, nu) line loads the line's Nl <= LMAX entries of Gamma once
// for its Nl outputs, lanes over rows at one nu, so a chi entry is one address
// per warp.  The rest form B: a warp per column, lanes over nu, chi[:, :, 32 nu]
// staged in shared memory ([l1 + Nl l2][lane], pitch 33) when it fits.
constexpr int NA_LMAX = 16, NA_STAGE = 13;  // Nl up to which chi is staged

template <int LMAX>
__device__ __forceinline__ void na_gamma_chi(const cplx* __restrict__ Gm, const cplx* __restrict__ ch,
                                             cplx* __restrict__ Ai, int Nz, int Nf, int Nl, int cta, int ncta) {
  const size_t lines = (size_t)Nz * Nf;
  for (size_t t = (size_t)cta * blockDim.x + threadIdx.x; t < lines; t += (size_t)ncta * blockDim.x) {
    const int row = (int)(t % Nz), nu = (int)(t / Nz);
    cplx g[LMAX];
#pragma unroll
    for (int l = 0; l < LMAX; l++)
      if (l < Nl) g[l] = Gm[row + (size_t)Nz * (l * Nf + nu)];
    for (int l2 = 0; l2 < Nl; l2++) {
      const cplx* c = ch + Nl * (l2 + (size_t)Nl * nu);
      cplx acc = tups::cmk(0.0, 0.0);
#pragma unroll
      for (int l = 0; l < LMAX; l++)
        if (l < Nl) acc = tups::cfma(g[l], c[l], acc);
      Ai[row + (size_t)Nz * (l2 * Nf + nu)] = acc;
    }
  }
}

template <int LMAX>
__global__ void __launch_bounds__(256) k_noalloc_prep(const cplx* __restrict__ G, const cplx* __restrict__ chi,
                                                      cplx* __restrict__ A, cplx* __restrict__ B, int i0, int Nz,
                                                      int Nf, int Nl, int nA) {
  extern __shared__ cplx chs[];
  const int li = blockIdx.y;
  const size_t n2 = (size_t)Nz * Nz;
  const cplx* Gm = G + n2 * (i0 + li);
  const cplx* ch = chi + (size_t)Nl * Nl * Nf * (i0 + li);
  if ((int)blockIdx.x < nA) {
    na_gamma_chi<LMAX>(Gm, ch, A + n2 * li, Nz, Nf, Nl, blockIdx.x, nA);
    return;
  }
  const int cta = blockIdx.x - nA, nchunk = (Nf + 31) / 32, nu0 = (cta % nchunk) * 32;
  const int lane = threadIdx.x & 31, nu = nu0 + lane, col = cta / nchunk * 8 + (threadIdx.x >> 5);
  const bool staged = Nl <= NA_STAGE;
  if (staged)
    for (int e = threadIdx.x; e < Nl * Nl * min(32, Nf - nu0); e += 256) {
      const int ll = e % (Nl * Nl), j = e / (Nl * Nl);
      chs[ll * 33 + j] = ch[(size_t)ll + (size_t)Nl * Nl * (nu0 + j)];
    }
  __syncthreads();
  if (nu >= Nf || col >= Nz) return;
  const cplx* Gc = Gm + (size_t)Nz * col + nu;
  cplx* Bc = B + n2 * li + (size_t)Nz * col + nu;
  cplx g[LMAX];
#pragma unroll
  for (int l = 0; l < LMAX; l++)
    if (l < Nl) g[l] = Gc[l * Nf];
  for (int l1 = 0; l1 < Nl; l1++) {
    auto c = [&](int l2) { return staged ? chs[(l1 + Nl * l2) * 33 + lane] : ch[l1 + Nl * (l2 + (size_t)Nl * nu)]; };
    cplx acc = tups::cmk(0.0, 0.0);
#pragma unroll
    for (int l = 0; l < LMAX; l++)
      if (l < Nl) acc = tups::cfma(c(l), g[l], acc);
    Bc[l1 * Nf] = acc;
  }
}

// The same with a thread per entry of A and of B: for one form factor, where a
// line holds one entry, for few frequencies, where the lanes of a column idle, and
// for more form factors than a line keeps in registers.  With the GEMM, lines
// against entries: 30000 of Nf = 16, Nl = 1 332 against 262 us, 3000 of 7 x 7 891
// against 745, 20000 of 5 x 5 916 and 842, 4096 of 8 x 5 571 and 581, 2000 of 10 x 5
// 454 and 483, 240 of 32 x 5 683 and 747, 100 of 40 x 20 41.7 and 37.5 ms.
__global__ void __launch_bounds__(256) k_noalloc_prep_each(const cplx* __restrict__ G, const cplx* __restrict__ chi,
                                                           cplx* __restrict__ A, cplx* __restrict__ B, int i0, int Nz,
                                                           int Nf, int Nl) {
  const int li = blockIdx.y;
  const size_t n2 = (size_t)Nz * Nz;
  const cplx* Gm = G + n2 * (i0 + li);
  const cplx* ch = chi + (size_t)Nl * Nl * Nf * (i0 + li);
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n2; e += (size_t)gridDim.x * blockDim.x) {
    const int row = (int)(e % Nz), col = (int)(e / Nz), l2 = col / Nf, nu = col % Nf, l1 = row / Nf, mu = row % Nf;
    cplx a = tups::cmk(0.0, 0.0), b = a;
    for (int l = 0; l < Nl; l++)
      a = tups::cfma(Gm[row + (size_t)Nz * (l * Nf + nu)], ch[l + Nl * (l2 + (size_t)Nl * nu)], a);
    for (int l = 0; l < Nl; l++)
      b = tups::cfma(ch[l1 + Nl * (l + (size_t)Nl * mu)], Gm[(l * Nf + mu) + (size_t)Nz * col], b);
    A[n2 * li + e] = a;
    B[n2 * li + e] = b;
  }
}

// Phi = s [A | F] [F ; B] + (1-f)(F - Gamma) over Gamma, the BSE GEMM's tile with
// four real products per complex one (three measured 12 % less exact here)
constexpr int NB_BK = 16;

template <class Tile, int PER_SM>
__global__ void __launch_bounds__(Tile::NT, PER_SM) k_noalloc_gemm(cplx* __restrict__ G, const cplx* __restrict__ F,
                                                                   const cplx* __restrict__ A,
                                                                   const cplx* __restrict__ B, int i0, int Nz, double s,
                                                                   double one_minus_f) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int li = blockIdx.y;
  const size_t n2 = (size_t)Nz * Nz;
  const cplx* Fi = F + n2 * (i0 + li);
  cplx* Gi = G + n2 * (i0 + li);
  const int tiles_m = (Nz + Tile::BM - 1) / Tile::BM;
  const int m0 = (int)(blockIdx.x % tiles_m) * Tile::BM, n0 = (int)(blockIdx.x / tiles_m) * Tile::BN;
  Tile t;
  t.run(tups::BseSource<NB_BK>{A + n2 * li, Fi, B + n2 * li, Nz, m0, n0}, reinterpret_cast<cplx*>(smraw), Nz - m0,
        Nz - n0);
  const auto at = [&](int row, int col) { return (m0 + row) + (size_t)Nz * (n0 + col); };
  t.each(
      Nz - m0, Nz - n0, [&](int row, int col) { return tups::ZgPair{Fi[at(row, col)], Gi[at(row, col)]}; },
      [&](int row, int col, cplx c, const tups::ZgPair& v) {
        Gi[at(row, col)] =
            tups::cmk(s * c.x + one_minus_f * (v.a.x - v.b.x), s * c.y + one_minus_f * (v.a.y - v.b.y));
      });
}

// a tile's kernel and launch on instances [i0, i0 + n)
struct NaGemm {
  bool (*prepare)();
  void (*launch)(cplx* G, const cplx* F, const cplx* A, const cplx* B, int i0, int n, int Nz, double s, double omf,
                 cudaStream_t st);
};

template <class Tile, int PER_SM>
NaGemm na_gemm() {
  return {[] {
            return cudaFuncSetAttribute(k_noalloc_gemm<Tile, PER_SM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)Tile::kSmem) == cudaSuccess;
          },
          [](cplx* G, const cplx* F, const cplx* A, const cplx* B, int i0, int n, int Nz, double s, double omf,
             cudaStream_t st) {
            const int tiles = ((Nz + Tile::BM - 1) / Tile::BM) * ((Nz + Tile::BN - 1) / Tile::BN);
            k_noalloc_gemm<Tile, PER_SM><<<dim3(tiles, n), Tile::NT, Tile::kSmem, st>>>(G, F, A, B, i0, Nz, s, omf);
          }};
}

// Up to 16 rows a tile of 16 x 16.  Otherwise 32 x 32: with the fragments read ahead,
// except below 256 rows where the last step of a half of K would be more than half
// padding, which only the plain form skips, and below 32.  Plain against
// read-ahead: 9000 of 17 rows 206 and 212 us, 5000 of 33 485 and 533, 200 of 165 807
// and 876, 240 of 180 1.26 and 1.32 ms; 240 of 160 672 and 625 us, 100 of 250 1100 and
// 1031, 100 of 520 10.9 and 10.1 ms.
NaGemm na_choose(int Nz) {
  using namespace tups;
  if (Nz <= 16) return na_gemm<ZgemmTile<1, 1, 1, 2, NB_BK, 2, false, false>, 12>();
  if (Nz < 32 || (Nz < 256 && Nz % 16 >= 1 && Nz % 16 <= 8))
    return na_gemm<ZgemmTile<1, 2, 2, 2, NB_BK, 2, false, false>, 5>();
  return na_gemm<ZgemmTile<1, 2, 2, 2, NB_BK, 3, false>, 4>();
}

}  // namespace

extern "C" int tups_bse_noalloc(int n_inst, int Nz, int Nf, int Nl, double* gamma_phi, const double* F,
                                const double* chi, double scale, double f_damping, void* stream) {
  if (n_inst < 1 || Nf < 1 || Nl < 1 || Nz != Nl * Nf || !gamma_phi || !F || !chi) return TUPS_ERR_BADARG;
  const size_t per = 2 * (size_t)Nz * Nz;
  if (per > kScratchComplex) {
    std::fprintf(stderr,
                 "tups_bse_noalloc: Nz = %d needs %zu bytes of scratch per instance; the static scratch holds %zu "
                 "bytes (Nz <= 1024)\n",
                 Nz, per * sizeof(cplx), kScratchComplex * sizeof(cplx));
    return TUPS_ERR_BADDIM;
  }
  // an error left by an earlier, unrelated call would otherwise be reported
  // as this call's launch failure
  (void)cudaGetLastError();
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return TUPS_ERR_CUDA;
  }
  cplx* scratch = nullptr;
  int rc = scratch_address(dev, &scratch);
  if (rc != TUPS_OK) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // instances per pass through the scratch, at most 65535 (gridDim.y of both
  // kernels), in passes of equal size.  Smaller passes whose last wave is full
  // gain nothing: 240 of 160 rows 625 us in 6 passes, 683 in 11 of 23
  const size_t n2 = (size_t)Nz * Nz;
  const int cap = (int)std::min<size_t>(std::min<size_t>(kScratchComplex / per, 65535), (size_t)n_inst);
  const int passes = (n_inst + cap - 1) / cap, chunk = (n_inst + passes - 1) / passes;
  cplx* A = scratch;
  cplx* B = scratch + (size_t)cap * n2;
  const bool lines = Nl >= 2 && Nl <= NA_LMAX && Nf >= 10;
  const int nA = (int)std::min<size_t>(((size_t)Nz * Nf + 255) / 256, 4096);
  const int nB = ((Nf + 31) / 32) * ((Nz + 7) / 8);
  const size_t smp = Nl <= NA_STAGE ? (size_t)Nl * Nl * 33 * sizeof(cplx) : 0;
  const auto prep = Nl <= 5 ? k_noalloc_prep<5> : Nl <= 9 ? k_noalloc_prep<9> : k_noalloc_prep<NA_LMAX>;
  const NaGemm gemm = na_choose(Nz);
  if ((lines && smp > 48 * 1024 &&
       cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smp) != cudaSuccess) ||
      !gemm.prepare()) {
    cudaGetLastError();
    return TUPS_ERR_CUDA;
  }
  cplx* G = reinterpret_cast<cplx*>(gamma_phi);
  const cplx* f = reinterpret_cast<const cplx*>(F);
  const cplx* ch = reinterpret_cast<const cplx*>(chi);
  for (int i0 = 0; i0 < n_inst; i0 += chunk) {
    const int n = n_inst - i0 < chunk ? n_inst - i0 : chunk;
    if (lines)
      prep<<<dim3(nA + nB, n), 256, smp, st>>>(G, ch, A, B, i0, Nz, Nf, Nl, nA);
    else
      k_noalloc_prep_each<<<dim3((unsigned)std::min<size_t>((n2 + 255) / 256, 1024), n), 256, 0, st>>>(G, ch, A, B, i0,
                                                                                                      Nz, Nf, Nl);
    if (cudaGetLastError() != cudaSuccess) return TUPS_ERR_CUDA;
    gemm.launch(G, f, A, B, i0, n, Nz, scale, 1.0 - f_damping, st);
    if (cudaGetLastError() != cudaSuccess) return TUPS_ERR_CUDA;
  }
  return TUPS_OK;
}
