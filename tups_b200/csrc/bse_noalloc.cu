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
// thread per (row, nu) line loads the line's Nl entries of Gamma once (NA_LMAX
// registers at a time) for its Nl outputs, lanes over rows at one nu, so a chi
// entry is one address per warp.  The rest form B: a warp per column, lanes
// over nu, chi[:, :, 32 nu] staged in shared memory ([l1 + Nl l2][lane], pitch
// 33) when it fits.
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
      for (int l = LMAX; l < Nl; l++) acc = tups::cfma(Gm[row + (size_t)Nz * (l * Nf + nu)], c[l], acc);
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
    for (int l = LMAX; l < Nl; l++) acc = tups::cfma(c(l), Gc[l * Nf], acc);
    Bc[l1 * Nf] = acc;
  }
}

// Phi = s [A | F] [F ; B] + (1-f)(F - Gamma) over Gamma, the BSE GEMM's tile with
// four real products per complex one (three measured 12 % less exact here)
constexpr int NB_BK = 16, NB_PER_SM = 4;
using NaTile = tups::ZgemmTile<1, 2, 2, 2, NB_BK, 3, false>;

__global__ void __launch_bounds__(NaTile::NT, NB_PER_SM) k_noalloc_gemm(cplx* __restrict__ G, const cplx* __restrict__ F,
                                                                        const cplx* __restrict__ A,
                                                                        const cplx* __restrict__ B, int i0, int Nz,
                                                                        double s, double one_minus_f) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int li = blockIdx.y;
  const size_t n2 = (size_t)Nz * Nz;
  const cplx* Fi = F + n2 * (i0 + li);
  cplx* Gi = G + n2 * (i0 + li);
  const int tiles_m = (Nz + NaTile::BM - 1) / NaTile::BM;
  const int m0 = (int)(blockIdx.x % tiles_m) * NaTile::BM, n0 = (int)(blockIdx.x / tiles_m) * NaTile::BN;
  NaTile t;
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
  // instances per pass through the scratch; the instance index is gridDim.y
  // of both kernels, at most 65535.  Of the pass sizes that fit, the one whose
  // GEMM grids fill their last waves best: 240 instances of Nz = 160 take 11
  // passes of 23 (0.97 waves each) instead of 6 of 40 (1.69)
  const size_t n2 = (size_t)Nz * Nz;
  const int cap = (int)std::min<size_t>(std::min<size_t>(kScratchComplex / per, 65535), (size_t)n_inst);
  const int tiles = ((Nz + NaTile::BM - 1) / NaTile::BM) * ((Nz + NaTile::BN - 1) / NaTile::BN);
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long slots = (long long)NB_PER_SM * sms;
  auto waves = [&](int chunk) {
    const long long full = (n_inst / chunk) * (((long long)chunk * tiles + slots - 1) / slots);
    return full + ((long long)(n_inst % chunk) * tiles + slots - 1) / slots;
  };
  int chunk = cap;
  for (int c = cap; c >= 1 && c > cap - 64 && 2 * c > cap; c--)
    if (waves(c) < waves(chunk)) chunk = c;
  cplx* A = scratch;
  cplx* B = scratch + (size_t)cap * n2;
  const int nA = (int)std::min<size_t>(((size_t)Nz * Nf + 255) / 256, 4096);
  const int nB = ((Nf + 31) / 32) * ((Nz + 7) / 8);
  const size_t smp = Nl <= NA_STAGE ? (size_t)Nl * Nl * 33 * sizeof(cplx) : 0;
  const auto prep = Nl <= 1 ? k_noalloc_prep<1> : Nl <= 5 ? k_noalloc_prep<5> : Nl <= 9 ? k_noalloc_prep<9>
                    : k_noalloc_prep<NA_LMAX>;
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if ((smp > 48 * 1024 && cudaFuncSetAttribute(prep, attr, (int)smp) != cudaSuccess) ||
      cudaFuncSetAttribute(k_noalloc_gemm, attr, (int)NaTile::kSmem) != cudaSuccess) {
    cudaGetLastError();
    return TUPS_ERR_CUDA;
  }
  for (int i0 = 0; i0 < n_inst; i0 += chunk) {
    const int n = n_inst - i0 < chunk ? n_inst - i0 : chunk;
    prep<<<dim3(nA + nB, n), 256, smp, st>>>(reinterpret_cast<const cplx*>(gamma_phi),
                                             reinterpret_cast<const cplx*>(chi), A, B, i0, Nz, Nf, Nl, nA);
    if (cudaGetLastError() != cudaSuccess) return TUPS_ERR_CUDA;
    k_noalloc_gemm<<<dim3(tiles, n), NaTile::NT, NaTile::kSmem, st>>>(
        reinterpret_cast<cplx*>(gamma_phi), reinterpret_cast<const cplx*>(F), A, B, i0, Nz, scale, 1.0 - f_damping);
    if (cudaGetLastError() != cudaSuccess) return TUPS_ERR_CUDA;
  }
  return TUPS_OK;
}
