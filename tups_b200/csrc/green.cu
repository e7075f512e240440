// Green's function, chemical-potential bisection and G(r, tau):
// calc_Gkw_Grt (SRC/parquet_chi.f90:18-210), fftf2d/fftb2d (SRC/MATH_mod.f90:215-259).
#include "tups_device.cuh"

namespace tups {

// parquet_chi.f90:120 compares against the single-precision literal 1e-6
__device__ __constant__ double kMuTol = 9.999999974752427e-07;

// (G - G0)(nu) = 1/(z0 - Sigma) - 1/z0 = Sigma / ((z0 - Sigma) z0), z0 = i nu + mu - e:
// one reciprocal, and no cancellation of the two
__device__ __forceinline__ cplx green_minus_free(cplx sigma, double x0, double fr) {
  const cplx w = cmul(cmk(x0 - sigma.x, fr - sigma.y), cmk(x0, fr));
  return cscale(cmul(sigma, cconj(w)), __drcp_rn(cabs2(w)));
}

// The bisection in one CTA: each step needs only the particle number
// n = -2 Re G(r=0, tau=beta) = -2 * mean over fine k of G(k, tau=beta), the
// r = 0 term of fftf2d.  The loop is capped; on overrun S_STATUS is set.
//
// A step is a chain of latencies (reciprocal, exponentials, reduction), so a
// round evaluates the next LEV levels of the bisection tree at once, a group of
// warps per midpoint, and then walks down it: the same midpoints and decisions
// as one at a time, in a third (LEV = 3) of the rounds.  The terms of a
// midpoint are spread over (k, nu); what does not depend on mu is kept in
// shared memory when it fits (CACHED).  LEV by the number of terms: 3 up to 1024
// (4x4 x 16: 83 us -> 15), 2 up to 4096, else 1, where a round is bound by its
// FP64 work and more midpoints would only add to it.
constexpr int kBisectThreads = 1024;
constexpr int kBisectCache = 4096;  // terms kept in shared memory, 48 bytes each

template <int LEV, bool CACHED>
__global__ void __launch_bounds__(kBisectThreads) k_bisection(const cplx* __restrict__ Sigma,
                                                              const double* __restrict__ Ekg,
                                                              const cplx* __restrict__ tw_tau, double* scal, int Nx,
                                                              int Ny, int Nf, int Ng, double beta, double U,
                                                              double nParticle, int cal_chi, int max_steps) {
  constexpr int NODES = (1 << LEV) - 1, WPN = LEV == 1 ? 32 : LEV == 2 ? 8 : 4, TPN = 32 * WPN;
  extern __shared__ double cache[];  // CACHED: sigma re, im, tw Sigma / beta re, im, e, nu of every term
  __shared__ double sh[2][32];
  const int npts = Nx * Ny * Ng * Ng, terms = npts * Nf, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int node = warp / WPN, tn = tid % TPN;
  double *sr = cache, *si = cache + terms, *cr = cache + 2 * terms, *ci = cache + 3 * terms;
  double *en = cache + 4 * terms, *fq = cache + 5 * terms;
  // term i: point pt = i / Nf (kxc fastest, as Ek_grain is laid out), frequency i % Nf
  auto sigma_of = [&](int pt, int nu) {
    const int r = pt / (Ng * Ng), kx = r % Nx, ky = r / Nx;
    return Sigma[((size_t)kx * Ny + ky) * Nf + nu];
  };
  auto twist = [&](int nu) { return cscale(tw_tau[(Nf - 1) + (size_t)Nf * nu], 1.0 / beta); };  // tau = beta
  if (CACHED) {
    for (int i = tid; i < terms; i += kBisectThreads) {
      const int pt = i / Nf, nu = i % Nf;
      const cplx s = sigma_of(pt, nu), c = cmul(twist(nu), s);
      sr[i] = s.x;
      si[i] = s.y;
      cr[i] = c.x;
      ci[i] = c.y;
      en[i] = Ekg[pt];
      fq[i] = matsubara(nu + 1, Nf, beta);
    }
    __syncthreads();
  }
  const double tau = beta / (Nf - 1) * (Nf - 1);
  double mu = scal[S_MU];
  double up = mu + U, lo = mu - U;
  double t1 = 3.0;
  int steps = 0, status = 0, buf = 0;
  bool more = fabs(t1 - nParticle) > kMuTol;
  while (more) {
    // this group's midpoint: nodes 1, 2 follow the root's decision down, up;
    // 3, 4 and 5, 6 theirs
    double u = up, l = lo, m = 0.5 * (up + lo);
    if (LEV > 1 && node > 0) {
      const int first = node > 2 ? (node - 1) / 2 : node;
      if (first == 1) u = m;
      else l = m;
      m = 0.5 * (u + l);
      if (node > 2) {
        if (node & 1) u = m;
        else l = m;
        m = 0.5 * (u + l);
      }
    }
    double part = 0.0;
    if (node < NODES) {
      for (int i = tn; i < terms; i += TPN) {
        if (CACHED) {
          // Re of tw Sigma conj(w) / (|w|^2 beta)
          const double x0 = m - en[i], fr = fq[i];
          const cplx w = cmul(cmk(x0 - sr[i], fr - si[i]), cmk(x0, fr));
          part = fma(cr[i] * w.x + ci[i] * w.y, __drcp_rn(cabs2(w)), part);
        } else {
          const int pt = i / Nf, nu = i % Nf;
          part += cmul(twist(nu), green_minus_free(sigma_of(pt, nu), m - Ekg[pt], matsubara(nu + 1, Nf, beta))).x;
        }
      }
      for (int pt = tn; pt < npts; pt += TPN) {
        const double e = Ekg[pt];
        part -= exp((beta - tau) * (e - m)) / (1.0 + exp(beta * (e - m)));
      }
    }
    part = warp_sum(part);
    if (lane == 0) sh[buf][warp] = part;
    __syncthreads();
    double sum = sh[buf][lane];  // every warp adds up every midpoint
#pragma unroll
    for (int o = 1; o < WPN; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    buf ^= 1;
    int at = 0;
#pragma unroll
    for (int level = 0; level < LEV; level++) {
      if (steps >= max_steps) {
        status = TUPS_ERR_MU_NOCONV;
        more = false;
        break;
      }
      mu = 0.5 * (up + lo);
      const double tot = __shfl_sync(0xffffffffu, sum, at * WPN);
      t1 = -2.0 * (tot / (double)(Nx * Ng) / (double)(Ny * Ng));
      steps++;
      if (cal_chi) {
        more = false;
        break;
      }
      if (t1 > nParticle) up = mu;
      else lo = mu;
      at = 2 * at + (t1 > nParticle ? 1 : 2);
      if (!(fabs(t1 - nParticle) > kMuTol)) {
        more = false;
        break;
      }
    }
  }
  if (threadIdx.x == 0) {
    if (steps > 0) scal[S_MU] = mu;
    scal[S_T1] = t1;
    scal[S_STEPS] = (double)steps;
    if (status) scal[S_STATUS] = (double)status;
  }
}

// G(k, tau) on the fine grid for the final mu, one CTA per fine-grid point,
// one thread per tau (SRC/parquet_chi.f90:124-174):
// sum_nu Re(tw(tau,nu) (G - G0)(nu))/beta - exp((beta-tau)(e-mu))/(1+exp(beta(e-mu))).
// Output indexed by the fine-grid position (idx1, idx2) of
// parquet_chi.f90:135-139.  The CTAs past the points, if any, form
// G(k, nu) = 1/(i nu - e_k + mu - Sigma) (:203-210) and Sigma_H(kx, ky) =
// Sigma(k, nu = Nf) (:105-111): one launch instead of three.
constexpr int kGrtThreads = 64;
__global__ void __launch_bounds__(kGrtThreads) k_grt_points(const cplx* __restrict__ Sigma,
                                                            const double* __restrict__ Ekg,
                                                            const double* __restrict__ Ek,
                                                            const cplx* __restrict__ tw_tau,
                                                            const double* __restrict__ scal, cplx* __restrict__ out,
                                                            cplx* __restrict__ Gkw, cplx* __restrict__ SigmaH, int Nx,
                                                            int Ny, int Nf, int Ng, double beta) {
  extern __shared__ cplx gd[];
  const int pt = blockIdx.x, npts = Nx * Ny * Ng * Ng;
  const double mu = scal[S_MU];
  if (pt >= npts) {
    const int idx = (pt - npts) * kGrtThreads + threadIdx.x;
    if (idx >= Nx * Ny * Nf) return;
    const int nu = idx % Nf, k = idx / Nf, kx = k / Ny, ky = k % Ny;
    const cplx s = Sigma[idx];
    Gkw[idx] = crecip(cmk(0.0 - Ek[kx + Nx * ky] + mu - s.x, matsubara(nu + 1, Nf, beta) - s.y));
    if (nu == Nf - 1) SigmaH[kx + Nx * ky] = s;
    return;
  }
  int kxc = pt % Ng, r = pt / Ng;
  int kyc = r % Ng;
  r /= Ng;
  int kx = r % Nx, ky = r / Nx;
  const double e = Ekg[pt];
  const cplx* sg = Sigma + ((size_t)kx * Ny + ky) * Nf;
  for (int nu = threadIdx.x; nu < Nf; nu += kGrtThreads)
    gd[nu] = cscale(green_minus_free(sg[nu], mu - e, matsubara(nu + 1, Nf, beta)), 1.0 / beta);
  __syncthreads();
  int idx1 = kx * Ng + (kxc + 1 - (Ng + 1) / 2);
  if (idx1 < 0) idx1 += Ng * Nx;
  int idx2 = ky * Ng + (kyc + 1 - (Ng + 1) / 2);
  if (idx2 < 0) idx2 += Ng * Ny;
  const int n1 = Nx * Ng, n2 = Ny * Ng;
  const double occ = 1.0 + exp(beta * (e - mu));
  for (int it = threadIdx.x; it < Nf; it += kGrtThreads) {
    const double tau = beta / (Nf - 1) * it;
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    int nu = 0;
    for (; nu + 4 <= Nf; nu += 4)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const cplx t = tw_tau[it + (size_t)Nf * (nu + j)], g = gd[nu + j];
        a[j] = fma(t.x, g.x, fma(-t.y, g.y, a[j]));
      }
    for (; nu < Nf; nu++) a[0] += cmul(tw_tau[it + (size_t)Nf * nu], gd[nu]).x;
    const double v = (a[0] + a[1]) + (a[2] + a[3]) - exp((beta - tau) * (e - mu)) / occ;
    out[idx1 + (size_t)n1 * (idx2 + (size_t)n2 * it)] = cmk(v, 0.0);
  }
}

// 2D DFT of every (n1, n2) slice: forward (e^{-i}, divided by n1 and n2) as
// fftf2d, or backward (e^{+i}, unnormalised) as fftb2d.  One CTA per slice;
// first along dim 1 then dim 2, like the reference.
__global__ void k_fft2d(const cplx* __restrict__ in, cplx* __restrict__ out, const cplx* __restrict__ tw1,
                        const cplx* __restrict__ tw2, int n1, int n2, int forward) {
  extern __shared__ cplx buf[];
  cplx* a = buf;            // n1*n2
  cplx* b = buf + n1 * n2;  // n1*n2
  const size_t off = (size_t)blockIdx.x * n1 * n2;
  for (int i = threadIdx.x; i < n1 * n2; i += blockDim.x) a[i] = in[off + i];
  __syncthreads();
  const double s1 = forward ? 1.0 / n1 : 1.0, s2 = forward ? 1.0 / n2 : 1.0;
  for (int i = threadIdx.x; i < n1 * n2; i += blockDim.x) {
    int x = i % n1, col = i / n1;
    cplx acc = cmk(0.0, 0.0);
    for (int aa = 0; aa < n1; aa++) {
      cplx t = tw1[(aa * x) % n1];
      if (!forward) t = cconj(t);
      acc = cfma(a[aa + n1 * col], t, acc);
    }
    b[i] = cscale(acc, s1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n1 * n2; i += blockDim.x) {
    int x = i % n1, y = i / n1;
    cplx acc = cmk(0.0, 0.0);
    for (int bb = 0; bb < n2; bb++) {
      cplx t = tw2[(bb * y) % n2];
      if (!forward) t = cconj(t);
      acc = cfma(b[x + n1 * bb], t, acc);
    }
    out[off + i] = cscale(acc, s2);
  }
}

// mu <- 0.5*((mu+U)+(mu-U)): the first bisection midpoint of the readout's
// calc_Gkw_Grt(.true.) call (SRC/parquet_chi.f90:114-122)
__global__ void k_output_mu(double* scal, double U) {
  double mu = scal[S_MU];
  scal[S_MU] = 0.5 * ((mu + U) + (mu - U));
}

template <int LEV, bool CACHED>
static int run_bisection(tups_ctx* ctx, int cal_chi, int max_steps) {
  const auto& d = ctx->d;
  const int terms = d.Nc * d.Ngrain * d.Ngrain * d.Nf;
  const size_t sm = CACHED ? (size_t)6 * terms * sizeof(double) : 0;
  if (sm > 40 * 1024) {  // with the kernel's static shared memory past the default 48 KiB
    cudaError_t e = cudaFuncSetAttribute(k_bisection<LEV, CACHED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         6 * kBisectCache * (int)sizeof(double));
    if (e != cudaSuccess) return cuda_check(ctx, e, "k_bisection smem attribute");
  }
  k_bisection<LEV, CACHED><<<1, kBisectThreads, sm, ctx->stream>>>(
      ctx->s.Sigma, ctx->t.Ekg, ctx->t.tw_tau, ctx->s.scal, d.Nx, d.Ny, d.Nf, d.Ngrain, ctx->p.beta, ctx->p.U,
      ctx->p.nParticle, cal_chi, max_steps);
  return after_launch(ctx, "k_bisection");
}

int launch_bisection(tups_ctx* ctx, int cal_chi, int max_steps) {
  const auto& d = ctx->d;
  const long long terms = (long long)d.Nc * d.Ngrain * d.Ngrain * d.Nf;
  // the readout's bisection is a single step
  if (terms > kBisectCache) return run_bisection<1, false>(ctx, cal_chi, max_steps);
  if (cal_chi) return run_bisection<1, true>(ctx, cal_chi, max_steps);
  return terms <= 1024 ? run_bisection<3, true>(ctx, cal_chi, max_steps)
                       : run_bisection<2, true>(ctx, cal_chi, max_steps);
}

static int run_grt(tups_ctx* ctx, cplx* out, bool with_g) {
  const auto& d = ctx->d;
  const int npts = d.Nc * d.Ngrain * d.Ngrain;
  const int grid = npts + (with_g ? cdiv(d.Nt, kGrtThreads) : 0);
  k_grt_points<<<grid, kGrtThreads, d.Nf * sizeof(cplx), ctx->stream>>>(
      ctx->s.Sigma, ctx->t.Ekg, ctx->t.Ek, ctx->t.tw_tau, ctx->s.scal, out, ctx->s.Gkw, ctx->s.SigmaH, d.Nx, d.Ny, d.Nf,
      d.Ngrain, ctx->p.beta);
  return after_launch(ctx, "k_grt_points");
}

int launch_grt_pre(tups_ctx* ctx, cplx* out) { return run_grt(ctx, out, false); }

int launch_green(tups_ctx* ctx) {
  int rc = run_grt(ctx, ctx->s.Grt_work, true);
  if (rc) return rc;
  return launch_fft2d(ctx, ctx->s.Grt_work, ctx->s.Grt, 1);
}

int launch_fft2d_batch(tups_ctx* ctx, const cplx* in, cplx* out, int nslices, int forward) {
  const auto& d = ctx->d;
  const int n1 = d.Nx * d.Ngrain, n2 = d.Ny * d.Ngrain;
  size_t sm = 2 * (size_t)n1 * n2 * sizeof(cplx);
  if (sm > 200 * 1024) return set_error(ctx, TUPS_ERR_BADDIM, "fine k grid too large for the in-CTA DFT");
  if (sm > 48 * 1024) cudaFuncSetAttribute(k_fft2d, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_fft2d<<<nslices, 256, sm, ctx->stream>>>(in, out, ctx->t.tw_x, ctx->t.tw_y, n1, n2, forward);
  return after_launch(ctx, "k_fft2d");
}

int launch_fft2d(tups_ctx* ctx, const cplx* in, cplx* out, int forward) {
  return launch_fft2d_batch(ctx, in, out, ctx->d.Nf, forward);
}

int launch_output_mu(tups_ctx* ctx) {
  k_output_mu<<<1, 1, 0, ctx->stream>>>(ctx->s.scal, ctx->p.U);
  return after_launch(ctx, "k_output_mu");
}

}  // namespace tups
