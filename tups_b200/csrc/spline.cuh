// Clamped cubic spline through Nf equidistant samples on [0, beta] and its exact
// integral against e^{i om tau}: FDfit and nfourier (SRC/MATH_mod.f90:95-212),
// shared by the U^2 self-energy (odd frequencies) and the chi0 readout (even).
//
// One CTA per sample line.  The tridiagonal elimination's multipliers do not
// depend on the samples: they come from a table made with the context, so the
// serial part (thread 0) is one FMA per step and direction instead of two
// divisions.  The phases e^{i om tau_j} are a table as well, and eight lanes share
// a frequency's sum over the intervals.  At the lowest frequencies the terms of
// the sum are some thousand times its value, so phases, divisions by the powers
// of om and interval coefficients are rounded as the reference's formulas are.
#pragma once

#include "tups_device.cuh"

namespace tups {

struct SplineShared {
  double *r, *q, *ip, *u, *xm, *b, *d;
};

constexpr int kSplineLanes = 8;

__host__ __device__ inline size_t spline_smem(int Nf) {
  return (size_t)7 * Nf * sizeof(double);
}

// carve dynamic shared memory of spline_smem(Nf) bytes
__device__ __forceinline__ SplineShared spline_bind(void* sm, int Nf) {
  SplineShared S;
  double* p = static_cast<double*>(sm);
  S.r = p;
  S.q = p + Nf;
  S.ip = p + 2 * Nf;
  S.u = p + 3 * Nf;
  S.xm = p + 4 * Nf;
  S.b = p + 5 * Nf;
  S.d = p + 6 * Nf;
  return S;
}

// second derivatives and interval coefficients of the samples S.r (stored, not
// yet synchronised); tab = [q | 1/p] of the elimination, Nf each
__device__ __forceinline__ void spline_fit(const SplineShared& S, const double* __restrict__ tab, int Nf, double beta) {
  const int L = Nf - 1;
  const double delta = beta / L;
  for (int t = threadIdx.x; t < Nf; t += blockDim.x) {
    S.q[t] = tab[t];
    S.ip[t] = tab[Nf + t];
  }
  __syncthreads();
  const double* r = S.r;
  const double idd = 3.0 / (delta * delta);
  for (int k = threadIdx.x + 1; k < L; k += blockDim.x) S.u[k] = idd * (r[k + 1] + r[k - 1] - 2.0 * r[k]) * S.ip[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    // FDfit (SRC/MATH_mod.f90:95-107)
    const double fd1 = (-25.0 * r[0] + 48.0 * r[1] - 36.0 * r[2] + 16.0 * r[3] - 3.0 * r[4]) / 12.0 / delta;
    const double fd2 =
        (25.0 * r[L] - 48.0 * r[L - 1] + 36.0 * r[L - 2] - 16.0 * r[L - 3] + 3.0 * r[L - 4]) / 12.0 / delta;
    // spline second derivatives (SRC/MATH_mod.f90:140-168)
    double u = (3.0 / delta) * ((r[1] - r[0]) / delta - fd1);
    S.u[0] = u;
    for (int k = 1; k < L; k++) {
      u = fma(-0.5 * S.ip[k], u, S.u[k]);
      S.u[k] = u;
    }
    const double ul = (3.0 / delta) * (fd2 - (r[L] - r[L - 1]) / delta), ql = 0.5;
    double x = (ul - ql * u) / (ql * S.q[L - 1] + 1.0);
    S.xm[L] = x;
    for (int k = L; k >= 1; k--) {
      x = fma(S.q[k - 1], x, S.u[k - 1]);
      S.xm[k - 1] = x;
    }
  }
  __syncthreads();
  for (int j = threadIdx.x + 1; j <= L; j += blockDim.x) {
    S.b[j] = (r[j] - r[j - 1]) / delta - (2.0 * S.xm[j - 1] + S.xm[j]) * delta / 6.0;
    S.d[j] = (S.xm[j] - S.xm[j - 1]) / (6.0 * delta);
  }
  __syncthreads();
}

// integral of the spline against e^{i om tau} by a group of kSplineLanes
// consecutive lanes (SRC/MATH_mod.f90:170-212); ph[j] = e^{i om j delta}, j < Nf;
// every lane of the group gets the result.  All lanes of the warp call it.
__device__ __forceinline__ cplx spline_transform(const SplineShared& S, double om, const cplx* __restrict__ ph, int Nf,
                                                 double beta) {
  const int L = Nf - 1, part = threadIdx.x % kSplineLanes;
  const double delta = beta / L;
  const bool zero = fabs(om) < 1e-6;
  const double om2 = om * om, om3 = om2 * om, om4 = om3 * om;
  double cr = 0.0, ci = 0.0;
  for (int j = part + 1; j <= L; j += kSplineLanes) {
    const double a = S.r[j - 1], b = S.b[j], c = S.xm[j - 1] / 2.0, d = S.d[j];
    if (zero) {
      cr += a * delta + 0.5 * b * delta * delta + c * delta * delta * delta / 3.0 +
            d * delta * delta * delta * delta / 4.0;
      continue;
    }
    const cplx ep = ph[j], em = ph[j - 1];
    // explus*(p1r + i p1i) + ex*(p2r + i p2i), SRC/MATH_mod.f90:200-207
    const double d4 = 6.0 * d / om4;
    const double p1r = -d4 + (b + 2.0 * delta * c + 3.0 * delta * delta * d) / om2;
    const double p1i =
        (2.0 * c + 6.0 * delta * d) / om3 + (-a - delta * b - delta * delta * c - delta * delta * delta * d) / om;
    const double p2r = d4 - b / om2;
    const double p2i = -2.0 * c / om3 + a / om;
    cr += ep.x * p1r - ep.y * p1i + em.x * p2r - em.y * p2i;
    ci += ep.x * p1i + ep.y * p1r + em.x * p2i + em.y * p2r;
  }
#pragma unroll
  for (int o = kSplineLanes / 2; o > 0; o >>= 1) {
    cr += __shfl_xor_sync(0xffffffffu, cr, o);
    ci += __shfl_xor_sync(0xffffffffu, ci, o);
  }
  return cmk(cr, ci);
}

}  // namespace tups
