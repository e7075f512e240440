// Multilayer perceptron of the learned warm start: forward, backward and Adam
// in FP32 on the device.  No counterpart in the reference.
//
// Network: n_in -> H -> ... -> H (n_layers hidden layers, SiLU) -> n_out
// (linear).  Layer l holds W_l (out_l, in_l) row-major and b_l (out_l); the
// flat parameter vector is [W_0, b_0, W_1, b_1, ...].  Loss: mean squared
// error over batch x n_out.  Batches are row-major (batch, features).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "../../include/tups_b200.h"

struct tups_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string err;
  long long launches = 0;
  int n_in = 0, n_hidden = 0, n_layers = 0, n_out = 0, max_batch = 0;
  std::vector<int> width;      // n_layers + 2 entries: n_in, H, ..., H, n_out
  std::vector<size_t> w_off;   // offset of W_l in the flat vector
  std::vector<size_t> b_off;   // offset of b_l
  size_t n_params = 0;
  float* params = nullptr;
  float* grads = nullptr;
  float* adam_m = nullptr;
  float* adam_v = nullptr;
  long long adam_t = 0;
  float* x = nullptr;          // input batch (max_batch, n_in)
  float* t = nullptr;          // target batch (max_batch, n_out)
  std::vector<float*> z, a;    // per hidden layer: pre-activation, activation
  float* y = nullptr;          // output (max_batch, n_out)
  std::vector<float*> dz;      // per linear layer: gradient of its output (max_batch, width)
  double* loss = nullptr;      // device loss slots
  int loss_slots = 0;
  float* data_x = nullptr;     // resident training set
  float* data_t = nullptr;
  int data_n = 0;
  int* idx = nullptr;          // minibatch row indices
  std::vector<void*> allocs;
};

namespace {

int mlp_error(tups_mlp* m, int code, const std::string& msg) {
  if (m) m->err = msg;
  return code;
}

int mlp_cuda(tups_mlp* m, cudaError_t e, const char* what) {
  if (e == cudaSuccess) return TUPS_OK;
  return mlp_error(m, e == cudaErrorMemoryAllocation ? TUPS_ERR_OOM : TUPS_ERR_CUDA,
                   std::string(what) + ": " + cudaGetErrorString(e));
}

#define MTRY(x)                     \
  do {                              \
    int _rc = (x);                  \
    if (_rc != TUPS_OK) return _rc; \
  } while (0)

template <typename T>
int mlp_alloc(tups_mlp* m, T** p, size_t count) {
  cudaError_t e = cudaMalloc((void**)p, count * sizeof(T) + 16);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return mlp_error(m, TUPS_ERR_OOM, "MLP device allocation failed");
  }
  m->allocs.push_back(*p);
  return TUPS_OK;
}

__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

// 4 floats of a row from k on, those past len (and, with !in, all) as zeros
__device__ __forceinline__ void cp_async4(float* dst, const float* src, int k, int len, bool vec, bool in) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  if (vec) {
    const unsigned sz = in && k < len ? 16u : 0u;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(sz ? src + k : src), "r"(sz));
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const unsigned sz = in && k + i < len ? 4u : 0u;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d + 4 * i), "l"(sz ? src + k + i : src),
                   "r"(sz));
    }
  }
}

// ---- layer products: C(m, n) = sum_k X(m, k) W(k, n) ------------------------------
//
// A minibatch has few rows (32 in training), so a layer is a thin product bound
// by latency: 32 x 16 output tiles, and the sum over k split over the four CTAs
// of a cluster (partial tiles added through distributed shared memory, in rank
// order) and over the eight warps of a CTA, each thread 4 x 4 outputs over
// float4 steps of k.  A CTA loads its whole k range (up to kKC) at once.
//   forward (WT = false): W(k, n) = W[n * ldw + k], rows of W along k
//   backward (WT = true): W(k, n) = W[k * ldw + n]
// rows: optional gather of X's rows by index.
// 964 -> 512 at 32 rows: 120 -> 8 us (eight CTAs of 64 x 64 before); 20 training
// steps of 964 -> 3 x 512 -> 968 at 32 rows with their uploads: 13.7 -> 1.73 ms.
enum { EPI_BIAS_SILU = 1, EPI_BIAS = 2, EPI_DSILU = 3, EPI_MSE = 4 };

struct LinArgs {
  int M, N, K;
  const float* X;
  const int* rows;
  const int* trows;   // the same of the targets
  const float* W;
  const float* bias;  // EPI_BIAS*, EPI_MSE
  const float* aux;   // EPI_DSILU: z (M, N); EPI_MSE: targets
  float* C;           // pre-activation, output or gradient (M, N)
  float* C2;          // EPI_BIAS_SILU: silu(C)
  double* loss;       // EPI_MSE: += sum (y - t)^2 / (M N); C = 2 (y - t) / (M N)
  double inv;
  bool w_fresh;       // W may have been written by the launch just before
};

// Programmatic dependent launch: a kernel starts while its predecessor drains,
// loads what that one does not write and then waits for it.  Dependents are
// released after the wait, so at any kernel's start everything up to its
// predecessor's predecessor is complete.
__device__ __forceinline__ void wait_predecessor() {
  asm volatile("griddepcontrol.wait;\ngriddepcontrol.launch_dependents;\n" ::: "memory");
}

// the output at offset o from its sum v; bias and aux as the epilogue reads them.
// Returns the squared error (EPI_MSE).
template <int EPI>
__device__ __forceinline__ double store(const LinArgs& a, size_t o, float v, float bias, float aux) {
  if (EPI == EPI_BIAS_SILU) {
    v += bias;
    a.C[o] = v;
    a.C2[o] = v * sigmoid(v);
  } else if (EPI == EPI_BIAS) {
    a.C[o] = v + bias;
  } else if (EPI == EPI_DSILU) {
    const float s = sigmoid(aux);
    a.C[o] = v * (s * (1.0f + aux * (1.0f - s)));
  } else {
    const float d = v + bias - aux;
    a.C[o] = (float)(2.0 * a.inv) * d;
    return (double)d * d;
  }
  return 0.0;
}

constexpr int kTM = 32, kTN = 16, kKC = 256, kSplit = 4, kLinThreads = 256;
constexpr int kXP = kKC + 4, kWP = kTN + 4;  // pitches: float4 rows on distinct banks
constexpr size_t kLinSmem = ((size_t)(kTM + kTN) * kXP > (size_t)kTM * kXP + (size_t)kKC * kWP
                                 ? (size_t)(kTM + kTN) * kXP : (size_t)kTM * kXP + (size_t)kKC * kWP) * sizeof(float);

template <int EPI, bool WT>
__global__ void __cluster_dims__(kSplit, 1, 1) __launch_bounds__(kLinThreads) k_mlp_linear(LinArgs a) {
  extern __shared__ __align__(16) float sm[];
  float* Xs = sm;             // [m][k]
  float* Ws = sm + kTM * kXP; // [n][k], WT: [k][n]
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int n0 = (int)(blockIdx.x / kSplit) * kTN, m0 = (int)blockIdx.y * kTM;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kper = ((a.K + kSplit - 1) / kSplit + 31) / 32 * 32;
  const int kbeg = rank * kper, kend = min(a.K, kbeg + kper);
  const bool xv = a.K % 4 == 0 && (reinterpret_cast<size_t>(a.X) & 15) == 0;
  const bool wv = (WT ? a.N : a.K) % 4 == 0 && (reinterpret_cast<size_t>(a.W) & 15) == 0;
  const int g = lane >> 2, q = lane & 3;
  float acc[4][4] = {};
  // a row is up to 64 float4 steps of k: 64 threads per row, all copies in flight at once
  const int k = tid % (kKC / 4) * 4, r0 = tid / (kKC / 4);
  constexpr int kRows = kLinThreads / (kKC / 4);
  auto load_w = [&](int kc) {
    const int len = min(kKC, kend - kc), len4 = (len + 3) / 4;
    if (!WT && k < 4 * len4) {
#pragma unroll
      for (int i = 0; i < kTN / kRows; i++) {
        const int n = r0 + i * kRows;
        const bool in = n0 + n < a.N;
        cp_async4(Ws + n * kXP + k, in ? a.W + (size_t)(n0 + n) * a.K + kc : a.W, k, len, wv, in);
      }
    }
    if (WT) {
      const int n = tid % (kTN / 4) * 4, left = min(kTN, a.N - n0);
      for (int kk = tid / (kTN / 4); kk < 4 * len4; kk += kLinThreads / (kTN / 4))
        cp_async4(Ws + kk * kWP + n, kk < len ? a.W + (size_t)(kc + kk) * a.N + n0 : a.W, n, left, wv, kk < len);
    }
  };
  if (!a.w_fresh && kbeg < kend) load_w(kbeg);
  wait_predecessor();
  // what this thread's output needs besides the product, ahead of it
  constexpr int kTile = kTM * kTN, kOwn = kTile / kSplit;  // each CTA finishes a quarter of the rows
  const int eo = rank * kOwn + tid, mo = m0 + eo / kTN, no = n0 + eo % kTN;
  const bool own = tid < kOwn && mo < a.M && no < a.N;
  const size_t oo = (size_t)mo * a.N + no;
  float bias = 0.0f, aux = 0.0f;
  if (own) {
    if (EPI != EPI_DSILU) bias = a.bias[no];
    if (EPI == EPI_DSILU) aux = a.aux[oo];
    if (EPI == EPI_MSE) aux = a.aux[a.trows ? (size_t)a.trows[mo] * a.N + no : oo];
  }
  for (int kc = kbeg; kc < kend; kc += kKC) {
    const int len = min(kKC, kend - kc), len4 = (len + 3) / 4;
    if (kc > kbeg) __syncthreads();
    if (kc > kbeg || a.w_fresh) load_w(kc);
    if (k < 4 * len4) {
#pragma unroll
      for (int i = 0; i < kTM / kRows; i++) {
        const int m = r0 + i * kRows;
        const bool in = m0 + m < a.M;
        const float* src = a.X;
        if (in) src += (size_t)(a.rows ? a.rows[m0 + m] : m0 + m) * a.K + kc;
        cp_async4(Xs + m * kXP + k, src, k, len, xv, in);
      }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    for (int k4 = warp; k4 < len4; k4 += kLinThreads / 32) {
      float4 x[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; i++) x[i] = *reinterpret_cast<const float4*>(Xs + (g + 8 * i) * kXP + 4 * k4);
#pragma unroll
      for (int j = 0; j < 4; j++)
        w[j] = *reinterpret_cast<const float4*>(WT ? Ws + (4 * k4 + j) * kWP + 4 * q : Ws + (q + 4 * j) * kXP + 4 * k4);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (WT) {
          const float xk[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            acc[i][0] = fmaf(xk[k], w[k].x, acc[i][0]);
            acc[i][1] = fmaf(xk[k], w[k].y, acc[i][1]);
            acc[i][2] = fmaf(xk[k], w[k].z, acc[i][2]);
            acc[i][3] = fmaf(xk[k], w[k].w, acc[i][3]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            acc[i][j] = fmaf(x[i].x, w[j].x, acc[i][j]);
            acc[i][j] = fmaf(x[i].y, w[j].y, acc[i][j]);
            acc[i][j] = fmaf(x[i].z, w[j].z, acc[i][j]);
            acc[i][j] = fmaf(x[i].w, w[j].w, acc[i][j]);
          }
        }
      }
    }
  }
  // the warps' partial tiles, then the cluster's
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) sm[warp * kTile + (g + 8 * i) * kTN + (WT ? 4 * q + j : q + 4 * j)] = acc[i][j];
  __syncthreads();
  float* part = sm + (kLinThreads / 32) * kTile;
  for (int e = tid; e < kTile; e += kLinThreads) {
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < kLinThreads / 32; w++) v += sm[w * kTile + e];
    part[e] = v;
  }
  cluster.sync();
  double sq = 0.0;
  if (own) {
    float v = 0.0f;
#pragma unroll
    for (int r = 0; r < kSplit; r++) v += cluster.map_shared_rank(part, r)[eo];
    sq = store<EPI>(a, oo, v, bias, aux);
  }
  if (EPI == EPI_MSE && tid < kOwn) {
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (lane == 0) atomicAdd(a.loss, sq * a.inv);
  }
  cluster.sync();  // the partial tile stays until every rank has read it
}

// The same product for batches of a thousand rows and more: a CTA per 64 x 64
// tile, the whole sum over k in steps of 16, 4 x 4 outputs per thread.  Bound by
// the FP32 pipe and shared memory, where the form above repeats W for every 32
// rows and adds up 32 partial tiles per output.  A forward pass and copies of
// 64 -> 3 x 512 -> 68 at 768, 1024, 4096, 16384 rows: 280, 292, 628, 1786 us
// against 255, 324, 1148, 4278 with the split sums; 200 -> 6 x 128 -> 204: 323,
// 374, 829, 2709 against 293, 409, 1208, 4454; so the line lies at 1024 rows.
constexpr int kBigTile = 64, kBigStep = 16, kBigRows = 1024;

template <int EPI, bool WT>
__global__ void __launch_bounds__(kLinThreads) k_mlp_tile(LinArgs a) {
  __shared__ float Xs[kBigStep][kBigTile + 4];
  __shared__ float Ws[kBigStep][kBigTile + 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, tiles_n = (a.N + kBigTile - 1) / kBigTile;
  const int n0 = (int)blockIdx.x % tiles_n * kBigTile, m0 = (int)blockIdx.x / tiles_n * kBigTile;
  wait_predecessor();
  // this thread's rows of X and the places it fills
  constexpr int kPer = kBigTile * kBigStep / kLinThreads;
  const float* x[kPer];
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const int m = m0 + ty + 16 * i;
    x[i] = m < a.M ? a.X + (size_t)(a.rows ? a.rows[m] : m) * a.K : nullptr;
  }
  float acc[4][4] = {};
  for (int k0 = 0; k0 < a.K; k0 += kBigStep) {
#pragma unroll
    for (int i = 0; i < kPer; i++) {
      Xs[tx][ty + 16 * i] = x[i] && k0 + tx < a.K ? x[i][k0 + tx] : 0.0f;
      if (WT) {  // W(k, n), n fastest
        const int e = tid + i * kLinThreads, k = k0 + e / kBigTile, n = n0 + e % kBigTile;
        Ws[e / kBigTile][e % kBigTile] = k < a.K && n < a.N ? a.W[(size_t)k * a.N + n] : 0.0f;
      } else {   // k fastest
        const int n = n0 + ty + 16 * i;
        Ws[tx][ty + 16 * i] = n < a.N && k0 + tx < a.K ? a.W[(size_t)n * a.K + k0 + tx] : 0.0f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kBigStep; k++) {
      float u[4], v[4];
#pragma unroll
      for (int i = 0; i < 4; i++) u[i] = Xs[k][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = Ws[k][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(u[i], v[j], acc[i][j]);
    }
    __syncthreads();
  }
  double sq = 0.0;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int mo = m0 + ty + 16 * i, no = n0 + tx + 16 * j;
      if (mo >= a.M || no >= a.N) continue;
      const size_t o = (size_t)mo * a.N + no;
      const float bias = EPI != EPI_DSILU ? a.bias[no] : 0.0f;
      float aux = 0.0f;
      if (EPI == EPI_DSILU) aux = a.aux[o];
      if (EPI == EPI_MSE) aux = a.aux[a.trows ? (size_t)a.trows[mo] * a.N + no : o];
      sq += store<EPI>(a, o, acc[i][j], bias, aux);
    }
  if (EPI == EPI_MSE) {
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((tid & 31) == 0) atomicAdd(a.loss, sq * a.inv);
  }
}

// ---- gradients of all layers, and the Adam step on them ------------------------------
//
// dW_l(o, i) = sum_b dZ_l[b, o] X_l[b, i] and db_l(o) = sum_b dZ_l[b, o], one
// launch over the 32 x 64 tiles of every layer; with ADAM the tile steps its
// parameters at once (Kingma & Ba 2015, bias-corrected step lr_t, decoupled
// weight decay on W only, Loshchilov & Hutter 2019) instead of storing the
// gradient: parameters and moments are read and written once.
constexpr int kMaxLinear = 17, kGradTO = 32;

struct GradLayer {
  const float* dz;    // (M, fout)
  const float* in;    // (., fin)
  const int* rows;    // optional gather of in's rows
  int fout, fin, tile0, tiles_i;
  size_t w_off, b_off;
};

struct GradArgs {
  GradLayer l[kMaxLinear];
  int layers, M;
  float* grads;              // ADAM = false
  float *p, *m, *v;          // ADAM = true
  float lr_t, b1, b2, eps_t, decay;
};

// one step of parameter p with moments m and v
__device__ __forceinline__ void adam(const GradArgs& a, float g, float decay, float& p, float& m, float& v) {
  m = a.b1 * m + (1.0f - a.b1) * g;
  v = a.b2 * v + (1.0f - a.b2) * g * g;
  p = p * decay - a.lr_t * m / (sqrtf(v) + a.eps_t);
}

template <bool ADAM>
__global__ void __launch_bounds__(kLinThreads, 4) k_mlp_grad(const __grid_constant__ GradArgs a) {
  constexpr int TO = kGradTO, TI = 64, KB = 32, PER = TO / 8;
  __shared__ __align__(16) float Ds[KB][TO];
  __shared__ __align__(16) float Is[KB][TI];
  int l = 0;
  while (l + 1 < a.layers && (int)blockIdx.x >= a.l[l + 1].tile0) l++;
  const GradLayer& L = a.l[l];
  const int t = (int)blockIdx.x - L.tile0;
  const int o0 = t / L.tiles_i * TO, i0 = t % L.tiles_i * TI;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool bias = i0 == 0 && tid < TO;
  float acc[PER][2] = {}, bsum = 0.0f;
  // the tile's parameters and moments do not depend on the gradient: their
  // loads go out first
  float p[PER][2], m[PER][2], v[PER][2];
  if (ADAM) {
#pragma unroll
    for (int k = 0; k < PER; k++)
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int o = o0 + warp * PER + k, i = i0 + lane + 32 * j;
        if (o < L.fout && i < L.fin) {
          const size_t w = L.w_off + (size_t)o * L.fin + i;
          p[k][j] = a.p[w];
          m[k][j] = a.m[w];
          v[k][j] = a.v[w];
        }
      }
  }
  wait_predecessor();
  for (int b0 = 0; b0 < a.M; b0 += KB) {
    if (b0 > 0) __syncthreads();
    const int nb = min(KB, a.M - b0);
#pragma unroll
    for (int e = tid; e < KB * TO; e += 256) {
      const int b = e / TO, c = e % TO;
      Ds[b][c] = b < nb && o0 + c < L.fout ? L.dz[(size_t)(b0 + b) * L.fout + o0 + c] : 0.0f;
    }
#pragma unroll
    for (int e = tid; e < KB * TI; e += 256) {
      const int b = e / TI, c = e % TI;
      Is[b][c] = b < nb && i0 + c < L.fin
                     ? L.in[(size_t)(L.rows ? L.rows[b0 + b] : b0 + b) * L.fin + i0 + c] : 0.0f;
    }
    __syncthreads();
#pragma unroll 8
    for (int b = 0; b < nb; b++) {
      const float4 d0 = *reinterpret_cast<const float4*>(&Ds[b][warp * PER]);
      const float d[PER] = {d0.x, d0.y, d0.z, d0.w};
      const float x0 = Is[b][lane], x1 = Is[b][lane + 32];
#pragma unroll
      for (int k = 0; k < PER; k++) {
        acc[k][0] = fmaf(d[k], x0, acc[k][0]);
        acc[k][1] = fmaf(d[k], x1, acc[k][1]);
      }
    }
    if (bias)
      for (int b = 0; b < nb; b++) bsum += Ds[b][tid];
  }
#pragma unroll
  for (int k = 0; k < PER; k++)
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int o = o0 + warp * PER + k, i = i0 + lane + 32 * j;
      if (o < L.fout && i < L.fin) {
        const size_t w = L.w_off + (size_t)o * L.fin + i;
        if (ADAM) {
          adam(a, acc[k][j], a.decay, p[k][j], m[k][j], v[k][j]);
          a.p[w] = p[k][j];
          a.m[w] = m[k][j];
          a.v[w] = v[k][j];
        } else {
          a.grads[w] = acc[k][j];
        }
      }
    }
  if (bias && o0 + tid < L.fout) {
    const size_t w = L.b_off + o0 + tid;
    if (ADAM) {
      float bp = a.p[w], bm = a.m[w], bv = a.v[w];
      adam(a, bsum, 1.0f, bp, bm, bv);
      a.p[w] = bp;
      a.m[w] = bm;
      a.v[w] = bv;
    } else {
      a.grads[w] = bsum;
    }
  }
}

template <class Args>
int launch_dependent(tups_mlp* m, const char* name, void (*kernel)(Args), dim3 grid, size_t smem, const Args& a) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kLinThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = m->stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  m->launches++;
  return mlp_cuda(m, cudaLaunchKernelEx(&cfg, kernel, a), name);
}

template <int EPI, bool WT>
int linear(tups_mlp* m, const LinArgs& a) {
  if (a.M >= kBigRows) {
    const long long tiles = ((a.M + kBigTile - 1LL) / kBigTile) * ((a.N + kBigTile - 1) / kBigTile);
    return launch_dependent(m, "k_mlp_tile", k_mlp_tile<EPI, WT>, dim3((unsigned)tiles), 0, a);
  }
  const dim3 grid((unsigned)((a.N + kTN - 1) / kTN * kSplit), (unsigned)((a.M + kTM - 1) / kTM));
  return launch_dependent(m, "k_mlp_linear", k_mlp_linear<EPI, WT>, grid, kLinSmem, a);
}

// opt-in shared memory of every instantiation that linear() launches
int linear_prepare(tups_mlp* m) {
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  MTRY(mlp_cuda(m, cudaFuncSetAttribute(k_mlp_linear<EPI_BIAS_SILU, false>, attr, (int)kLinSmem), "k_mlp_linear"));
  MTRY(mlp_cuda(m, cudaFuncSetAttribute(k_mlp_linear<EPI_BIAS, false>, attr, (int)kLinSmem), "k_mlp_linear"));
  MTRY(mlp_cuda(m, cudaFuncSetAttribute(k_mlp_linear<EPI_MSE, false>, attr, (int)kLinSmem), "k_mlp_linear"));
  return mlp_cuda(m, cudaFuncSetAttribute(k_mlp_linear<EPI_DSILU, true>, attr, (int)kLinSmem), "k_mlp_linear");
}

int n_linear(const tups_mlp* m) { return m->n_layers + 1; }

// forward of `batch` rows of x (gathered by rows, or consecutive); the last
// layer gives m->y, or with targets t the loss into loss and its gradient
// with respect to the output
int forward(tups_mlp* m, int batch, const float* x, const int* rows, const float* t, double* loss) {
  const float* in = x;
  for (int l = 0; l < n_linear(m); l++) {
    LinArgs a{};
    a.M = batch;
    a.N = m->width[l + 1];
    a.K = m->width[l];
    a.X = in;
    a.rows = l == 0 ? rows : nullptr;
    a.w_fresh = l == 0;  // the previous step's update
    a.W = m->params + m->w_off[l];
    a.bias = m->params + m->b_off[l];
    if (l < m->n_layers) {
      a.C = m->z[l];
      a.C2 = m->a[l];
      MTRY((linear<EPI_BIAS_SILU, false>(m, a)));
      in = m->a[l];
    } else if (!t) {
      a.C = m->y;
      MTRY((linear<EPI_BIAS, false>(m, a)));
    } else {
      a.C = m->dz[l];
      a.aux = t;
      a.trows = rows;
      a.loss = loss;
      a.inv = 1.0 / ((double)batch * m->n_out);
      MTRY((linear<EPI_MSE, false>(m, a)));
    }
  }
  return TUPS_OK;
}

// gradients of the batch whose forward (with targets) just ran: into m->grads,
// or with `adam` as one step of it
int backward(tups_mlp* m, int batch, const float* x, const int* rows, bool adam, float lr, float weight_decay) {
  for (int l = n_linear(m) - 1; l > 0; l--) {
    // dZ_{l-1}(b, i) = sum_o dZ_l[b, o] W_l[o, i] silu'(Z_{l-1}(b, i))
    LinArgs a{};
    a.M = batch;
    a.N = m->width[l];
    a.K = m->width[l + 1];
    a.X = m->dz[l];
    a.W = m->params + m->w_off[l];
    a.aux = m->z[l - 1];
    a.C = m->dz[l - 1];
    MTRY((linear<EPI_DSILU, true>(m, a)));
  }
  GradArgs g{};
  g.layers = n_linear(m);
  g.M = batch;
  int tiles = 0;
  for (int l = 0; l < g.layers; l++) {
    GradLayer& L = g.l[l];
    L.dz = m->dz[l];
    L.in = l == 0 ? x : m->a[l - 1];
    L.rows = l == 0 ? rows : nullptr;
    L.fout = m->width[l + 1];
    L.fin = m->width[l];
    L.tile0 = tiles;
    L.tiles_i = (L.fin + 63) / 64;
    L.w_off = m->w_off[l];
    L.b_off = m->b_off[l];
    tiles += (L.fout + kGradTO - 1) / kGradTO * L.tiles_i;
  }
  g.grads = m->grads;
  if (adam) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    m->adam_t++;
    const double bc1 = 1.0 - std::pow((double)b1, (double)m->adam_t);
    const double bc2 = 1.0 - std::pow((double)b2, (double)m->adam_t);
    // step with bias correction folded into the step size and epsilon
    g.p = m->params;
    g.m = m->adam_m;
    g.v = m->adam_v;
    g.b1 = b1;
    g.b2 = b2;
    g.lr_t = (float)(lr * std::sqrt(bc2) / bc1);
    g.eps_t = (float)(eps * std::sqrt(bc2));
    g.decay = weight_decay > 0.0f ? 1.0f - lr * weight_decay : 1.0f;
    return launch_dependent(m, "k_mlp_grad", k_mlp_grad<true>, dim3(tiles), 0, g);
  }
  return launch_dependent(m, "k_mlp_grad", k_mlp_grad<false>, dim3(tiles), 0, g);
}

int h2d(tups_mlp* m, void* dst, const void* src, size_t bytes) {
  if (!src) return mlp_error(m, TUPS_ERR_BADARG, "NULL host buffer");
  return mlp_cuda(m, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, m->stream), "H2D");
}

int d2h(tups_mlp* m, void* dst, const void* src, size_t bytes) {
  if (!dst) return mlp_error(m, TUPS_ERR_BADARG, "NULL host buffer");
  MTRY(mlp_cuda(m, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, m->stream), "D2H"));
  return mlp_cuda(m, cudaStreamSynchronize(m->stream), "synchronize");
}

int set_dev(tups_mlp* m) { return mlp_cuda(m, cudaSetDevice(m->device), "cudaSetDevice"); }

int check_batch(tups_mlp* m, int batch) {
  if (batch < 1 || batch > m->max_batch) return mlp_error(m, TUPS_ERR_BADDIM, "batch outside 1..max_batch");
  return TUPS_OK;
}

// splitmix64 for the minibatch shuffles
uint64_t mix64(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

void free_mlp(tups_mlp* m) {
  for (void* p : m->allocs) cudaFree(p);
  m->allocs.clear();
  if (m->stream) cudaStreamDestroy(m->stream);
  m->stream = nullptr;
}

}  // namespace

extern "C" int tups_mlp_create(int n_in, int n_hidden, int n_layers, int n_out, int max_batch, int device,
                               tups_mlp** out) {
  if (!out) return TUPS_ERR_BADARG;
  *out = nullptr;
  if (n_in < 1 || n_hidden < 1 || n_layers < 1 || n_out < 1 || max_batch < 1 || n_layers > 16)
    return TUPS_ERR_BADDIM;
  tups_mlp* m = new tups_mlp();
  m->device = device;
  m->n_in = n_in;
  m->n_hidden = n_hidden;
  m->n_layers = n_layers;
  m->n_out = n_out;
  m->max_batch = max_batch;
  m->width.push_back(n_in);
  for (int l = 0; l < n_layers; l++) m->width.push_back(n_hidden);
  m->width.push_back(n_out);
  size_t off = 0;
  for (int l = 0; l <= n_layers; l++) {
    m->w_off.push_back(off);
    off += (size_t)m->width[l] * m->width[l + 1];
    m->b_off.push_back(off);
    off += (size_t)m->width[l + 1];
  }
  m->n_params = off;
  int rc = set_dev(m);
  if (!rc) rc = mlp_cuda(m, cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking), "stream");
  if (!rc) rc = linear_prepare(m);
  // every buffer of the network in one allocation (one cudaMalloc and one
  // cudaFree instead of one per buffer)
  m->z.assign(n_layers, nullptr);
  m->a.assign(n_layers, nullptr);
  m->dz.assign(n_layers + 1, nullptr);
  std::vector<std::pair<float**, size_t>> want = {
      {&m->params, m->n_params}, {&m->grads, m->n_params}, {&m->adam_m, m->n_params}, {&m->adam_v, m->n_params},
      {&m->x, (size_t)max_batch * n_in}, {&m->t, (size_t)max_batch * n_out}, {&m->y, (size_t)max_batch * n_out}};
  for (int l = 0; l < n_layers; l++) {
    want.push_back({&m->z[l], (size_t)max_batch * n_hidden});
    want.push_back({&m->a[l], (size_t)max_batch * n_hidden});
  }
  for (int l = 0; l <= n_layers; l++) want.push_back({&m->dz[l], (size_t)max_batch * m->width[l + 1]});
  size_t total = 0;
  for (const auto& w : want) total += (w.second + 63) / 64 * 64;
  float* arena = nullptr;
  if (!rc) rc = mlp_alloc(m, &arena, total);
  for (const auto& w : want) {
    *w.first = arena;
    if (arena) arena += (w.second + 63) / 64 * 64;
  }
  if (!rc) rc = mlp_cuda(m, cudaMemsetAsync(m->params, 0, m->n_params * sizeof(float), m->stream), "memset");
  if (!rc) rc = mlp_cuda(m, cudaMemsetAsync(m->adam_m, 0, m->n_params * sizeof(float), m->stream), "memset");
  if (!rc) rc = mlp_cuda(m, cudaMemsetAsync(m->adam_v, 0, m->n_params * sizeof(float), m->stream), "memset");
  if (!rc) rc = mlp_cuda(m, cudaStreamSynchronize(m->stream), "synchronize");
  if (rc) {
    free_mlp(m);
    delete m;
    return rc;
  }
  *out = m;
  return TUPS_OK;
}

extern "C" int tups_mlp_destroy(tups_mlp* m) {
  if (!m) return TUPS_OK;
  cudaSetDevice(m->device);
  free_mlp(m);
  delete m;
  return TUPS_OK;
}

extern "C" const char* tups_mlp_last_error(const tups_mlp* m) { return m ? m->err.c_str() : "NULL MLP"; }

extern "C" long long tups_mlp_num_params(const tups_mlp* m) { return m ? (long long)m->n_params : -1; }

extern "C" long long tups_mlp_kernel_launches(const tups_mlp* m) { return m ? m->launches : -1; }

extern "C" int tups_mlp_set_params(tups_mlp* m, const float* host) {
  if (!m) return TUPS_ERR_BADARG;
  MTRY(set_dev(m));
  MTRY(h2d(m, m->params, host, m->n_params * sizeof(float)));
  // a new parameter set restarts the optimiser
  MTRY(mlp_cuda(m, cudaMemsetAsync(m->adam_m, 0, m->n_params * sizeof(float), m->stream), "memset"));
  MTRY(mlp_cuda(m, cudaMemsetAsync(m->adam_v, 0, m->n_params * sizeof(float), m->stream), "memset"));
  m->adam_t = 0;
  return mlp_cuda(m, cudaStreamSynchronize(m->stream), "synchronize");
}

extern "C" int tups_mlp_get_params(tups_mlp* m, float* host) {
  if (!m) return TUPS_ERR_BADARG;
  MTRY(set_dev(m));
  return d2h(m, host, m->params, m->n_params * sizeof(float));
}

extern "C" int tups_mlp_forward(tups_mlp* m, const float* x, int batch, float* y) {
  if (!m) return TUPS_ERR_BADARG;
  MTRY(set_dev(m));
  MTRY(check_batch(m, batch));
  MTRY(h2d(m, m->x, x, (size_t)batch * m->n_in * sizeof(float)));
  MTRY(forward(m, batch, m->x, nullptr, nullptr, nullptr));
  return d2h(m, y, m->y, (size_t)batch * m->n_out * sizeof(float));
}

extern "C" int tups_mlp_gradients(tups_mlp* m, const float* x, const float* t, int batch, float* grad,
                                  double* loss) {
  if (!m) return TUPS_ERR_BADARG;
  MTRY(set_dev(m));
  MTRY(check_batch(m, batch));
  if (m->loss_slots < 1) {
    MTRY(mlp_alloc(m, &m->loss, 1));
    m->loss_slots = 1;
  }
  MTRY(h2d(m, m->x, x, (size_t)batch * m->n_in * sizeof(float)));
  MTRY(h2d(m, m->t, t, (size_t)batch * m->n_out * sizeof(float)));
  MTRY(mlp_cuda(m, cudaMemsetAsync(m->loss, 0, sizeof(double), m->stream), "memset"));
  MTRY(forward(m, batch, m->x, nullptr, m->t, m->loss));
  MTRY(backward(m, batch, m->x, nullptr, false, 0.0f, 0.0f));
  if (loss) MTRY(d2h(m, loss, m->loss, sizeof(double)));
  if (grad) MTRY(d2h(m, grad, m->grads, m->n_params * sizeof(float)));
  return mlp_cuda(m, cudaStreamSynchronize(m->stream), "synchronize");
}

extern "C" int tups_mlp_train(tups_mlp* m, const float* x, const float* t, int n_samples, int batch, int epochs,
                              float lr, float weight_decay, unsigned long long seed, double* loss_per_epoch) {
  if (!m) return TUPS_ERR_BADARG;
  if (n_samples < 1 || epochs < 0 || lr <= 0.0f || weight_decay < 0.0f)
    return mlp_error(m, TUPS_ERR_BADARG, "bad training arguments");
  MTRY(set_dev(m));
  batch = std::min(batch, n_samples);
  MTRY(check_batch(m, batch));
  if (n_samples > m->data_n) {
    MTRY(mlp_alloc(m, &m->data_x, (size_t)n_samples * m->n_in));
    MTRY(mlp_alloc(m, &m->data_t, (size_t)n_samples * m->n_out));
    MTRY(mlp_alloc(m, &m->idx, (size_t)n_samples));
    m->data_n = n_samples;
  }
  if (m->loss_slots < epochs) {
    MTRY(mlp_alloc(m, &m->loss, (size_t)epochs));
    m->loss_slots = epochs;
  }
  MTRY(h2d(m, m->data_x, x, (size_t)n_samples * m->n_in * sizeof(float)));
  MTRY(h2d(m, m->data_t, t, (size_t)n_samples * m->n_out * sizeof(float)));
  if (epochs > 0) MTRY(mlp_cuda(m, cudaMemsetAsync(m->loss, 0, (size_t)epochs * sizeof(double), m->stream), "memset"));
  const int per_epoch = (n_samples + batch - 1) / batch;
  std::vector<int> perm(n_samples);
  std::vector<int> all_idx((size_t)epochs * n_samples);
  uint64_t s = seed;
  for (int e = 0; e < epochs; e++) {
    for (int i = 0; i < n_samples; i++) perm[i] = i;
    for (int i = n_samples - 1; i > 0; i--) std::swap(perm[i], perm[(int)(mix64(s) % (uint64_t)(i + 1))]);
    std::memcpy(all_idx.data() + (size_t)e * n_samples, perm.data(), n_samples * sizeof(int));
  }
  for (int e = 0; e < epochs; e++) {
    // index upload per epoch: the host vector stays alive for the whole call
    MTRY(h2d(m, m->idx, all_idx.data() + (size_t)e * n_samples, n_samples * sizeof(int)));
    for (int b = 0; b < per_epoch; b++) {
      const int r0 = b * batch, rows = std::min(batch, n_samples - r0);
      MTRY(forward(m, rows, m->data_x, m->idx + r0, m->data_t, m->loss + e));
      MTRY(backward(m, rows, m->data_x, m->idx + r0, true, lr, weight_decay));
    }
  }
  if (loss_per_epoch && epochs > 0) {
    MTRY(d2h(m, loss_per_epoch, m->loss, (size_t)epochs * sizeof(double)));
    for (int e = 0; e < epochs; e++) loss_per_epoch[e] /= per_epoch;
  }
  return mlp_cuda(m, cudaStreamSynchronize(m->stream), "synchronize");
}
