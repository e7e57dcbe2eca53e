// FP64 dense tail on the GPU: the generalized edge spectrum of one sector for
// many confinement strengths (the kappa sweep of the batched form).
//
// Reference: ges::generalizedEigenproblem (modules/eigensolver/
// generalized_eigenproblem.cpp:38-95) solves H c = E M c once per call on the
// host through a Cholesky of M.  Here M is factorised once per sector on the
// device by canonical orthogonalisation, which tolerates the near-singular
// metric of power-sum states at large dL:
//   M = U diag(m) U^H,  keep m_k > eps * max(m)  (rank r),  X = U_r diag(m_r^-1/2),
//   E_j = eig(X^H H_j X),  H_j = omega_j H2 + kappa_j H4   (all normalised).
// The eigen decompositions are cuSOLVER's Hermitian divide-and-conquer solver,
// the two products per strength cuBLAS ZGEMMs; everything stays in FP64.
//
// Row-major complex input is read as column-major, i.e. as the conjugate
// matrices; the generalized eigenvalues of (conj H, conj M) are those of (H, M).
#include <cublas_v2.h>
#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <cmath>
#include <limits>
#include <vector>

#include "lemc_internal.h"

namespace lemc {
namespace {

// Normalise and Hermitise: X[a][b] = (Y[a][b] + conj(Y[b][a])) / 2 / sqrt(S_aa S_bb)
__global__ void normalise_kernel(int D, const double2* __restrict__ S, const double2* __restrict__ Y,
                                 double2* __restrict__ X) {
  const int a = blockIdx.y * blockDim.y + threadIdx.y;
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= D || b >= D) return;
  const double n = sqrt(S[size_t(a) * D + a].x * S[size_t(b) * D + b].x);
  const double2 y = Y[size_t(a) * D + b], yt = Y[size_t(b) * D + a];
  X[size_t(a) * D + b] = make_double2(0.5 * (y.x + yt.x) / n, 0.5 * (y.y - yt.y) / n);
}

// column k of U (of the kept r) scaled by 1/sqrt(m), into X (D x r, column-major)
__global__ void scale_columns_kernel(int D, int r, int first, const double2* __restrict__ U,
                                     const double* __restrict__ m, double2* __restrict__ X) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y;
  if (i >= D || k >= r) return;
  const double s = 1.0 / sqrt(m[first + k]);
  const double2 u = U[size_t(first + k) * D + i];
  X[size_t(k) * D + i] = make_double2(u.x * s, u.y * s);
}

__global__ void combine_kernel(int n, double w2, const double2* __restrict__ H2, double w4,
                               const double2* __restrict__ H4, double2* __restrict__ H) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  H[i] = make_double2(w2 * H2[i].x + w4 * H4[i].x, w2 * H2[i].y + w4 * H4[i].y);
}

struct Gpu {
  cusolverDnHandle_t sol = nullptr;
  cublasHandle_t blas = nullptr;
  std::vector<void*> bufs;
  ~Gpu() {
    for (void* p : bufs) cudaFree(p);
    if (blas) cublasDestroy(blas);
    if (sol) cusolverDnDestroy(sol);
  }
  template <class T>
  T* alloc(size_t n) {
    void* p = nullptr;
    if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess) return nullptr;
    bufs.push_back(p);
    return static_cast<T*>(p);
  }
};

}  // namespace
}  // namespace lemc

using namespace lemc;

extern "C" int lemc_geneig_sweep(int D, const double* S, const double* H2, const double* H4,
                                 const double* omega, const double* kappa, int n, double eps,
                                 double* evals, int* rank) {
  if (D <= 0 || n <= 0 || !S || !H2 || !H4 || !omega || !kappa || !evals || !(eps >= 0.0))
    return LEMC_ERR_ARG;
  for (int a = 0; a < D; ++a)
    if (!(S[2 * (size_t(a) * D + a)] > 0.0)) return LEMC_ERR_NUMERIC;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return LEMC_ERR_NODEVICE;
  }
  Gpu g;
  if (cusolverDnCreate(&g.sol) != CUSOLVER_STATUS_SUCCESS) return LEMC_ERR_CUDA;
  if (cublasCreate(&g.blas) != CUBLAS_STATUS_SUCCESS) return LEMC_ERR_CUDA;
  const size_t DD = size_t(D) * D;
  double2 *dS = g.alloc<double2>(DD), *dH2 = g.alloc<double2>(DD), *dH4 = g.alloc<double2>(DD);
  double2 *M = g.alloc<double2>(DD), *N2 = g.alloc<double2>(DD), *N4 = g.alloc<double2>(DD);
  double2 *X = g.alloc<double2>(DD), *H = g.alloc<double2>(DD), *T = g.alloc<double2>(DD);
  double2* A = g.alloc<double2>(DD);
  double* w = g.alloc<double>(D);
  int* info = g.alloc<int>(1);
  if (!dS || !dH2 || !dH4 || !M || !N2 || !N4 || !X || !H || !T || !A || !w || !info)
    return LEMC_ERR_CUDA;
  if (cudaMemcpy(dS, S, DD * sizeof(double2), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(dH2, H2, DD * sizeof(double2), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(dH4, H4, DD * sizeof(double2), cudaMemcpyHostToDevice) != cudaSuccess)
    return LEMC_ERR_CUDA;
  const dim3 tb(16, 16), gb((D + 15) / 16, (D + 15) / 16);
  normalise_kernel<<<gb, tb>>>(D, dS, dS, M);
  normalise_kernel<<<gb, tb>>>(D, dS, dH2, N2);
  normalise_kernel<<<gb, tb>>>(D, dS, dH4, N4);
  if (cudaPeekAtLastError() != cudaSuccess) return LEMC_ERR_CUDA;

  // M = U diag(m) U^H (eigenvalues ascending, U overwrites M)
  int lwork = 0;
  if (cusolverDnZheevd_bufferSize(g.sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, D,
                                  reinterpret_cast<cuDoubleComplex*>(M), D, w, &lwork) !=
      CUSOLVER_STATUS_SUCCESS)
    return LEMC_ERR_CUDA;
  double2* work = g.alloc<double2>(size_t(std::max(1, lwork)));
  if (!work) return LEMC_ERR_CUDA;
  if (cusolverDnZheevd(g.sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, D,
                       reinterpret_cast<cuDoubleComplex*>(M), D, w,
                       reinterpret_cast<cuDoubleComplex*>(work), lwork, info) !=
      CUSOLVER_STATUS_SUCCESS)
    return LEMC_ERR_CUDA;
  std::vector<double> m(D);
  int h_info = 0;
  if (cudaMemcpy(m.data(), w, D * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(&h_info, info, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
    return LEMC_ERR_CUDA;
  if (h_info != 0) return LEMC_ERR_NUMERIC;
  const double mmax = m[D - 1];
  if (!(mmax > 0.0)) return LEMC_ERR_NUMERIC;
  int first = 0;
  while (first < D && !(m[first] > eps * mmax)) ++first;
  const int r = D - first;
  if (rank) *rank = r;
  scale_columns_kernel<<<dim3((D + 127) / 128, r), 128>>>(D, r, first, M, w, X);
  if (cudaPeekAtLastError() != cudaSuccess) return LEMC_ERR_CUDA;

  int lwork2 = 0;
  if (cusolverDnZheevd_bufferSize(g.sol, CUSOLVER_EIG_MODE_NOVECTOR, CUBLAS_FILL_MODE_LOWER, r,
                                  reinterpret_cast<cuDoubleComplex*>(A), r, w, &lwork2) !=
      CUSOLVER_STATUS_SUCCESS)
    return LEMC_ERR_CUDA;
  double2* work2 = g.alloc<double2>(size_t(std::max(1, lwork2)));
  if (!work2) return LEMC_ERR_CUDA;
  const cuDoubleComplex one = make_cuDoubleComplex(1.0, 0.0), zero = make_cuDoubleComplex(0.0, 0.0);
  std::vector<double> e(r);
  for (int j = 0; j < n; ++j) {
    combine_kernel<<<(int(DD) + 255) / 256, 256>>>(int(DD), omega[j], N2, kappa[j], N4, H);
    if (cudaPeekAtLastError() != cudaSuccess) return LEMC_ERR_CUDA;
    // T = H X (D x r), A = X^H T (r x r)
    if (cublasZgemm(g.blas, CUBLAS_OP_N, CUBLAS_OP_N, D, r, D, &one,
                    reinterpret_cast<cuDoubleComplex*>(H), D, reinterpret_cast<cuDoubleComplex*>(X),
                    D, &zero, reinterpret_cast<cuDoubleComplex*>(T), D) != CUBLAS_STATUS_SUCCESS ||
        cublasZgemm(g.blas, CUBLAS_OP_C, CUBLAS_OP_N, r, r, D, &one,
                    reinterpret_cast<cuDoubleComplex*>(X), D, reinterpret_cast<cuDoubleComplex*>(T),
                    D, &zero, reinterpret_cast<cuDoubleComplex*>(A), r) != CUBLAS_STATUS_SUCCESS)
      return LEMC_ERR_CUDA;
    if (cusolverDnZheevd(g.sol, CUSOLVER_EIG_MODE_NOVECTOR, CUBLAS_FILL_MODE_LOWER, r,
                         reinterpret_cast<cuDoubleComplex*>(A), r, w,
                         reinterpret_cast<cuDoubleComplex*>(work2), lwork2, info) !=
        CUSOLVER_STATUS_SUCCESS)
      return LEMC_ERR_CUDA;
    if (cudaMemcpy(e.data(), w, r * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(&h_info, info, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
      return LEMC_ERR_CUDA;
    if (h_info != 0) return LEMC_ERR_NUMERIC;
    for (int k = 0; k < D; ++k)
      evals[size_t(j) * D + k] = k < r ? e[k] : std::numeric_limits<double>::quiet_NaN();
  }
  return cudaDeviceSynchronize() == cudaSuccess ? LEMC_OK : LEMC_ERR_CUDA;
}

// ---- time evolution in the S-orthonormal basis ------------------------------
// Reference: timeEvolution::edgeDensityResponse_compute (modules/dynamics/
// dynamics.cpp:24-53, :149-308) integrates M dC/dt = -i (H + f(t) U) C on the
// host with an adaptive Cash-Karp pair.  Here, on the GPU in FP64: with the
// canonical orthogonalisation X of M (X^H M X = 1), C = X y and
//   dy/dt = -i (H' + f(t) U') y,   H' = X^H H X - e I,  U' = X^H U X,
// e = tr(H')/r removed as a global phase (no observable depends on it, and it
// keeps h |H'| small).  Classical RK4 with h = save_step / substeps, up to
// kObsBatch save points in one launch (rk4_kernel), then the observables
// C^H rho_l C = y^H (X^H rho_l X) y and C^H M C = y^H y of the whole batch.
namespace lemc {
namespace {

// row-major complex input -> column-major device layout (a transpose)
__global__ void to_colmajor_kernel(int D, const double2* __restrict__ in, double2* __restrict__ out) {
  const int i = blockIdx.y * blockDim.y + threadIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < D && j < D) out[size_t(j) * D + i] = in[size_t(i) * D + j];
}

// column-major r x r -> row-major, minus e on the diagonal
__global__ void to_rowmajor_shift_kernel(int r, const double2* __restrict__ in, double e,
                                         double2* __restrict__ out) {
  const int i = blockIdx.y * blockDim.y + threadIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < r && j < r) {
    double2 v = in[size_t(j) * r + i];
    if (i == j) v.x -= e;
    out[size_t(i) * r + j] = v;
  }
}

__global__ void diag_mean_kernel(int r, const double2* __restrict__ A, double* __restrict__ out) {
  __shared__ double s[256];
  double v = 0.0;
  for (int i = threadIdx.x; i < r; i += blockDim.x) v += A[size_t(i) * r + i].x;
  s[threadIdx.x] = v;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = s[0] / r;
}

__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}

// Classical RK4 over many steps in one cooperative launch: k = -i (H + f U)(y + a k').
//
// A CTA owns `rpc` rows of H' and U' and keeps them in shared memory for the
// whole launch (32 r^2 bytes over all CTAs: 60 KB each at r = 526; rows stay in
// global memory, i.e. in L2, when they do not fit), with its own copy of y and
// of the running RK sum, so a stage only exchanges the r entries of one k
// vector through L2.  The stages are a serial chain of 4 grid barriers a step:
// what bounds a step is their latency, not the r^2 work (8.8 MB of L2 reads or
// 4.4 MFLOP a stage at r = 526).  Warps split a CTA's rows and columns.
// One launch per stage and two warp-row products from L2 took 7.2 us a stage
// plus the launch gaps; now 3.6 us a stage (526 states, 500 steps: 15.1 -> 7.1 ms).
// Every grid barrier is bounded in time; on expiry the CTA raises *err and
// leaves, and the others leave when they see it.
constexpr int kObsBatch = 1024;  // save points per launch: bounds the Y buffer at 16 KB r
constexpr int kRkThreads = 512;
constexpr int kRkWarps = kRkThreads / 32;
constexpr long long kRkWaitCycles = 4000000000LL;  // about 2 s

struct RkArgs {
  int r, rpc, parts;        // rows per CTA; warps per row (a power of two)
  int rows_in_smem;
  double2* ws;              // rows not in shared memory: 3 r entries a CTA for y, the sum, v
  int v_in_smem;
  const double2 *H, *U;     // row-major r x r
  double2* y;               // state, in and out
  double2* k;               // [2][r] exchange buffers
  const double* f;          // profile at the three stage times of each step
  double h;
  int substeps, n_save;     // save points of this launch, substeps steps each
  double2* Y;               // [n_save][r]: y at each save point
  unsigned int* bar;        // arrivals so far
  unsigned int bar0;        // arrivals before this launch
  int* err;
};

// All CTAs arrive; true when every arrival up to `target` is visible.
__device__ __forceinline__ bool rk_barrier(const RkArgs& a, unsigned int target, int* ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(a.bar, 1u);
    const long long t0 = clock64();
    int good = 1;
    // counts are compared modulo 2^32
    while (int(*(volatile unsigned int*)a.bar - target) < 0) {
      if (*(volatile int*)a.err) { good = 0; break; }
      if (clock64() - t0 > kRkWaitCycles) {
        atomicExch(a.err, LEMC_ERR_TIMEOUT);
        good = 0;
        break;
      }
    }
    __threadfence();
    *ok = good;
  }
  __syncthreads();
  return *ok != 0;
}

__global__ void __launch_bounds__(kRkThreads, 1) rk4_kernel(const RkArgs a) {
  extern __shared__ __align__(16) double2 rk_smem[];
  __shared__ double2 part[kRkWarps];
  __shared__ int ok;
  const int r = a.r, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // y and the sum are read and written by one thread per entry; v is shared
  double2* own = a.rows_in_smem ? rk_smem + r : a.ws + size_t(blockIdx.x) * 3 * r;
  double2* y = own;                                     // [r]
  double2* ks = own + r;                                // [r] k1 + 2 k2 + 2 k3
  double2* v = a.v_in_smem ? rk_smem : own + 2 * r;     // [r] the stage's argument
  double2* hs = rk_smem + 3 * r;                        // [rpc][r] (rows in shared memory)
  double2* us = hs + size_t(a.rpc) * r;
  const int row0 = blockIdx.x * a.rpc;
  const int nrow = min(a.rpc, r - row0);
  const double2* Hrow = a.H + size_t(row0) * r;
  const double2* Urow = a.U + size_t(row0) * r;
  if (a.rows_in_smem) {
    for (int e = tid; e < nrow * r; e += kRkThreads) {
      hs[e] = Hrow[e];
      us[e] = Urow[e];
    }
    Hrow = hs;
    Urow = us;
  }
  for (int j = tid; j < r; j += kRkThreads) y[j] = a.y[j];
  __syncthreads();
  const int rows_at_once = kRkWarps / a.parts;
  unsigned int target = a.bar0;
  size_t step = 0;
  bool good = true;
  for (int s = 0; s < a.n_save && good; ++s) {
    for (int q = 0; q < a.substeps && good; ++q, ++step) {
#pragma unroll 1
      for (int st = 0; st < 4 && good; ++st) {
        // argument of this stage from the previous stage's k
        const double2* kin = a.k + size_t((st + 1) & 1) * r;
        double2* kout = a.k + size_t(st & 1) * r;
        const double c = st == 3 ? a.h : 0.5 * a.h;
        if (st == 0) {
          for (int j = tid; j < r; j += kRkThreads) v[j] = y[j];
        } else {
          for (int j = tid; j < r; j += kRkThreads) {
            const double2 kj = __ldcg(kin + j);
            const double2 yj = y[j];
            v[j] = make_double2(fma(c, kj.x, yj.x), fma(c, kj.y, yj.y));
            if (st == 1) {
              ks[j] = kj;
            } else {
              ks[j].x += 2.0 * kj.x;
              ks[j].y += 2.0 * kj.y;
            }
          }
        }
        __syncthreads();
        const double f = a.f[3 * step + (st == 0 ? 0 : st == 3 ? 2 : 1)];
        for (int b = 0; b < nrow; b += rows_at_once) {
          const int row = b + warp / a.parts, p = warp % a.parts;
          double2 sh = make_double2(0.0, 0.0), su = sh;
          if (row < nrow) {
            const double2* hr = Hrow + size_t(row) * r;
            const double2* ur = Urow + size_t(row) * r;
#pragma unroll 4
            for (int j = p * 32 + lane; j < r; j += 32 * a.parts) {
              const double2 x = v[j];
              sh = cfma(hr[j], x, sh);
              su = cfma(ur[j], x, su);
            }
          }
          double2 t = make_double2(fma(f, su.x, sh.x), fma(f, su.y, sh.y));
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
            t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
          }
          if (lane == 0) part[warp] = t;
          __syncthreads();
          if (tid < rows_at_once && b + tid < nrow) {
            double2 u = part[tid * a.parts];
            for (int w = 1; w < a.parts; ++w) {
              u.x += part[tid * a.parts + w].x;
              u.y += part[tid * a.parts + w].y;
            }
            __stcg(kout + row0 + b + tid, make_double2(u.y, -u.x));  // -i u
          }
          __syncthreads();
        }
        target += gridDim.x;
        good = rk_barrier(a, target, &ok);
      }
      if (!good) break;
      const double c6 = a.h / 6.0;
      const double2* k4 = a.k + size_t(1) * r;
      for (int j = tid; j < r; j += kRkThreads) {
        const double2 kj = __ldcg(k4 + j);
        y[j].x += c6 * (ks[j].x + kj.x);
        y[j].y += c6 * (ks[j].y + kj.y);
      }
      __syncthreads();
    }
    if (good)
      for (int j = row0 + tid; j < row0 + nrow; j += kRkThreads) a.Y[size_t(s) * r + j] = y[j];
  }
  if (good)
    for (int j = row0 + tid; j < row0 + nrow; j += kRkThreads) a.y[j] = y[j];
}

// out[z][s][l] = sum over row tiles x = z, z + Z, ... of y_s^H R_l y_s, for a
// batch of save points (rows of Y) at once; l == L gives y^H y.  A block takes 32
// save points of one l: R_l Y^T in 32 x 32 tiles (2 x 2 entries a thread, operands
// staged in shared memory), each multiplied by conj(y) as it is done.  4 FP64 FMAs
// per entry, so the FP64 pipe bounds it; one thread per matrix row and save point
// (uncoalesced rows, L + 1 blocks) took 191 us a save point
// (526 states, 9 components; now 1.3 us).
constexpr int kObsT = 32, kObsThreads = 256, kObsZ = 4;

__global__ void __launch_bounds__(kObsThreads)
observe_kernel(int r, int L, const double2* __restrict__ R, const double2* __restrict__ Y, int n,
               double2* __restrict__ out) {
  __shared__ double2 ra[kObsT][kObsT + 1], ys[kObsT][kObsT + 1];  // [j][row], [j][save]
  const int s0 = blockIdx.x * kObsT, l = blockIdx.y, z = blockIdx.z;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const double2 zero = make_double2(0.0, 0.0);
  double2 acc[2] = {zero, zero};  // save points s0 + tx, s0 + tx + 16
  const double2* A = R + size_t(l < L ? l : 0) * r * r;
  for (int i0 = z * kObsT; i0 < r; i0 += kObsZ * kObsT) {
    double2 t[2][2] = {{zero, zero}, {zero, zero}};  // [row][save]
    if (l < L) {
      for (int j0 = 0; j0 < r; j0 += kObsT) {
        __syncthreads();
        for (int e = tid; e < kObsT * kObsT; e += kObsThreads) {
          const int j = e & 31, q = e >> 5;
          ra[j][q] = (i0 + q < r && j0 + j < r) ? A[size_t(i0 + q) * r + j0 + j] : zero;
          ys[j][q] = (s0 + q < n && j0 + j < r) ? Y[size_t(s0 + q) * r + j0 + j] : zero;
        }
        __syncthreads();
#pragma unroll 8
        for (int j = 0; j < kObsT; ++j) {
          const double2 a0 = ra[j][ty], a1 = ra[j][ty + 16];
          const double2 b0 = ys[j][tx], b1 = ys[j][tx + 16];
          t[0][0] = cfma(a0, b0, t[0][0]);
          t[0][1] = cfma(a0, b1, t[0][1]);
          t[1][0] = cfma(a1, b0, t[1][0]);
          t[1][1] = cfma(a1, b1, t[1][1]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int row = i0 + ty + 16 * i, s = s0 + tx + 16 * q;
        if (row >= r || s >= n) continue;
        const double2 y = Y[size_t(s) * r + row];
        const double2 m = l < L ? t[i][q] : y;
        acc[q] = cfma(make_double2(y.x, -y.y), m, acc[q]);
      }
  }
  __syncthreads();
  ra[ty][tx] = acc[0];
  ra[ty][tx + 16] = acc[1];
  __syncthreads();
  if (tid < kObsT && s0 + tid < n) {
    double2 v = ra[0][tid];
    for (int q = 1; q < 16; ++q) {
      v.x += ra[q][tid].x;
      v.y += ra[q][tid].y;
    }
    out[(size_t(z) * n + s0 + tid) * (L + 1) + l] = v;
  }
}

// sums of the kObsZ partial observables of a batch: obs[n][L] and nrm[n]
__global__ void observe_sum_kernel(int n, int L, const double2* __restrict__ part,
                                   double2* __restrict__ obs, double* __restrict__ nrm) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * (L + 1)) return;
  double2 v = part[e];
  for (int z = 1; z < kObsZ; ++z) {
    const double2 p = part[size_t(z) * n * (L + 1) + e];
    v.x += p.x;
    v.y += p.y;
  }
  const int s = e / (L + 1), l = e % (L + 1);
  if (l < L)
    obs[size_t(s) * L + l] = v;
  else
    nrm[s] = v.x;
}

}  // namespace
}  // namespace lemc

extern "C" int lemc_evolve_device(int D, const double* M, const double* H, const double* U, int L,
                                  const double* rho, lemc_profile_fn f, void* user,
                                  double end_time, double save_step, int substeps, double eps,
                                  double* out, double* norms, int* n_save, int* rank) {
  if (D <= 0 || !M || !H || !U || L < 0 || (L > 0 && !rho) || !(save_step > 0) ||
      !(end_time > 0) || substeps < 1 || !(eps >= 0.0))
    return LEMC_ERR_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return LEMC_ERR_NODEVICE;
  }
  const int ns = int(std::ceil(end_time / save_step));
  if (n_save) *n_save = ns;
  Gpu g;
  if (cusolverDnCreate(&g.sol) != CUSOLVER_STATUS_SUCCESS) return LEMC_ERR_CUDA;
  if (cublasCreate(&g.blas) != CUBLAS_STATUS_SUCCESS) return LEMC_ERR_CUDA;
  const size_t DD = size_t(D) * D;
  const int NM = 3 + L;  // M, H, U, rho_0..rho_{L-1}
  double2* raw = g.alloc<double2>(DD);
  double2* cm = g.alloc<double2>(DD * NM);  // column-major copies
  double2* X = g.alloc<double2>(DD);
  double2* T = g.alloc<double2>(DD);
  double2* P = g.alloc<double2>(DD);
  double* w = g.alloc<double>(D);
  int* info = g.alloc<int>(1);
  if (!raw || !cm || !X || !T || !P || !w || !info) return LEMC_ERR_CUDA;
  const dim3 tb(16, 16), gb((D + 15) / 16, (D + 15) / 16);
  for (int q = 0; q < NM; ++q) {
    const double* src = q == 0 ? M : q == 1 ? H : q == 2 ? U : rho + size_t(2) * DD * (q - 3);
    if (cudaMemcpy(raw, src, DD * sizeof(double2), cudaMemcpyHostToDevice) != cudaSuccess)
      return LEMC_ERR_CUDA;
    to_colmajor_kernel<<<gb, tb>>>(D, raw, cm + DD * q);
  }
  // canonical orthogonalisation of M (column-major copy 0 is overwritten by U)
  if (cudaMemcpy(P, cm, DD * sizeof(double2), cudaMemcpyDeviceToDevice) != cudaSuccess)
    return LEMC_ERR_CUDA;
  int lwork = 0;
  if (cusolverDnZheevd_bufferSize(g.sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, D,
                                  reinterpret_cast<cuDoubleComplex*>(P), D, w, &lwork) !=
      CUSOLVER_STATUS_SUCCESS)
    return LEMC_ERR_CUDA;
  double2* work = g.alloc<double2>(size_t(std::max(1, lwork)));
  if (!work) return LEMC_ERR_CUDA;
  if (cusolverDnZheevd(g.sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, D,
                       reinterpret_cast<cuDoubleComplex*>(P), D, w,
                       reinterpret_cast<cuDoubleComplex*>(work), lwork, info) != CUSOLVER_STATUS_SUCCESS)
    return LEMC_ERR_CUDA;
  std::vector<double> m(D);
  int h_info = 0;
  if (cudaMemcpy(m.data(), w, D * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(&h_info, info, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
    return LEMC_ERR_CUDA;
  if (h_info != 0 || !(m[D - 1] > 0.0)) return LEMC_ERR_NUMERIC;
  int first = 0;
  while (first < D && !(m[first] > eps * m[D - 1])) ++first;
  const int r = D - first;
  if (rank) *rank = r;
  scale_columns_kernel<<<dim3((D + 127) / 128, r), 128>>>(D, r, first, P, w, X);
  // projected matrices, row-major on the device: H', U', rho'_l
  const size_t RR = size_t(r) * r;
  double2* Hr = g.alloc<double2>(RR);
  double2* Ur = g.alloc<double2>(RR);
  double2* Rr = g.alloc<double2>(RR * std::max(1, L));
  double2* A = g.alloc<double2>(RR);
  double* emean = g.alloc<double>(1);
  const int batch = std::min(ns, kObsBatch);
  const double h = save_step / substeps;
  const size_t nsteps = size_t(ns > 1 ? ns - 1 : 0) * substeps;
  double2 *y = g.alloc<double2>(r), *kx = g.alloc<double2>(2 * size_t(r));
  double2* Y = g.alloc<double2>(size_t(batch) * r);
  double2* obs_part = g.alloc<double2>(size_t(kObsZ) * batch * (L + 1));
  double2* obs = g.alloc<double2>(size_t(ns) * std::max(1, L));
  double* nrm = g.alloc<double>(ns);
  double* dfv = g.alloc<double>(std::max<size_t>(1, 3 * nsteps));
  int* sync = g.alloc<int>(2);  // barrier arrivals, error word
  if (!Hr || !Ur || !Rr || !A || !emean || !y || !kx || !Y || !obs_part || !obs || !nrm || !dfv ||
      !sync)
    return LEMC_ERR_CUDA;
  const cuDoubleComplex one = make_cuDoubleComplex(1.0, 0.0), zero = make_cuDoubleComplex(0.0, 0.0);
  auto project = [&](const double2* Bcm) -> bool {  // A = X^H B X (column-major r x r)
    return cublasZgemm(g.blas, CUBLAS_OP_N, CUBLAS_OP_N, D, r, D, &one,
                       reinterpret_cast<const cuDoubleComplex*>(Bcm), D,
                       reinterpret_cast<const cuDoubleComplex*>(X), D, &zero,
                       reinterpret_cast<cuDoubleComplex*>(T), D) == CUBLAS_STATUS_SUCCESS &&
           cublasZgemm(g.blas, CUBLAS_OP_C, CUBLAS_OP_N, r, r, D, &one,
                       reinterpret_cast<const cuDoubleComplex*>(X), D,
                       reinterpret_cast<const cuDoubleComplex*>(T), D, &zero,
                       reinterpret_cast<cuDoubleComplex*>(A), r) == CUBLAS_STATUS_SUCCESS;
  };
  const dim3 gr((r + 15) / 16, (r + 15) / 16);
  if (!project(cm + DD)) return LEMC_ERR_CUDA;
  diag_mean_kernel<<<1, 256>>>(r, A, emean);
  double e = 0.0;
  if (cudaMemcpy(&e, emean, sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return LEMC_ERR_CUDA;
  to_rowmajor_shift_kernel<<<gr, tb>>>(r, A, e, Hr);
  if (!project(cm + 2 * DD)) return LEMC_ERR_CUDA;
  to_rowmajor_shift_kernel<<<gr, tb>>>(r, A, 0.0, Ur);
  for (int l = 0; l < L; ++l) {
    if (!project(cm + DD * (3 + l))) return LEMC_ERR_CUDA;
    to_rowmajor_shift_kernel<<<gr, tb>>>(r, A, 0.0, Rr + RR * l);
  }
  // y(0) = X^H M e_0 (C(0) = e_0)
  if (cublasZgemv(g.blas, CUBLAS_OP_C, D, r, &one, reinterpret_cast<const cuDoubleComplex*>(X), D,
                  reinterpret_cast<const cuDoubleComplex*>(cm), 1, &zero,
                  reinterpret_cast<cuDoubleComplex*>(y), 1) != CUBLAS_STATUS_SUCCESS)
    return LEMC_ERR_CUDA;
  if (cudaPeekAtLastError() != cudaSuccess) return LEMC_ERR_CUDA;
  // profile values at every stage time, evaluated on the host
  std::vector<double> fv(3 * nsteps);
  for (size_t k = 0; k < nsteps; ++k) {
    const double t = double(k) * h;
    fv[3 * k] = f ? f(t, user) : 0.0;
    fv[3 * k + 1] = f ? f(t + 0.5 * h, user) : 0.0;
    fv[3 * k + 2] = f ? f(t + h, user) : 0.0;
  }
  if (nsteps > 0 && cudaMemcpy(dfv, fv.data(), sizeof(double) * fv.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    return LEMC_ERR_CUDA;
  if (cudaMemset(sync, 0, 2 * sizeof(int)) != cudaSuccess) return LEMC_ERR_CUDA;
  // One CTA per SM at most, at least four rows each (a barrier costs more with
  // more CTAs than fewer rows save); rows in shared memory when they fit.
  int dev = 0, sms = 148, smem_max = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return LEMC_ERR_CUDA;
  RkArgs ra{};
  ra.r = r;
  ra.rpc = std::max(4, (r + sms - 1) / sms);
  ra.parts = kRkWarps;
  while (ra.parts > 1 && kRkWarps / ra.parts < ra.rpc) ra.parts /= 2;
  const size_t vec_bytes = sizeof(double2) * size_t(r);
  const size_t row_bytes = 2 * vec_bytes * size_t(ra.rpc);
  const size_t smem_cap = size_t(smem_max) - 1024;  // the kernel's static shared memory
  ra.rows_in_smem = 3 * vec_bytes + row_bytes <= smem_cap;
  ra.v_in_smem = vec_bytes <= smem_cap;
  const size_t rk_smem_bytes = ra.rows_in_smem ? 3 * vec_bytes + row_bytes : ra.v_in_smem ? vec_bytes : 0;
  if (cudaFuncSetAttribute(rk4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           int(rk_smem_bytes)) != cudaSuccess)
    return LEMC_ERR_CUDA;
  const int rk_ctas = (r + ra.rpc - 1) / ra.rpc;
  if (!ra.rows_in_smem) {
    ra.ws = g.alloc<double2>(size_t(rk_ctas) * 3 * r);
    if (!ra.ws) return LEMC_ERR_CUDA;
  }
  ra.H = Hr;
  ra.U = Ur;
  ra.y = y;
  ra.k = kx;
  ra.h = h;
  ra.substeps = substeps;
  ra.bar = reinterpret_cast<unsigned int*>(sync);
  ra.err = sync + 1;
  // save point 0 is the initial state; the others follow in batches
  if (cudaMemcpyAsync(Y, y, sizeof(double2) * r, cudaMemcpyDeviceToDevice) != cudaSuccess)
    return LEMC_ERR_CUDA;
  for (int s0 = 0, first = 1; s0 < ns; first = 0) {
    const int n = std::min(batch, ns - s0);
    ra.n_save = n - first;
    ra.Y = Y + size_t(first) * r;
    ra.f = dfv + 3 * size_t(s0 + first - 1) * substeps;
    if (ra.n_save > 0) {
      void* kargs[] = {&ra};
      if (cudaLaunchCooperativeKernel(reinterpret_cast<void*>(rk4_kernel), dim3(rk_ctas),
                                      dim3(kRkThreads), kargs, rk_smem_bytes, nullptr) != cudaSuccess)
        return LEMC_ERR_CUDA;
      ra.bar0 += 4u * unsigned(ra.n_save) * unsigned(substeps) * unsigned(rk_ctas);
    }
    observe_kernel<<<dim3((n + kObsT - 1) / kObsT, L + 1, kObsZ), kObsThreads>>>(r, L, Rr, Y, n,
                                                                                obs_part);
    observe_sum_kernel<<<(n * (L + 1) + 255) / 256, 256>>>(n, L, obs_part, obs + size_t(s0) * L,
                                                          nrm + s0);
    s0 += n;
  }
  if (cudaPeekAtLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess)
    return LEMC_ERR_CUDA;
  int rk_err = 0;
  if (cudaMemcpy(&rk_err, ra.err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
    return LEMC_ERR_CUDA;
  if (rk_err != 0) return LEMC_ERR_TIMEOUT;
  if (L > 0 && out) {
    std::vector<double2> all(size_t(ns) * L);
    if (cudaMemcpy(all.data(), obs, all.size() * sizeof(double2), cudaMemcpyDeviceToHost) != cudaSuccess)
      return LEMC_ERR_CUDA;
    for (size_t q = 0; q < all.size(); ++q) {
      out[2 * q] = all[q].x;
      out[2 * q + 1] = all[q].y;
    }
  }
  if (norms && cudaMemcpy(norms, nrm, ns * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
    return LEMC_ERR_CUDA;
  return LEMC_OK;
}

// Edge density on an angular grid from its Fourier components (reference
// observer::edgeDensity_reconstruct, dynamics.cpp:110-125, gives the
// components <rho_l>(t) = C^H rho_l C; the density itself is
// n(theta) = (1/2pi) [<rho_0> + 2 Re sum_{l>0} e^{-i l theta} <rho_l>]).
namespace lemc {
namespace {

__global__ void density_grid_kernel(int L, const int* __restrict__ ls, int n_times,
                                    const double2* __restrict__ rho, const double2* __restrict__ ref,
                                    int n_theta, double* __restrict__ out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int t = blockIdx.y;
  if (g >= n_theta || t >= n_times) return;
  const double theta = 2.0 * M_PI * double(g) / double(n_theta);
  double acc = 0.0;
  for (int q = 0; q < L; ++q) {
    const double2 r = rho[size_t(t) * L + q];
    const double2 r0 = ref[q];
    const double dr = r.x - r0.x, di = r.y - r0.y;
    const int l = ls[q];
    if (l == 0) {
      acc += dr;
    } else {
      double s, c;
      sincos(double(l) * theta, &s, &c);
      acc += 2.0 * (dr * c + di * s);  // 2 Re(e^{-i l theta} (dr + i di))
    }
  }
  out[size_t(t) * n_theta + g] = acc / (2.0 * M_PI);
}

}  // namespace
}  // namespace lemc

extern "C" int lemc_edge_density_grid(int L, const int32_t* l, int n_times, const double* rho_t,
                                      const double* rho_ref, int n_theta, double* out) {
  using namespace lemc;
  if (L <= 0 || !l || n_times <= 0 || !rho_t || n_theta <= 0 || !out) return LEMC_ERR_ARG;
  for (int q = 0; q < L; ++q)
    if (l[q] < 0) return LEMC_ERR_ARG;
  int* d_l = nullptr;
  double2 *d_rho = nullptr, *d_ref = nullptr;
  double* d_out = nullptr;
  int st = LEMC_OK;
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess && st == LEMC_OK) st = LEMC_ERR_CUDA;
    return st == LEMC_OK;
  };
  const size_t nr = size_t(n_times) * L;
  if (ok(cudaMalloc(&d_l, sizeof(int) * L)) && ok(cudaMalloc(&d_rho, sizeof(double2) * nr)) &&
      ok(cudaMalloc(&d_ref, sizeof(double2) * L)) &&
      ok(cudaMalloc(&d_out, sizeof(double) * size_t(n_times) * n_theta)) &&
      ok(cudaMemcpy(d_l, l, sizeof(int) * L, cudaMemcpyHostToDevice)) &&
      ok(cudaMemcpy(d_rho, rho_t, sizeof(double2) * nr, cudaMemcpyHostToDevice)) &&
      ok(cudaMemcpy(d_ref, rho_ref ? rho_ref : rho_t, sizeof(double2) * L, cudaMemcpyHostToDevice))) {
    const dim3 grid((n_theta + 127) / 128, n_times);
    density_grid_kernel<<<grid, 128>>>(L, d_l, n_times, d_rho, d_ref, n_theta, d_out);
    if (ok(cudaGetLastError()))
      ok(cudaMemcpy(out, d_out, sizeof(double) * size_t(n_times) * n_theta, cudaMemcpyDeviceToHost));
  }
  cudaFree(d_l);
  cudaFree(d_rho);
  cudaFree(d_ref);
  cudaFree(d_out);
  return st;
}
