// Orbital occupation numbers <f_L| a^dagger_l a_l |f_R> with the two-state
// walker (reference modules/green_function/green_function.cu:199-373 and
// gf_occupation_numbers.cu:16-239), all (L, R) pairs of a sector in one launch.
//
// A walker carries N+1 particles z_0..z_N: f_L depends on z_0..z_{N-1}, f_R
// on z_1..z_N, and the walker samples |f_L| |f_R| with
// f = P_row(z) prod_{i<j} (z_i - z_j)^m exp(-sum |z|^2 / 4).  One sweep moves
// particle 0, then 1..N-1, then N, each with its own Metropolis test:
//   0:      |J_0|^m |P_L'/P_L| exp((|z|^2 - |z'|^2)/4)
//   1..N-1: |c|^m |P_L'/P_L| |P_R'/P_R| |J|^{2m} exp((|z|^2 - |z'|^2)/2),
//           c = (z'-z_0)(z'-z_N) / ((z-z_0)(z-z_N))
//   N:      |J_N|^m |P_R'/P_R| exp((|z|^2 - |z'|^2)/4)
// evaluated as log-ratios.  After every sweep the estimator
//   sum_l exp(-ln(2 pi l!) + l ln(z_0 conj(z_N)/2) - (|z_0|^2+|z_N|^2)/4 + i phase),
//   phase = arg(P_R/P_L) + m arg prod_{i=1}^{N-1} (z_i - z_N)/(z_0 - z_i),
// is accumulated per walker in FP64 (magnitudes by a log-domain recurrence,
// so nothing under- or overflows for large N), and reduced per pair at the end.
//
// G lanes per walker on G or G / 2 threads; positions in shared memory.
// Random numbers: Philox counter {particle, sweep, walker, 2}, init tag 3.
#include <cuda_runtime.h>

#include <climits>
#include <cmath>
#include <mutex>
#include <vector>

#include "lemc_internal.h"
#include "lemc_rng.h"
#include "partitions.hpp"

namespace lemc {
namespace {

constexpr uint32_t kTagOccMove = 2u, kTagOccInit = 3u;

struct OccArgs {
  int W, N, m, D, Lc;
  float sigma;
  float invR;
  uint32_t k0, k1;
  int burn, sweeps;
  const int32_t* pairs;   // [D][2*kMaxGuideParts] (part, mult)
  const int32_t* npairs;  // [D]
  double2* acc;           // [Lc][W] per-walker sums
  uint32_t* accepted;     // [W]
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ double2 cpow_d(double2 z, int k) {
  double2 r = make_double2(1.0, 0.0), b = z;
  while (k) {
    if (k & 1) r = cmul(r, b);
    k >>= 1;
    if (k) b = cmul(b, b);
  }
  return r;
}

// G lanes per walker on P consecutive threads of a warp, thread gl standing for the
// V = G / P lanes gl + v P: lane g owns the shared particles j = 1 + g + tG of the
// Jastrow sums; the estimator's partial products and orbitals and the guide's sums go
// over the threads.  Xor-butterfly reductions within the group give every thread
// bit-identical sums, hence the same accept decision.  Every shuffle sits in control
// flow that is uniform over the warp (the guide loops run over all kMaxGuideParts
// slots, the walkers beyond W compute and do not write), so full-warp masks are exact.
constexpr int kOccLanesThreads = 128;

template <int P>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = P / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, P);
  return v;
}

// The FP32 sum over a walker's G lanes held by P threads, thread gl with the V = G / P
// lanes gl + v P: the butterfly's steps across v come first, in registers, so the sum
// (and with it the chain of decisions) is the one that G threads form.
template <int P, int V>
__device__ __forceinline__ float group_sumf(float (&x)[V]) {
#pragma unroll
  for (int h = V / 2; h > 0; h >>= 1)
#pragma unroll
    for (int v = 0; v < h; ++v) x[v] += x[v + h];
  float s = x[0];
#pragma unroll
  for (int o = P / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, P);
  return s;
}

// A walker's guide factors: its left row's nL distinct parts and its right row's nR
// are nL + nR slots, slot s on thread s % P; the thread keeps that part's power sum and
// forms its FP64 log-ratio in every move, and a butterfly adds the terms up.
//
// Bound: issue (a third of the instructions integer) and the serial part of a move.
// With every lane forming all of its walker's terms (two powers and a division each) out
// of indexed local arrays, N=50 at 65536 walkers took 0.91 ms a sweep; with the slots
// over the lanes 0.52, and with two lanes a thread 0.41.  Five blocks an SM (96 registers)
// against six: 4.10 and 4.24 ms for ten sweeps.  Keeping the orbital sums in shared
// memory over the sweeps saves 1 ms of traffic in twenty and costs more in resident
// blocks (19.1 against 16.7 ms for thirty sweeps, measured with six).
template <int G, int P>
__global__ void __launch_bounds__(kOccLanesThreads, 5) occupation_kernel(const OccArgs a) {
  extern __shared__ __align__(16) double occ_smem[];
  constexpr int V = G / P;  // lanes of the walker that a thread stands for
  constexpr int WPB = kOccLanesThreads / P;
  constexpr int SL = (2 * kMaxGuideParts + P - 1) / P;  // slots per thread
  const int t = threadIdx.x;
  const int gl = t % P, wl = t / P;
  const int w = blockIdx.x * WPB + wl;
  const bool live = w < a.W;
  const int N = a.N, NP = a.N + 1;
  // ln(l!) for the estimator's orbitals, then the walkers' positions
  double* lnfact = occ_smem;
  float2* zs = reinterpret_cast<float2*>(lnfact + a.Lc) + size_t(wl) * NP;
  for (int l = t; l < a.Lc; l += kOccLanesThreads) lnfact[l] = lgamma(double(l) + 1.0);

  const int wr = live ? w : a.W - 1;  // walkers beyond W compute, never write
  const int pair = int((int64_t(wr) * a.D * a.D) / a.W);
  const int rowL = pair / a.D, rowR = pair % a.D;
  const int nL = a.npairs[rowL], nR = a.npairs[rowR];
  const int32_t* partsL = a.pairs + rowL * 2 * kMaxGuideParts;
  const int32_t* partsR = a.pairs + rowR * 2 * kMaxGuideParts;
  int gk[SL], gr[SL];
  bool right[SL];
  double2 gp[SL];
#pragma unroll
  for (int q = 0; q < SL; ++q) {
    const int s = gl + q * P;
    right[q] = s >= nL;
    const int32_t* part = right[q] ? partsR + 2 * (s - nL) : partsL + 2 * s;
    gk[q] = s < nL + nR ? part[0] : 0;
    gr[q] = s < nL + nR ? part[1] : 0;
    gp[q] = make_double2(0.0, 0.0);
  }
  // warp-uniform bounds of the part loops
  const int maxL = __reduce_max_sync(0xffffffffu, nL), maxR = __reduce_max_sync(0xffffffffu, nR);
  const int max_slots = __reduce_max_sync(0xffffffffu, nL + nR);
  // initial positions: uniform in the disk of radius sqrt(2 m N)
  const float r0 = sqrtf(2.f * a.m * N);
  for (int j = gl; j < NP; j += P) {
    const U4 r = philox4x32_10(U4{uint32_t(j), 0u, uint32_t(w), kTagOccInit}, a.k0, a.k1);
    const float rho = r0 * sqrtf(u01(r.x));
    float sn, cs;
    sincospif(2.f * u01(r.y), &sn, &cs);
    zs[j] = make_float2(rho * cs, rho * sn);
  }
  __syncthreads();
  uint32_t nacc = 0;
  const float sigma = a.sigma;
  const double mm = double(a.m);
  int mine[V];  // shared particles of each lane
#pragma unroll
  for (int v = 0; v < V; ++v)
    mine[v] = N - 1 > gl + v * P ? (N - 2 - gl - v * P) / G + 1 : 0;
  const int last = N - 2;  // index of the last shared particle from zs + 1
  // power sums of part q of one side over its particles [j0, j1), to the slot's lane
  auto refresh = [&](int q, int n, const int32_t* parts, int s, int j0, int j1) {
    const int k = q < n ? parts[2 * q] : 0;
    double re = 0.0, im = 0.0;
    if (k > 0)
      for (int j = j0 + gl; j < j1; j += P) {
        const double2 v = cpow_d(make_double2(zs[j].x * a.invR, zs[j].y * a.invR), k);
        re += v.x;
        im += v.y;
      }
    const double2 p = make_double2(group_sum<P>(re), group_sum<P>(im));
#pragma unroll
    for (int u = 0; u < SL; ++u)
      if (q < n && gl + u * P == s) gp[u] = p;
  };
  for (int s = 0; s < a.burn + a.sweeps; ++s) {
    // refresh guide power sums: left over 0..N-1, right over 1..N
    for (int q = 0; q < maxL; ++q) refresh(q, nL, partsL, q, 0, N);
    for (int q = 0; q < maxR; ++q) refresh(q, nR, partsR, nL + q, 1, NP);
    float dx_l = 0.f, dy_l = 0.f;
    double lu_l = 0.0;
    for (int i = 0; i < NP; ++i) {
      // the randoms of move i, Philox {i, sweep, walker, 2}: lane gl draws
      // those of move i0 + gl for the block of P moves starting at i0
      if (i % P == 0) {
        const U4 r = philox4x32_10(U4{uint32_t(i + gl), uint32_t(s), uint32_t(w), kTagOccMove},
                                   a.k0, a.k1);
        const float rad = sqrtf(-2.f * logf(u01(r.x)));
        float sn, cs;
        sincospif(2.f * u01(r.y), &sn, &cs);
        dx_l = sigma * (rad * cs);
        dy_l = sigma * (rad * sn);
        lu_l = log(double(u01(r.z)));
      }
      const float ddx = __shfl_sync(0xffffffffu, dx_l, i % P, P);
      const float ddy = __shfl_sync(0xffffffffu, dy_l, i % P, P);
      const double lu = __shfl_sync(0xffffffffu, lu_l, i % P, P);
      const float2 zo = zs[i];
      const float2 zn = make_float2(zo.x + ddx, zo.y + ddy);
      // Jastrow log|ratio| over the shared particles 1..N-1 but i: FP32 products of
      // the squared distances, four terms at a time, one log2 per product.  Term u
      // of a lane is its particle u, or u + 1 from its own particle i on; the terms of
      // the last, partial product are masked (a factor 1).
      float lj2[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int g = gl + v * P;
        const int skip = i >= 1 && i < N && (i - 1) % G == g ? (i - 1) / G : INT_MAX;
        const int terms = mine[v] - (skip != INT_MAX);
        const float2* z = zs + 1;
        float pn = 1.f, po = 1.f;
        auto factors = [&](float2 zj, float& fn, float& fo) {
          const float dx = zn.x - zj.x, dy = zn.y - zj.y, ex = zo.x - zj.x, ey = zo.y - zj.y;
          fn = fmaf(dx, dx, dy * dy);
          fo = fmaf(ex, ex, ey * ey);
        };
        lj2[v] = 0.f;
        int u = 0;
        for (; u + 4 <= terms; u += 4) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float fn, fo;
            factors(z[(u + c) * G + (u + c >= skip ? G + g : g)], fn, fo);
            pn *= fn;
            po *= fo;
          }
          lj2[v] += __log2f(pn) - __log2f(po);
          pn = po = 1.f;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float fn, fo;
          factors(z[min((u + c) * G + (u + c >= skip ? G + g : g), last)], fn, fo);
          pn *= u + c < terms ? fn : 1.f;
          po *= u + c < terms ? fo : 1.f;
        }
        lj2[v] += __log2f(pn) - __log2f(po);
      }
      const double lj = 0.5 * 0.6931471805599453 * double(group_sumf<P>(lj2));
      const double gz = double(zo.x) * zo.x + double(zo.y) * zo.y - (double(zn.x) * zn.x + double(zn.y) * zn.y);
      // guide: this lane's log|P'/P| terms of the sides that move (0 moves the left
      // state only, N the right one).  The ratio of squared moduli is formed in FP64,
      // its log in FP32 (a power sum before and after one particle moved; an infinite
      // or zero ratio gives +-inf as the FP64 log did).
      const double2 wo = make_double2(zo.x * a.invR, zo.y * a.invR);
      const double2 wn = make_double2(zn.x * a.invR, zn.y * a.invR);
      double2 gn[SL];
      double gd = 0.0;
#pragma unroll
      for (int q = 0; q < SL; ++q) {
        gn[q] = gp[q];
        if (q * P < max_slots && gk[q] > 0 && (right[q] ? i > 0 : i < N)) {
          const double2 p0 = cpow_d(wo, gk[q]), p1 = cpow_d(wn, gk[q]);
          gn[q].x += p1.x - p0.x;
          gn[q].y += p1.y - p0.y;
          const double ratio = (gn[q].x * gn[q].x + gn[q].y * gn[q].y) /
                               (gp[q].x * gp[q].x + gp[q].y * gp[q].y);
          gd += 0.5 * 0.6931471805599453 * gr[q] * double(__log2f(float(ratio)));
        }
      }
      gd = group_sum<P>(gd);
      double delta;
      if (i == 0 || i == N) {
        delta = mm * lj + gd + 0.25 * gz;
      } else {
        const float2 z0 = zs[0], zN = zs[N];
        // ln|z' - z_0| - ln|z - z_0| and the same for z_N, in FP32 like the
        // Jastrow chains
        const float c02 = __log2f(fmaf(zn.x - z0.x, zn.x - z0.x, (zn.y - z0.y) * (zn.y - z0.y))) -
                          __log2f(fmaf(zo.x - z0.x, zo.x - z0.x, (zo.y - z0.y) * (zo.y - z0.y)));
        const float cN2 = __log2f(fmaf(zn.x - zN.x, zn.x - zN.x, (zn.y - zN.y) * (zn.y - zN.y))) -
                          __log2f(fmaf(zo.x - zN.x, zo.x - zN.x, (zo.y - zN.y) * (zo.y - zN.y)));
        const double c0 = 0.5 * 0.6931471805599453 * double(c02);
        const double cN = 0.5 * 0.6931471805599453 * double(cN2);
        delta = mm * (c0 + cN) + gd + 2.0 * mm * lj + 0.5 * gz;
      }
      const bool acc = delta >= lu;
      __syncwarp();
      if (acc) {
        if (gl == 0) zs[i] = zn;
        ++nacc;
#pragma unroll
        for (int q = 0; q < SL; ++q) gp[q] = gn[q];
      }
      __syncwarp();
    }
    if (s < a.burn) continue;
    // estimator: u = prod_{i=1}^{N-1} (z_i - z_N) conj(z_0 - z_i), of which only the
    // argument counts: group partial products, brought back to unit modulus every
    // eight factors (at most 1e4 each) and combined by the butterfly
    const float2 z0 = zs[0], zN = zs[N];
    double2 u = make_double2(1.0, 0.0);
    auto unit = [&]() {
      const double nu = sqrt(u.x * u.x + u.y * u.y);
      if (nu > 0) {
        u.x /= nu;
        u.y /= nu;
      }
    };
    int c8 = 0;
    for (int i = 1 + gl; i < N; i += P) {
      const float2 zi = zs[i];
      const double2 num = make_double2(zi.x - zN.x, zi.y - zN.y);
      const double2 den = make_double2(z0.x - zi.x, z0.y - zi.y);
      u = cmul(u, make_double2(num.x * den.x + num.y * den.y, num.y * den.x - num.x * den.y));
      if ((++c8 & 7) == 0) unit();
    }
    unit();
#pragma unroll
    for (int o = P / 2; o > 0; o >>= 1)
      u = cmul(u, make_double2(__shfl_xor_sync(0xffffffffu, u.x, o, P),
                               __shfl_xor_sync(0xffffffffu, u.y, o, P)));
    double arg = 0.0;  // arg P_R - arg P_L
#pragma unroll
    for (int q = 0; q < SL; ++q)
      if (q * P < max_slots && gk[q] > 0) {
        const double v = gr[q] * atan2(gp[q].y, gp[q].x);
        arg += right[q] ? v : -v;
      }
    const double phase = group_sum<P>(arg) + mm * atan2(u.y, u.x);
    const double2 q0 = make_double2(0.5 * (double(z0.x) * zN.x + double(z0.y) * zN.y),
                                    0.5 * (double(z0.y) * zN.x - double(z0.x) * zN.y));  // z0 conj(zN) / 2
    const double lx = 0.5 * log(q0.x * q0.x + q0.y * q0.y);
    const double phi = atan2(q0.y, q0.x);
    const double base = -0.25 * (double(z0.x) * z0.x + double(z0.y) * z0.y + double(zN.x) * zN.x +
                                 double(zN.y) * zN.y) - log(2.0 * 3.14159265358979323846);
    if (!live) continue;
    // e^{i (l phi + phase)} by rotations of P phi, one per orbital of the lane
    double2 e, rot;
    sincos(gl * phi + phase, &e.y, &e.x);
    sincos(P * phi, &rot.y, &rot.x);
    for (int l = gl; l < a.Lc; l += P) {
      // log magnitude of term l: base + l ln|z_0 conj(z_N)/2| - ln l!
      const double la = base + double(l) * lx - lnfact[l];
      if (la > -700.0) {
        const double mag = exp(la);
        double2* p = a.acc + size_t(l) * a.W + w;
        p->x += mag * e.x;
        p->y += mag * e.y;
      }
      e = cmul(e, rot);
    }
  }
  if (live && gl == 0) a.accepted[w] = nacc;
}

// Lanes per walker for N + 1 particles: about eight particles per lane.
int occupation_lanes(int N) {
  int G = 4;
  while (G < 32 && (N + G - 1) / G > 8) G *= 2;
  return G;
}

size_t occupation_smem(int N, int Lc, int threads) {
  return sizeof(double) * size_t(Lc) + sizeof(float2) * size_t(kOccLanesThreads / threads) * (N + 1);
}
size_t occupation_smem(int N, int Lc) { return occupation_smem(N, Lc, occupation_lanes(N)); }

template <int G, int P>
int launch_occ_g(const OccArgs& a, cudaStream_t st) {
  const size_t smem = occupation_smem(a.N, a.Lc, P);
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(occupation_kernel<G, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           int(smem)) != cudaSuccess)
    return LEMC_ERR_CUDA;
  constexpr int WPB = kOccLanesThreads / P;
  occupation_kernel<G, P><<<(a.W + WPB - 1) / WPB, kOccLanesThreads, smem, st>>>(a);
  return cudaPeekAtLastError() == cudaSuccess ? LEMC_OK : LEMC_ERR_CUDA;
}

// A thread stands for two of a walker's lanes from eight lanes on, where the halved
// warps still fill fifteen of an SM's twenty places and a block's positions leave room for
// five: what a warp does once per move is then shared by twice the walkers.  Ten sweeps,
// one lane -> two lanes a thread, ms: N=50, 65536 walkers 4.99 -> 4.10; 20000 (17 warps
// an SM) 1.76 -> 1.61; N=90, 30000 7.02 -> 5.35; but N=60, 7000 (6 warps) 0.92 -> 1.33.
// Four lanes a thread lose the overlap of the lanes' products (N=50: 6.4), and of four
// lanes two a thread lose too (N=20: 1.45 -> 1.82).
constexpr int kOccMinWarps = 15, kOccSMs = 148;
template <int G>
int launch_occ_lanes(const OccArgs& a, cudaStream_t st) {
  constexpr int P = G >= 8 ? G / 2 : G;
  if (int64_t(a.W) * P / 32 >= kOccMinWarps * kOccSMs && occupation_smem(a.N, a.Lc, P) <= 40 * 1024)
    return launch_occ_g<G, P>(a, st);
  return launch_occ_g<G, G>(a, st);
}

int launch_occupation(const OccArgs& a, cudaStream_t st) {
  if (occupation_smem(a.N, a.Lc) > 227 * 1024) return LEMC_ERR_CAPACITY;
  switch (occupation_lanes(a.N)) {
    case 4: return launch_occ_lanes<4>(a, st);
    case 8: return launch_occ_lanes<8>(a, st);
    case 16: return launch_occ_lanes<16>(a, st);
    default: return launch_occ_lanes<32>(a, st);
  }
}

// Sum over a pair's walkers, one warp per (orbital, pair), lanes along the walkers
// (a thread each read rows W apart: 370 us at 25 pairs of 162 orbitals, now 34).
constexpr int kOccReduceWarps = 8;
__global__ void __launch_bounds__(32 * kOccReduceWarps)
occupation_reduce(const double2* acc, int W, int D, int Lc, double2* out) {
  const int l = blockIdx.x * kOccReduceWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int pair = blockIdx.y;
  if (l >= Lc) return;
  const int w0 = int((int64_t(pair) * W + (int64_t(D) * D) - 1) / (int64_t(D) * D));
  const int w1 = int((int64_t(pair + 1) * W + (int64_t(D) * D) - 1) / (int64_t(D) * D));
  double2 s = make_double2(0.0, 0.0);
  for (int w = w0 + lane; w < w1; w += 32) {
    const double2 v = acc[size_t(l) * W + w];
    s.x += v.x;
    s.y += v.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
  }
  if (lane == 0) out[size_t(pair) * Lc + l] = s;
}

}  // namespace
}  // namespace lemc

using namespace lemc;

extern "C" int lemc_occupation(const lemc_occupation_config* cfg, double* out, double* acceptance) {
  if (!cfg || !out) return LEMC_ERR_ARG;
  const int N = cfg->particles, m = cfg->inverse_filling, W = cfg->n_walkers, Lc = cfg->l_cutoff;
  if (N < 2 || m < 1 || W < 1 || Lc < 1 || cfg->dL < 0 || cfg->dL > kMaxDegree || cfg->sweeps < 1 ||
      cfg->burn_in < 0 || !(cfg->step_sigma > 0.f))
    return LEMC_ERR_ARG;
  if (occupation_smem(N, Lc) > 227 * 1024) return LEMC_ERR_CAPACITY;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return LEMC_ERR_NODEVICE;
  }
  const Basis B = build_basis(N, {cfg->dL});
  const int D = int(B.rows.size());
  if (W < D * D) return LEMC_ERR_ARG;  // at least one walker per pair
  std::vector<int32_t> pairs(size_t(D) * 2 * kMaxGuideParts, 0), np(D, 0);
  for (int r = 0; r < D; ++r) {
    const auto& pr = B.rows[r].pairs;
    if (int(pr.size()) > kMaxGuideParts) return LEMC_ERR_CAPACITY;
    np[r] = int(pr.size());
    for (size_t q = 0; q < pr.size(); ++q) {
      pairs[size_t(r) * 2 * kMaxGuideParts + 2 * q] = pr[q].part;
      pairs[size_t(r) * 2 * kMaxGuideParts + 2 * q + 1] = pr[q].part > 0 ? pr[q].mult : 0;
    }
  }
  int32_t *d_pairs = nullptr, *d_np = nullptr;
  double2 *d_acc = nullptr, *d_out = nullptr;
  uint32_t* d_accp = nullptr;
  int st = LEMC_OK;
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess && st == LEMC_OK) st = LEMC_ERR_CUDA;
    return st == LEMC_OK;
  };
  ok(cudaMalloc(&d_pairs, pairs.size() * 4));
  ok(cudaMalloc(&d_np, np.size() * 4));
  ok(cudaMalloc(&d_acc, sizeof(double2) * size_t(Lc) * W));
  ok(cudaMalloc(&d_out, sizeof(double2) * size_t(D) * D * Lc));
  ok(cudaMalloc(&d_accp, sizeof(uint32_t) * W));
  if (st == LEMC_OK) {
    ok(cudaMemcpy(d_pairs, pairs.data(), pairs.size() * 4, cudaMemcpyHostToDevice));
    ok(cudaMemcpy(d_np, np.data(), np.size() * 4, cudaMemcpyHostToDevice));
    ok(cudaMemset(d_acc, 0, sizeof(double2) * size_t(Lc) * W));
  }
  if (st == LEMC_OK) {
    OccArgs a;
    a.W = W;
    a.N = N;
    a.m = m;
    a.D = D;
    a.Lc = Lc;
    a.sigma = cfg->step_sigma;
    a.invR = float(1.0 / std::sqrt(2.0 * m * N));
    a.k0 = uint32_t(cfg->seed);
    a.k1 = uint32_t(cfg->seed >> 32);
    a.burn = cfg->burn_in;
    a.sweeps = cfg->sweeps;
    a.pairs = d_pairs;
    a.npairs = d_np;
    a.acc = d_acc;
    a.accepted = d_accp;
    if (st == LEMC_OK) {
      const int ls = launch_occupation(a, nullptr);
      if (ls != LEMC_OK && st == LEMC_OK) st = ls;
      occupation_reduce<<<dim3((Lc + kOccReduceWarps - 1) / kOccReduceWarps, D * D),
                          32 * kOccReduceWarps>>>(d_acc, W, D, Lc, d_out);
      ok(cudaPeekAtLastError());
      ok(cudaDeviceSynchronize());
    }
  }
  if (st == LEMC_OK) {
    std::vector<double2> h(size_t(D) * D * Lc);
    std::vector<uint32_t> acc(W);
    ok(cudaMemcpy(h.data(), d_out, sizeof(double2) * h.size(), cudaMemcpyDeviceToHost));
    ok(cudaMemcpy(acc.data(), d_accp, sizeof(uint32_t) * W, cudaMemcpyDeviceToHost));
    if (st == LEMC_OK) {
      double tot = 0;
      for (uint32_t v : acc) tot += v;
      if (acceptance)
        *acceptance = tot / (double(W) * (N + 1) * (cfg->burn_in + cfg->sweeps));
      for (int pr = 0; pr < D * D; ++pr) {
        const int w0 = int((int64_t(pr) * W + (int64_t(D) * D) - 1) / (int64_t(D) * D));
        const int w1 = int((int64_t(pr + 1) * W + (int64_t(D) * D) - 1) / (int64_t(D) * D));
        const double n = double(w1 - w0) * cfg->sweeps;
        for (int l = 0; l < Lc; ++l) {
          out[2 * (size_t(pr) * Lc + l)] = h[size_t(pr) * Lc + l].x / n;
          out[2 * (size_t(pr) * Lc + l) + 1] = h[size_t(pr) * Lc + l].y / n;
        }
      }
    }
  }
  cudaFree(d_pairs);
  cudaFree(d_np);
  cudaFree(d_acc);
  cudaFree(d_out);
  cudaFree(d_accp);
  return st;
}

// ---- allocation-free variant ----------------------------------------------
// lemc_occupation_static runs the same two kernels as lemc_occupation, but all
// device memory beyond the caller's host buffers comes from one fixed,
// file-scope device array instead of cudaMalloc: the row table, the per-walker
// accumulators, the per-pair sums and the acceptance counters.  It is for
// callers that must not allocate device memory during the call: a process
// whose device memory is already handed to a caching allocator (so cudaMalloc
// would fail or fragment it), or a loop that cannot afford the implicit device
// synchronisation of cudaFree.
namespace lemc {
namespace {

constexpr size_t kOccStaticBytes = size_t(LEMC_OCC_STATIC_SCRATCH_BYTES);
constexpr int kOccStaticDevices = 64;

static __device__ __align__(256) unsigned char g_occ_scratch[kOccStaticBytes];

std::mutex g_occ_scratch_mu;
void* g_occ_scratch_ptr[kOccStaticDevices] = {};

// Address of g_occ_scratch on the current device, resolved once per device
// with that device current.
int occ_scratch_address(void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return LEMC_ERR_NODEVICE;
  }
  if (dev < 0 || dev >= kOccStaticDevices) return LEMC_ERR_CAPACITY;
  std::lock_guard<std::mutex> lock(g_occ_scratch_mu);
  if (!g_occ_scratch_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_occ_scratch);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      return LEMC_ERR_CUDA;
    }
    g_occ_scratch_ptr[dev] = p;
  }
  *out = g_occ_scratch_ptr[dev];
  return LEMC_OK;
}

constexpr size_t occ_align256(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace
}  // namespace lemc

extern "C" int lemc_occupation_static(const lemc_occupation_config* cfg, double* out,
                                      double* acceptance) {
  if (!cfg || !out) return LEMC_ERR_ARG;
  const int N = cfg->particles, m = cfg->inverse_filling, W = cfg->n_walkers, Lc = cfg->l_cutoff;
  if (N < 2 || m < 1 || W < 1 || Lc < 1 || cfg->dL < 0 || cfg->dL > kMaxDegree || cfg->sweeps < 1 ||
      cfg->burn_in < 0 || !(cfg->step_sigma > 0.f))
    return LEMC_ERR_ARG;
  if (occupation_smem(N, Lc) > 227 * 1024) return LEMC_ERR_CAPACITY;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return LEMC_ERR_NODEVICE;
  }
  const Basis B = build_basis(N, {cfg->dL});
  const int D = int(B.rows.size());
  if (W < D * D) return LEMC_ERR_ARG;  // at least one walker per pair
  std::vector<int32_t> table(size_t(D) * 2 * kMaxGuideParts + D, 0);
  int32_t* pairs = table.data();
  int32_t* np = table.data() + size_t(D) * 2 * kMaxGuideParts;
  for (int r = 0; r < D; ++r) {
    const auto& pr = B.rows[r].pairs;
    if (int(pr.size()) > kMaxGuideParts) return LEMC_ERR_CAPACITY;
    np[r] = int(pr.size());
    for (size_t q = 0; q < pr.size(); ++q) {
      pairs[size_t(r) * 2 * kMaxGuideParts + 2 * q] = pr[q].part;
      pairs[size_t(r) * 2 * kMaxGuideParts + 2 * q + 1] = pr[q].part > 0 ? pr[q].mult : 0;
    }
  }
  // scratch layout: [row table][accepted W][acc Lc x W][out D*D x Lc], 256-B aligned parts
  const size_t b_table = occ_align256(table.size() * sizeof(int32_t));
  const size_t b_accp = occ_align256(sizeof(uint32_t) * size_t(W));
  const size_t b_acc = occ_align256(sizeof(double2) * size_t(Lc) * W);
  const size_t b_out = occ_align256(sizeof(double2) * size_t(D) * D * Lc);
  if (b_table + b_accp + b_acc + b_out > kOccStaticBytes) return LEMC_ERR_CAPACITY;
  void* base = nullptr;
  int st = occ_scratch_address(&base);
  if (st != LEMC_OK) return st;
  unsigned char* s = static_cast<unsigned char*>(base);
  int32_t* d_table = reinterpret_cast<int32_t*>(s);
  uint32_t* d_accp = reinterpret_cast<uint32_t*>(s + b_table);
  double2* d_acc = reinterpret_cast<double2*>(s + b_table + b_accp);
  double2* d_out = reinterpret_cast<double2*>(s + b_table + b_accp + b_acc);
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess && st == LEMC_OK) st = LEMC_ERR_CUDA;
    return st == LEMC_OK;
  };
  // Only the per-walker accumulators must start at zero: the kernel adds
  // into them.  The table is copied, and the counters and per-pair sums are
  // written in full by the kernels.
  ok(cudaMemcpy(d_table, table.data(), table.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
  ok(cudaMemset(d_acc, 0, sizeof(double2) * size_t(Lc) * W));
  if (st == LEMC_OK) {
    OccArgs a;
    a.W = W;
    a.N = N;
    a.m = m;
    a.D = D;
    a.Lc = Lc;
    a.sigma = cfg->step_sigma;
    a.invR = float(1.0 / std::sqrt(2.0 * m * N));
    a.k0 = uint32_t(cfg->seed);
    a.k1 = uint32_t(cfg->seed >> 32);
    a.burn = cfg->burn_in;
    a.sweeps = cfg->sweeps;
    a.pairs = d_table;
    a.npairs = d_table + size_t(D) * 2 * kMaxGuideParts;
    a.acc = d_acc;
    a.accepted = d_accp;
    if (st == LEMC_OK) {
      const int ls = launch_occupation(a, nullptr);
      if (ls != LEMC_OK && st == LEMC_OK) st = ls;
      occupation_reduce<<<dim3((Lc + kOccReduceWarps - 1) / kOccReduceWarps, D * D),
                          32 * kOccReduceWarps>>>(d_acc, W, D, Lc, d_out);
      ok(cudaPeekAtLastError());
      ok(cudaDeviceSynchronize());
    }
  }
  if (st == LEMC_OK) {
    std::vector<double2> h(size_t(D) * D * Lc);
    std::vector<uint32_t> acc(W);
    ok(cudaMemcpy(h.data(), d_out, sizeof(double2) * h.size(), cudaMemcpyDeviceToHost));
    ok(cudaMemcpy(acc.data(), d_accp, sizeof(uint32_t) * W, cudaMemcpyDeviceToHost));
    if (st == LEMC_OK) {
      double tot = 0;
      for (uint32_t v : acc) tot += v;
      if (acceptance)
        *acceptance = tot / (double(W) * (N + 1) * (cfg->burn_in + cfg->sweeps));
      for (int pr = 0; pr < D * D; ++pr) {
        const int w0 = int((int64_t(pr) * W + (int64_t(D) * D) - 1) / (int64_t(D) * D));
        const int w1 = int((int64_t(pr + 1) * W + (int64_t(D) * D) - 1) / (int64_t(D) * D));
        const double n = double(w1 - w0) * cfg->sweeps;
        for (int l = 0; l < Lc; ++l) {
          out[2 * (size_t(pr) * Lc + l)] = h[size_t(pr) * Lc + l].x / n;
          out[2 * (size_t(pr) * Lc + l) + 1] = h[size_t(pr) * Lc + l].y / n;
        }
      }
    }
  }
  return st;
}
