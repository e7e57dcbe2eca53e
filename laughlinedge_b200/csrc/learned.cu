// Learned Metropolis-Hastings proposal for the Laughlin target (sm_100a).
//
// A small permutation-invariant network proposes the single-particle move:
// for particle i at z_i, the displacements to its 16 nearest other particles,
// rotated into the local (radial, tangential) frame of z_i and scaled by 1/2,
// pass through phi (2 -> 64, ReLU); their mean, with r_i/R - 1 appended,
// passes through rho (65 -> 64, ReLU -> 4) giving (mu_r, mu_t, log s_r, log s_t)
// of an axis-aligned Gaussian in that frame:
//   z' = z_i + Rot(theta_i) (mu + s * eps),   eps ~ N(0, 1)^2.
// The acceptance is the exact Metropolis-Hastings ratio
//   A = |Psi(z')|^2 q(z | z') / (|Psi(z)|^2 q(z' | z)),
// where q(z | z') is the same network evaluated at the proposed configuration
// (its own neighbours and frame), so the chain samples |Psi_m|^2 exactly
// whatever the weights are.  Weights are stored in BF16, arithmetic is FP32.
// Since ln s >= 0, ln q(z | z') <= 0: a sweep evaluates the reverse network
// only when ln u < ln A_forward (everything in ln A but the reverse density),
// which skips it for moves that would be rejected whatever its value, with
// the same decisions as the full ratio.
//
// Sampler layout: one walker per warp, positions in shared memory, lane l
// owns particles l, l+32, ...  The 16 neighbours are found from packed
// (distance^2, index) keys: each lane sorts its ceil(N/32) keys once, then 16
// rounds of a warp-wide minimum (redux.sync) of the lane heads pop them in
// ascending order; lane n keeps the n-th neighbour and forms its frame
// coordinates, which reach every lane through a per-warp shared-memory buffer.
// Each lane evaluates two of the 64 hidden units of each layer with packed FP32x2
// arithmetic; the mean phi features go through the same buffer; every reduction is
// an xor butterfly, so all lanes hold bitwise identical values and take the same
// accept decision.
// Random numbers: Philox {i, sweep, walker, 4}, drawn 32 moves at a time (one
// move per lane) and broadcast by shuffles.
//
// Training (evolution strategies + Adam, forward-only kernels): the objective
// J = E[min(1, A) |z' - z_i|^2] over (configuration, particle, eps) samples
// is estimated for 2P antithetic parameter perturbations with common random
// numbers; the ES gradient drives an Adam step on FP32 master weights.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <type_traits>
#include <vector>

#include "lemc_internal.h"
#include "lemc_rng.h"

namespace lemc {
namespace {

constexpr int kH = 64;      // hidden width
constexpr int kNbr = 16;    // neighbours
constexpr int kIn = kH + 1; // rho input: mean(phi) and r/R - 1
constexpr int kOffW1 = 0;                  // [kH][2]
constexpr int kOffB1 = kOffW1 + kH * 2;    // [kH]
constexpr int kOffW2 = kOffB1 + kH;        // [kH][kIn]
constexpr int kOffB2 = kOffW2 + kH * kIn;  // [kH]
constexpr int kOffW3 = kOffB2 + kH;        // [4][kH]
constexpr int kOffB3 = kOffW3 + 4 * kH;    // [4]
constexpr int kNParams = kOffB3 + 4;
constexpr float kInScale = 0.5f;           // displacement feature scale (1 / 2 l_B)
// proposal scales s in [1, 4] (units of l_B): the lower bound also bounds the
// reverse density, which lets a sweep skip it for hopeless moves.  Measured at
// N=200 (trained, W=65536): the network puts s at the upper bound; a lower
// bound of 1/4, 1/2 or 1 gives the same tau_int within its error and sweeps of
// 23.1, 21.7 and 20.6 ms; an upper bound of 8 doubles tau_int.
constexpr float kLogSMin = 0.f;            // log 1
constexpr float kLogSMax = 1.386294f;      // log 4
constexpr int kMaxN = 256;                 // packed kNN keys carry 8 index bits
constexpr int kMaxSlots = kMaxN / 32;      // most particles per lane
constexpr uint32_t kTagLearned = 4u, kTagTrain = 5u, kTagEs = 6u;
constexpr int kWarpsPerBlock = 4;   // sampler / evaluation blocks
// Resident sweep blocks per SM: seven leave 72 registers, room for the held parameters.
// Four sweeps at N=200, 65536 walkers: nothing held 71.1 ms with eight blocks, 72.5 with
// seven; held, 68.7 with seven, 70.8 with six; a part of them 69.6 to 72.0; records of W2
// too, 71.8 (two, five blocks) to 75.1 (ten, four).  With the four output sums in one
// butterfly (head_sums) 67.0.
constexpr int kSweepBlocks = 7;
constexpr int kTrainBlocks = 592;   // ES blocks of a step: four per SM
constexpr int kMaxDirections = 512; // perturbation directions formed at a time (19 KB each)
constexpr int kMaxSamples = 32768;  // training samples formed at a time (384 bytes each)
constexpr int kTrainWarps = 16;     // ES blocks share one perturbed weight set
constexpr float kLn2 = 0.6931471805599453f;

struct NetOut {
  float mr, mt, lr, lt;
};

// Shared-memory slot of canonical parameter k.  W2 ([kH][kIn]) is stored for
// the packed rho layer: for input column v < 32 and lane l, the 16-byte record
// (v * 32 + l) holds {W2[l][v], W2[l+32][v], W2[l][v+32], W2[l+32][v+32]};
// column kH (the r/R weight) follows at kW2Packed + hidden unit.
constexpr int kW2Packed = (kH / 2) * 32 * 4;
static_assert(kH == 64, "the packed W2 layout assumes two hidden units per lane");
__device__ __forceinline__ int p_slot(int k) {
  if (k < kOffW2 || k >= kOffB2) return k;
  const int e = k - kOffW2, h = e / kIn, c = e % kIn;
  if (c == kH) return kOffW2 + kW2Packed + h;
  return kOffW2 + ((((c & 31) * 32 + (h & 31)) << 2) | ((c >> 5) << 1) | (h >> 5));
}

// Ascending sort of a lane's S keys: comparator networks of 0, 1, 3, 5, 9, 12, 16
// and 19 comparators (each checked against the 0-1 principle).
template <int S>
__device__ __forceinline__ void sort_keys(uint32_t* k) {
  auto cx = [&](int i, int j) {
    const uint32_t a = min(k[i], k[j]), b = max(k[i], k[j]);
    k[i] = a;
    k[j] = b;
  };
  if constexpr (S == 2) {
    cx(0, 1);
  } else if constexpr (S == 3) {
    cx(0, 2); cx(0, 1); cx(1, 2);
  } else if constexpr (S == 4) {
    cx(0, 2); cx(1, 3); cx(0, 1); cx(2, 3); cx(1, 2);
  } else if constexpr (S == 5) {
    cx(0, 3); cx(1, 4); cx(0, 2); cx(1, 3); cx(0, 1); cx(2, 4); cx(1, 2); cx(3, 4); cx(2, 3);
  } else if constexpr (S == 6) {
    cx(0, 5); cx(1, 3); cx(2, 4); cx(1, 2); cx(3, 4); cx(0, 3); cx(2, 5); cx(0, 1); cx(2, 3);
    cx(4, 5); cx(1, 2); cx(3, 4);
  } else if constexpr (S == 7) {
    cx(0, 6); cx(2, 3); cx(4, 5); cx(0, 2); cx(1, 4); cx(3, 6); cx(0, 1); cx(2, 5); cx(3, 4);
    cx(1, 2); cx(4, 6); cx(2, 3); cx(4, 5); cx(1, 2); cx(3, 4); cx(5, 6);
  } else if constexpr (S == 8) {
    cx(0, 2); cx(1, 3); cx(4, 6); cx(5, 7); cx(0, 4); cx(1, 5); cx(2, 6); cx(3, 7); cx(0, 1);
    cx(2, 3); cx(4, 5); cx(6, 7); cx(2, 4); cx(3, 5); cx(1, 4); cx(3, 6); cx(1, 2); cx(3, 4);
    cx(5, 6);
  }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// warp_sum of four values at once: the first two steps of the butterfly hand half of the
// values over each, so ten shuffles do for twenty; the same pairs are added.
__device__ __forceinline__ void head_sums(float (&o)[4], int lane) {
  const bool h16 = lane & 16, h8 = lane & 8;
  float a = h16 ? o[2] : o[0], b = h16 ? o[3] : o[1];
  a += __shfl_xor_sync(0xffffffffu, h16 ? o[0] : o[2], 16);
  b += __shfl_xor_sync(0xffffffffu, h16 ? o[1] : o[3], 16);
  float s = h8 ? b : a;
  s += __shfl_xor_sync(0xffffffffu, h8 ? a : b, 8);
#pragma unroll
  for (int d = 4; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] = __shfl_sync(0xffffffffu, s, 8 * q);
}

// Squared distance of slot t's particle from zc, and whether the lane has one
// there (not `self`): S = ceil(N / 32), so only the last slot can be past the end.
template <int S>
__device__ __forceinline__ bool slot_d2(const float2* zs, int N, int self, float2 zc, int lane, int t,
                                        float& d2) {
  const int j = lane + 32 * t;
  if (!(t < S - 1 || j < N) || j == self) return false;
  const float dx = zs[j].x - zc.x, dy = zs[j].y - zc.y;
  d2 = fmaf(dx, dx, dy * dy);
  return true;
}
__device__ __forceinline__ uint32_t pack_key(float d2, int j) {
  return (__float_as_uint(d2) & 0xFFFFFF00u) | uint32_t(j);
}

// Keys of the lane's particles, and the products of their squared distances four
// slots at a time (the Jastrow factors of the centre, see propose_forward).
template <int S>
__device__ __forceinline__ void make_keys(const float2* zs, int N, int self, float2 zc, int lane,
                                          uint32_t* key, float* prod) {
#pragma unroll
  for (int t = 0; t < S; ++t) {
    float d2;
    key[t] = 0xFFFFFFFFu;
    if (t % 4 == 0) prod[t / 4] = 1.f;
    if (slot_d2<S>(zs, N, self, zc, lane, t, d2)) {
      key[t] = pack_key(d2, lane + 32 * t);
      prod[t / 4] *= d2;
    }
  }
}

// The 16 nearest in ascending key order from each lane's sorted keys: every round
// takes the warp minimum of the lane heads and its lane pops it; lane n keeps the
// n-th.  Depth = keys a lane can give; a shift of the whole list costs an
// instruction per key and round, so only the first four of more are used, and
// `lost` says (0.4 % of the time at 200 particles) that a fifth one belongs in.
template <int Depth, int S>
__device__ __forceinline__ uint32_t pop_nearest(uint32_t* key, int cnt, int lane, bool& lost) {
  uint32_t mine = 0xFFFFFFFFu, m = 0u;
#pragma unroll
  for (int n = 0; n < kNbr; ++n) {
    if (S > 1 || n < cnt) {  // S > 1: at least 32 other particles
      m = __reduce_min_sync(0xffffffffu, key[0]);
      const bool pop = key[0] == m;  // keys are unique: exactly one lane pops
#pragma unroll
      for (int t = 0; t < Depth - 1; ++t) key[t] = pop ? key[t + 1] : key[t];
      key[Depth - 1] = pop ? 0xFFFFFFFFu : key[Depth - 1];
      mine = lane == n ? m : mine;
    }
  }
  lost = false;
  if constexpr (Depth < S)
    lost = __any_sync(0xffffffffu, key[0] == 0xFFFFFFFFu && key[Depth] < m);
  return mine;
}

// The n-th nearest for lane n from every key of a lane: the rare case that
// pop_nearest reports, kept out of line for the instruction cache's sake.
template <int S>
__device__ __noinline__ uint32_t nearest_full(const float2* zs, int N, int self, float2 zc, int lane) {
  uint32_t key[S];
  float prod[2];
  bool lost;
  make_keys<S>(zs, N, self, zc, lane, key, prod);
  sort_keys<S>(key);
  return pop_nearest<S, S>(key, min(kNbr, N - 1), lane, lost);
}

// The rotation into the local (radial, tangential) frame of zc.
__device__ __forceinline__ float2 local_frame(float2 zc, float r2) {
  if (!(r2 > 1e-20f)) return make_float2(1.f, 0.f);
  const float ri = rsqrtf(r2);
  return make_float2(zc.x * ri, zc.y * ri);
}

// Frame coordinates of the lane's neighbour of zc (lane < min(kNbr, N - 1)), from the
// lane's keys about zc; the other lanes' value is unspecified.
template <int S>
__device__ __forceinline__ float2 neighbour(const float2* zs, int N, int self, float2 zc, float2 frame,
                                            int lane, uint32_t (&key)[S]) {
  static_assert(kNbr <= 32, "one neighbour per lane");
  constexpr int kDepth = S > 4 ? 4 : S;
  const int cnt = min(kNbr, N - 1);
  sort_keys<S>(key);
  bool lost;
  uint32_t mine = pop_nearest<kDepth, S>(key, cnt, lane, lost);
  if constexpr (kDepth < S) {
    if (lost) mine = nearest_full<S>(zs, N, self, zc, lane);  // warp-uniform
  }
  if (lane >= cnt) return make_float2(0.f, 0.f);
  const int j = int(mine & 0xFFu);
  const float dx = zs[j].x - zc.x, dy = zs[j].y - zc.y;
  const float xr = (dx * frame.x + dy * frame.y) * kInScale;
  const float xt = (dy * frame.x - dx * frame.y) * kInScale;
  return make_float2(xr, xt);
}

// Parameters that a lane keeps in registers over its moves: the words of hidden units
// lane, lane + 32 outside W2.  The shared-memory pipe is the busiest unit (80 %, now 76), a move
// reads them once per network evaluation, and a word costs a register here against a
// load each time; W2's records, four words a load, do not pay (see kSweepBlocks).
struct Held {
  float2 w1x, w1y, b1, w2r, b2, w3[4];
  __device__ __forceinline__ Held(const float* P, int lane) {
    w1x = make_float2(P[kOffW1 + 2 * lane], P[kOffW1 + 2 * (lane + 32)]);
    w1y = make_float2(P[kOffW1 + 2 * lane + 1], P[kOffW1 + 2 * (lane + 32) + 1]);
    b1 = make_float2(P[kOffB1 + lane], P[kOffB1 + lane + 32]);
    w2r = make_float2(P[kOffW2 + kW2Packed + lane], P[kOffW2 + kW2Packed + lane + 32]);
    b2 = make_float2(P[kOffB2 + lane], P[kOffB2 + lane + 32]);
#pragma unroll
    for (int q = 0; q < 4; ++q) w3[q] = make_float2(P[kOffW3 + q * kH + lane], P[kOffW3 + q * kH + lane + 32]);
  }
};

// The network at centre zc for particle `self` of the walker whose positions
// are zs[0..N), from the lane's keys about zc, or from its neighbours' frame
// coordinates where they are given.  All 32 lanes call it; every lane
// returns the same values.  P holds the parameters in their shared-memory slots
// (p_slot); gbuf is the warp's shared scratch of kH floats.
template <int S>
__device__ __forceinline__ NetOut net_eval(const Held& held, const float* __restrict__ P, const float2* zs, int N,
                                           int self, float2 zc, float invR, int lane, float* gbuf,
                                           uint32_t (&key)[S], const float2* given = nullptr) {
  const float r2 = zc.x * zc.x + zc.y * zc.y;
  const int cnt = min(kNbr, N - 1);
  // each lane forms the frame coordinates of its own neighbour once; phi then
  // runs over the neighbours in the same ascending order, two hidden units per lane
  // as one packed pair
  float2* nb = reinterpret_cast<float2*>(gbuf);
  if (given) {
    if (lane < cnt) nb[lane] = given[lane];
  } else {
    const float2 x = neighbour<S>(zs, N, self, zc, local_frame(zc, r2), lane, key);
    if (lane < cnt) nb[lane] = x;
  }
  __syncwarp();
  float2 g = make_float2(0.f, 0.f);
#pragma unroll
  for (int n = 0; n < kNbr; n += 2) {
    const float4 x = reinterpret_cast<const float4*>(nb)[n / 2];
    if (S > 1 || n < cnt) {
      const float2 h = __ffma2_rn(held.w1x, make_float2(x.x, x.x), __ffma2_rn(held.w1y, make_float2(x.y, x.y), held.b1));
      g = __fadd2_rn(g, make_float2(fmaxf(h.x, 0.f), fmaxf(h.y, 0.f)));
    }
    if (S > 1 || n + 1 < cnt) {
      const float2 h = __ffma2_rn(held.w1x, make_float2(x.z, x.z), __ffma2_rn(held.w1y, make_float2(x.w, x.w), held.b1));
      g = __fadd2_rn(g, make_float2(fmaxf(h.x, 0.f), fmaxf(h.y, 0.f)));
    }
  }
  if (cnt > 0) {
    const float inv = 1.f / float(cnt);
    g = __fmul2_rn(g, make_float2(inv, inv));
  }
  const float sf = sqrtf(r2) * invR - 1.f;
  // rho: the mean features reach every lane through shared memory (broadcast
  // reads); each W2 record feeds two packed FMAs for units lane, lane + 32
  __syncwarp();
  gbuf[lane] = g.x;
  gbuf[lane + 32] = g.y;
  __syncwarp();
  const float4* G4 = reinterpret_cast<const float4*>(gbuf);
  const float4* W4 = reinterpret_cast<const float4*>(P + kOffW2) + lane;
  float2 kk = make_float2(fmaf(held.w2r.x, sf, held.b2.x), fmaf(held.w2r.y, sf, held.b2.y));
  auto rho_in = [&](int v, float ga, float gb) {
    const float4 w = W4[v * 32];
    kk = __ffma2_rn(make_float2(w.z, w.w), make_float2(gb, gb), kk);
    kk = __ffma2_rn(make_float2(w.x, w.y), make_float2(ga, ga), kk);
  };
#pragma unroll
  for (int v4 = 0; v4 < 8; ++v4) {
    const float4 ga = G4[v4], gb = G4[8 + v4];
    rho_in(4 * v4, ga.x, gb.x);
    rho_in(4 * v4 + 1, ga.y, gb.y);
    rho_in(4 * v4 + 2, ga.z, gb.z);
    rho_in(4 * v4 + 3, ga.w, gb.w);
  }
  const float k0 = fmaxf(kk.x, 0.f), k1 = fmaxf(kk.y, 0.f);
  float o[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] = fmaf(held.w3[q].x, k0, held.w3[q].y * k1);
  head_sums(o, lane);
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] += P[kOffB3 + q];
  return NetOut{o[0], o[1], fminf(fmaxf(o[2], kLogSMin), kLogSMax),
                fminf(fmaxf(o[3], kLogSMin), kLogSMax)};
}

// Everything one proposed move needs, identical on all lanes.
struct Move {
  float2 zn;       // proposed position
  float log_a;     // natural log of the Metropolis-Hastings ratio
  float jump2;     // |z' - z|^2
};

// What a training sample's configuration gives all perturbations alike: the frame
// coordinates of the 16 nearest about z_i and each lane's products of squared distances.
struct Sample {
  float2 nb[kNbr];
  float po[2][32];
};

// The forward half of a move: the network at z_i, the proposed position, and
// part = ln|Psi(z')|^2 - ln|Psi(z)|^2 - ln q(z' | z), so that
// ln A = part + ln q(z | z') (reverse_log_density) in FP32 as written.
struct Forward {
  float2 zn;
  float part;
  float jump2;
};

// ln q(z | z') = -|u|^2 / 2 - ln s_r' - ln s_t' <= -2 kLogSMin, because
// ln s >= kLogSMin after the clamp and every FP32 rounding is monotone; hence
// ln A = part + ln q(z | z') never exceeds part + kLogQbMax in FP32 either.
constexpr float kLogQbMax = -2.f * kLogSMin;

// key: out, the lane's keys about the proposed position; po: the products of the
// squared distances from z, formed with the keys about it
template <int S>
__device__ __forceinline__ Forward propose_forward(const NetOut& f, const float2* zs, int N, int i,
                                                   float2 zo, const float (&po)[2], float m, float e_r,
                                                   float e_t, int lane, uint32_t (&key)[S]) {
  const float sr = __expf(f.lr), st = __expf(f.lt);
  const float dr = fmaf(sr, e_r, f.mr), dt = fmaf(st, e_t, f.mt);
  const float r2 = zo.x * zo.x + zo.y * zo.y;
  float c = 1.f, s = 0.f;
  if (r2 > 1e-20f) {
    const float ri = rsqrtf(r2);
    c = zo.x * ri;
    s = zo.y * ri;
  }
  Forward fw;
  fw.zn = make_float2(zo.x + (c * dr - s * dt), zo.y + (s * dr + c * dt));
  const float log_qf = -0.5f * (e_r * e_r + e_t * e_t) - f.lr - f.lt;
  // target ratio: m sum_j ln(|z'-z_j|^2 / |z-z_j|^2) - (|z'|^2 - |z|^2) / 2
  // FP32 products of four squared distances, one log2 per product: for
  // distances between 1e-4 and 1e4 a product stays within 1e-32 .. 1e32.
  // The distances from z' give the keys that the reverse network will need.
  float lj = 0.f;
  float pn[2];
  make_keys<S>(zs, N, i, fw.zn, lane, key, pn);
#pragma unroll
  for (int q = 0; q < (S + 3) / 4; ++q) lj += __log2f(pn[q]) - __log2f(po[q]);
  lj = warp_sum(lj);
  const float rn2 = fw.zn.x * fw.zn.x + fw.zn.y * fw.zn.y;
  const float dlp = m * kLn2 * lj - 0.5f * (rn2 - r2);
  fw.part = dlp - log_qf;
  fw.jump2 = fmaf(c * dr - s * dt, c * dr - s * dt, (s * dr + c * dt) * (s * dr + c * dt));
  return fw;
}

// ln q(z_i | z') from the network b at the proposed configuration (particle i at zn).
__device__ __forceinline__ float reverse_log_density(const NetOut& b, float2 zo, float2 zn) {
  const float rn2 = zn.x * zn.x + zn.y * zn.y;
  float cb = 1.f, sb = 0.f;
  if (rn2 > 1e-20f) {
    const float ri = rsqrtf(rn2);
    cb = zn.x * ri;
    sb = zn.y * ri;
  }
  const float bx = zo.x - zn.x, by = zo.y - zn.y;
  const float br = bx * cb + by * sb, bt = by * cb - bx * sb;
  const float ur = (br - b.mr) * __expf(-b.lr), ut = (bt - b.mt) * __expf(-b.lt);
  return -0.5f * (ur * ur + ut * ut) - b.lr - b.lt;
}

// One proposed move of particle i: the network at z, the move, and, where `wanted`
// says so, the network at the proposed configuration; lq is ln q(z | z') then, and
// the result whether it was formed.  Both networks run through one copy of the code
// (a rolled loop), which leaves the instruction cache room for its loops unrolled:
// a copy each took 73.0 ms for four sweeps at N=200, W=65536, this 72.0 (67.0 now).
template <int S, class Wanted>
__device__ __forceinline__ bool move_step(const Held& held, const float* __restrict__ P, const float2* zs, int N, int i,
                                          float invR, float m, float e_r, float e_t, int lane,
                                          float* gbuf, Forward& fw, float& lq, Wanted&& wanted,
                                          const Sample* given = nullptr) {
  const float2 zo = zs[i];
  float2 zc = zo;
  float po[2];
  uint32_t key[S];
  if (given) {
#pragma unroll
    for (int q = 0; q < (S + 3) / 4; ++q) po[q] = given->po[q][lane];
  } else {
    make_keys<S>(zs, N, i, zo, lane, key, po);
  }
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const NetOut net = net_eval<S>(held, P, zs, N, i, zc, invR, lane, gbuf, key,
                                   pass == 0 && given ? given->nb : nullptr);
    if (pass == 0) {
      fw = propose_forward<S>(net, zs, N, i, zo, po, m, e_r, e_t, lane, key);
      zc = fw.zn;
      if (!wanted(fw)) return false;
    } else {
      lq = reverse_log_density(net, zo, zc);
    }
  }
  return true;
}

template <int S>
__device__ __forceinline__ Move propose(const Held& held, const float* __restrict__ P, const float2* zs, int N, int i,
                                        float invR, float m, float e_r, float e_t, int lane,
                                        float* gbuf, const Sample* given = nullptr) {
  Forward fw;
  float lq = 0.f;
  move_step<S>(held, P, zs, N, i, invR, m, e_r, e_t, lane, gbuf, fw, lq, [](const Forward&) { return true; },
               given);
  Move mv;
  mv.zn = fw.zn;
  mv.log_a = fw.part + lq;
  mv.jump2 = fw.jump2;
  return mv;
}

__device__ __forceinline__ void box_muller(uint32_t a, uint32_t b, float& e0, float& e1) {
  const float rad = sqrtf(-2.f * __logf(u01(a)));
  float sn, cs;
  sincospif(2.f * u01(b), &sn, &cs);
  e0 = rad * cs;
  e1 = rad * sn;
}

__device__ void load_params(float* P, const __nv_bfloat16* w) {
  for (int k = threadIdx.x; k < kNParams; k += blockDim.x) P[p_slot(k)] = __bfloat162float(w[k]);
}

// w^k -> w^{k+1}, with the fused products spelt out (as in the powers skipped
// below): the recorded power sums then do not depend on how the compiler contracts
// them in its context.
__device__ __forceinline__ float2 next_power(float2 pw, float2 w) {
  return make_float2(fmaf(pw.x, w.x, -__fmul_rn(pw.y, w.y)), fmaf(pw.y, w.x, __fmul_rn(pw.x, w.y)));
}

// One walker's record from its positions, by one warp.
__device__ __forceinline__ void learned_record(const SweepArgs& a, const float2* zs, int w, int lane) {
  const int N = a.N;
  // measurement record, the plain sweep's layout: four degrees per pass over
  // the particles (w^k by the same sequence of multiplications in every pass),
  // then r^2 / r^4, then one pass per probe, so that few registers are live
  const int K = a.K;
  for (int k0 = 0; k0 < K; k0 += 4) {
    float2 acc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = make_float2(0.f, 0.f);
    for (int j = lane; j < N; j += 32) {
      const float2 z = zs[j];
      const float2 wv = make_float2(z.x * a.invR, z.y * a.invR);
      float2 pw = wv;
      for (int k = 0; k < k0; ++k)
        pw = make_float2(fmaf(pw.x, wv.x, -__fmul_rn(pw.y, wv.y)),
                         fmaf(pw.x, wv.y, __fmul_rn(pw.y, wv.x)));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        acc[k].x += pw.x;
        acc[k].y += pw.y;
        pw = next_power(pw, wv);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float sx = warp_sum(acc[k].x), sy = warp_sum(acc[k].y);
      if (k0 + k < K && ((k0 + k) & 31) == lane)
        a.rec_p[size_t(k0 + k) * a.W + w] = make_float2(sx, sy);
    }
  }
  const size_t ldw = a.ldw;
  {
    float h2 = 0.f, h4 = 0.f;
    for (int j = lane; j < N; j += 32) {
      const float2 z = zs[j];
      const float r2 = fmaf(z.x, z.x, z.y * z.y);
      h2 += r2;
      h4 = fmaf(r2, r2, h4);
    }
    h2 = warp_sum(h2);
    h4 = warp_sum(h4);
    if (lane == 0) {
      a.rec_w[LEMC_W_ONE * ldw + w] = 1.f;
      a.rec_w[LEMC_W_R2 * ldw + w] = h2;
      a.rec_w[LEMC_W_R4 * ldw + w] = h4;
      a.rec_w[LEMC_W_USER * ldw + w] = 0.f;
    }
  }
#pragma unroll
  for (int q = 0; q < LEMC_MAX_PROBES; ++q) {  // constant indices into the argument struct
    if (q >= a.n_probes) break;
    const float l = float(a.probes[q]);
    float hc = 0.f, hs = 0.f;
    for (int j = lane; j < N; j += 32) {
      const float2 z = zs[j];
      float sn, cs;
      sincosf(l * atan2f(z.y, z.x), &sn, &cs);
      hc += cs;
      hs += sn;
    }
    hc = warp_sum(hc);
    hs = warp_sum(hs);
    if (lane == 0) {
      a.rec_w[(LEMC_W_PROBE0 + 2 * q) * ldw + w] = hc;
      a.rec_w[(LEMC_W_PROBE0 + 2 * q + 1) * ldw + w] = hs;
    }
  }
}

// What bounds the sweep: shared-memory bandwidth (353 wavefronts a move, 81 % of the
// peak, half of them the W2 records) with 1220 instructions a move at 72 % of the
// issue slots.  Measured (B200, N=200, W=65536): 21.5 -> 18.0 ms a sweep, from 1492
// instructions: slots compiled for ceil(N/32), four keys a lane in the 16 rounds,
// the distances of the Jastrow factors shared with the searches, neighbour
// coordinates read back two at a time.  Two walkers a warp, which reads W2 once for
// both (264 wavefronts), took 19.1 ms: 96 registers leave 20 warps.
template <int S>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, kSweepBlocks)
learned_sweep_kernel(const SweepArgs a, const __nv_bfloat16* __restrict__ wts) {
  __shared__ __align__(16) float P[kNParams];
  __shared__ __align__(16) float gsm[kWarpsPerBlock][kH];
  extern __shared__ float2 zsm[];
  load_params(P, wts);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int w = blockIdx.x * kWarpsPerBlock + wib;
  const bool live = w < a.W;
  const int N = a.N;
  float2* zs = zsm + size_t(wib) * N;
  if (live)
    for (int j = lane; j < N; j += 32) zs[j] = a.pos[size_t(w) * N + j];
  __syncthreads();
  if (!live) return;
  __syncwarp();
  const Held held(P, lane);
  const uint32_t sweep_base = a.sweep0 + (a.sweep_ctr ? *a.sweep_ctr : 0u);
  const float m = float(a.m);
  uint32_t nacc = 0, nrev = 0;
  for (int sw = 0; sw < a.n_sweeps; ++sw) {
    const uint32_t sweep = sweep_base + uint32_t(sw);
    float er_l = 0.f, et_l = 0.f, lu_l = 0.f;
    for (int i = 0; i < N; ++i) {
      // the randoms of move i come from Philox {i, sweep, walker, 4}: lane l
      // draws those of move 32 b + l for the whole block b of 32 moves
      if ((i & 31) == 0) {
        const U4 r = philox4x32_10(U4{uint32_t(i + lane), sweep, uint32_t(w), kTagLearned},
                                   a.seed_lo, a.seed_hi);
        box_muller(r.x, r.y, er_l, et_l);
        lu_l = __logf(u01(r.z));
      }
      const float er = __shfl_sync(0xffffffffu, er_l, i & 31);
      const float et = __shfl_sync(0xffffffffu, et_l, i & 31);
      const float lu = __shfl_sync(0xffffffffu, lu_l, i & 31);
      // the reverse density is only evaluated when it can change the decision:
      // if ln u >= part + kLogQbMax, ln u >= ln A in FP32 and the move is
      // rejected as the full ratio would reject it (warp-uniform test)
      Forward fw;
      float lq = 0.f;
      bool acc = false;
      if (move_step<S>(held, P, zs, N, i, a.invR, m, er, et, lane, gsm[wib], fw, lq,
                       [&](const Forward& f) { return lu < f.part + kLogQbMax; })) {
        acc = lu < fw.part + lq;
        ++nrev;
      }
      __syncwarp();
      if (acc) {
        if (lane == (i & 31)) zs[i] = fw.zn;
        ++nacc;
      }
      __syncwarp();
    }
  }
  for (int j = lane; j < N; j += 32) a.pos[size_t(w) * N + j] = zs[j];
  if (a.accepted && lane == 0) a.accepted[w] += nacc;
  if (a.reverse_evals && lane == 0) a.reverse_evals[w] += nrev;
  if (a.measure) learned_record(a, zs, w, lane);
}

// Network outputs and proposal densities for given (configuration, particle,
// eps): out[s] = {mu_r, mu_t, log s_r, log s_t, z'.x, z'.y, ln A, |z'-z|^2}.
template <int S>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
learned_eval_kernel(const float2* __restrict__ cfgs, int n, int N, float invR, float m,
                    const int32_t* __restrict__ particle, const float* __restrict__ eps,
                    const __nv_bfloat16* __restrict__ wts, float* __restrict__ out) {
  __shared__ __align__(16) float P[kNParams];
  __shared__ __align__(16) float gsm[kWarpsPerBlock][kH];
  extern __shared__ float2 zsm[];
  load_params(P, wts);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int sidx = blockIdx.x * kWarpsPerBlock + wib;
  float2* zs = zsm + size_t(wib) * N;
  if (sidx < n)
    for (int j = lane; j < N; j += 32) zs[j] = cfgs[size_t(sidx) * N + j];
  __syncthreads();
  if (sidx >= n) return;
  __syncwarp();
  const int i = particle[sidx];
  uint32_t key[S];
  float po[2];
  make_keys<S>(zs, N, i, zs[i], lane, key, po);
  const Held held(P, lane);
  const NetOut f = net_eval<S>(held, P, zs, N, i, zs[i], invR, lane, gsm[wib], key);
  const Move mv = propose<S>(held, P, zs, N, i, invR, m, eps[2 * sidx], eps[2 * sidx + 1], lane, gsm[wib]);
  if (lane == 0) {
    float* o = out + size_t(sidx) * 8;
    o[0] = f.mr;
    o[1] = f.mt;
    o[2] = f.lr;
    o[3] = f.lt;
    o[4] = mv.zn.x;
    o[5] = mv.zn.y;
    o[6] = mv.log_a;
    o[7] = mv.jump2;
  }
}

// Direction `pair` of a step's perturbations, parameter k.
__device__ __forceinline__ float es_noise(int k, int pair, uint32_t step, uint32_t k0, uint32_t k1) {
  const U4 r = philox4x32_10(U4{uint32_t(k), uint32_t(pair), step, kTagEs}, k0, k1);
  float e0, e1;
  box_muller(r.x, r.y, e0, e1);
  return e0;
}

// The directions of `steps` steps from `step0` on, [step][pair][parameter].
__global__ void __launch_bounds__(256)
es_noise_kernel(uint32_t step0, int steps, int pairs, uint32_t k0, uint32_t k1,
                float* __restrict__ noise) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= steps * pairs * kNParams) return;
  const int k = e % kNParams, q = e / kNParams;
  noise[e] = es_noise(k, q % pairs, step0 + uint32_t(q / pairs), k0, k1);
}

// Samples first .. first + count of the run that starts at step `step0`, `batch` a step:
// a warp each.
template <int S>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
es_samples_kernel(const float2* __restrict__ cfgs, int n_cfg, int N, uint32_t step0, uint32_t k0,
                  uint32_t k1, int first, int batch, int count, Sample* __restrict__ samples) {
  extern __shared__ float2 zsm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int q = blockIdx.x * kWarpsPerBlock + wib;
  if (q >= count) return;
  const int g = first + q;
  const U4 r = philox4x32_10(U4{uint32_t(g % batch), step0 + uint32_t(g / batch), 0u, kTagTrain}, k0, k1);
  const int c = int(r.x % uint32_t(n_cfg)), i = int(r.y % uint32_t(N));
  float2* zs = zsm + size_t(wib) * N;
  for (int j = lane; j < N; j += 32) zs[j] = cfgs[size_t(c) * N + j];
  __syncwarp();
  const float2 zo = zs[i];
  uint32_t key[S];
  float po[2];
  make_keys<S>(zs, N, i, zo, lane, key, po);
#pragma unroll
  for (int v = 0; v < (S + 3) / 4; ++v) samples[q].po[v][lane] = po[v];
  const float2 x = neighbour<S>(zs, N, i, zo, local_frame(zo, zo.x * zo.x + zo.y * zo.y), lane, key);
  if (lane < kNbr) samples[q].nb[lane] = x;
}

// ES objective: the blocks (x, pert) share the batch of a perturbation, each
// evaluating kTrainWarps samples at a time with the parameters
// theta + sign * sigma * e_pair; J[pert] += sum of min(1, A) |dz|^2.
// A block takes as many rounds of samples as leave about four blocks per SM (launch
// below): with one round each, the parameters cost a block as much as its samples, 307 us
// a step at 64 perturbations of 1024 samples (N=200); now 147 us (152, two blocks per SM
// 158, eight 166 before a lane held its parameters).  What does not depend on the block is formed ahead: the directions e_pair
// (es_noise_kernel; up to kMaxDirections, more are formed by each block) and what the
// network at z_i reads of a sample's configuration, the same for every perturbation
// (es_samples_kernel).  Without the first 162 us, without either 171; the two launches
// cost 1.8 us a step.  Bound: latency, 32 warps an SM (64 registers).
template <int S>
__global__ void __launch_bounds__(kTrainWarps * 32)
es_objective_kernel(const float2* __restrict__ cfgs, int n_cfg, int N, float invR, float m,
                    const float* __restrict__ theta, float es_sigma, uint32_t step, uint32_t k0,
                    uint32_t k1, int first, int batch, const Sample* __restrict__ samples,
                    const float* __restrict__ noise, double* __restrict__ J) {
  __shared__ __align__(16) float P[kNParams];
  __shared__ __align__(16) float gsm[kTrainWarps][kH];
  __shared__ double part[kTrainWarps];
  extern __shared__ float2 zsm[];
  const int pert = blockIdx.y;
  const int pair = pert >> 1;
  const float sgn = (pert & 1) ? -es_sigma : es_sigma;
  for (int k = threadIdx.x; k < kNParams; k += blockDim.x) {
    const float e0 = noise ? noise[size_t(pair) * kNParams + k] : es_noise(k, pair, step, k0, k1);
    P[p_slot(k)] = theta[k] + sgn * e0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const Held held(P, lane);
  float2* zs = zsm + size_t(wib) * N;
  double sum = 0.0;
  for (int q = blockIdx.x * kTrainWarps + wib; q < batch; q += gridDim.x * kTrainWarps) {
    const U4 r = philox4x32_10(U4{uint32_t(first + q), step, 0u, kTagTrain}, k0, k1);
    const int c = int(r.x % uint32_t(n_cfg)), i = int(r.y % uint32_t(N));
    __syncwarp();  // the previous sample's positions are read
    for (int j = lane; j < N; j += 32) zs[j] = cfgs[size_t(c) * N + j];
    __syncwarp();
    float er, et;
    box_muller(r.z, r.w, er, et);
    const Move mv = propose<S>(held, P, zs, N, i, invR, m, er, et, lane, gsm[wib], samples + q);
    const float val = (mv.log_a >= 0.f ? 1.f : __expf(mv.log_a)) * mv.jump2;
    if (val == val) sum += val;
  }
  if (lane == 0) part[wib] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int q = 0; q < kTrainWarps; ++q) s += part[q];
    atomicAdd(&J[pert], s);
  }
}

// ES gradient (ascent on J) and one Adam step; the BF16 copy follows the
// FP32 master weights.  *trace = mean J over all perturbations (trace may be null).
// kAdamLanes threads share a parameter's sum over the pairs (a thread alone runs
// pairs Philox draws in a row on 19 blocks: 11 us; with eight 4.8, with the directions read 2.9).
constexpr int kAdamLanes = 8;
__global__ void __launch_bounds__(256)
es_adam_kernel(float* __restrict__ theta, float* __restrict__ am,
               float* __restrict__ av, __nv_bfloat16* __restrict__ wts,
               const double* __restrict__ J, int pairs, int batch, float es_sigma,
               float lr, uint32_t step, uint32_t k0, uint32_t k1,
               const float* __restrict__ noise, double* __restrict__ trace) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0 && trace) {
    double s = 0.0;
    for (int p = 0; p < 2 * pairs; ++p) s += J[p];
    *trace = s / (2.0 * pairs * batch);
  }
  const int k = t / kAdamLanes, part = t % kAdamLanes;
  double g = 0.0;
  for (int p = part; p < pairs; p += kAdamLanes) {
    if (k >= kNParams) break;
    const float e0 = noise ? noise[size_t(p) * kNParams + k] : es_noise(k, p, step, k0, k1);
    g += (J[2 * p] - J[2 * p + 1]) * double(e0);
  }
#pragma unroll
  for (int o = kAdamLanes / 2; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
  if (k >= kNParams || part != 0) return;
  const float grad = float(g / (2.0 * pairs * batch * es_sigma));
  const float b1 = 0.9f, b2 = 0.999f;
  const float mk = b1 * am[k] + (1.f - b1) * grad;
  const float vk = b2 * av[k] + (1.f - b2) * grad * grad;
  am[k] = mk;
  av[k] = vk;
  const float tt = float(step + 1);
  const float mh = mk / (1.f - powf(b1, tt)), vh = vk / (1.f - powf(b2, tt));
  const float th = theta[k] + lr * mh / (sqrtf(vh) + 1e-8f);
  theta[k] = th;
  wts[k] = __float2bfloat16_rn(th);
}

__global__ void to_bf16_kernel(const float* __restrict__ theta, __nv_bfloat16* __restrict__ wts) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < kNParams) wts[k] = __float2bfloat16_rn(theta[k]);
}

// f(integral constant S) for the S = ceil(N / 32) particle slots per lane that the
// kernels are compiled for (N <= kMaxN)
template <class F>
void with_slots(int N, F&& f) {
  static_assert(kMaxSlots == 8, "one case per slot count");
  switch ((N + 31) / 32) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 7: f(std::integral_constant<int, 7>{}); break;
    default: f(std::integral_constant<int, 8>{}); break;
  }
}

size_t walker_smem(int N, int warps = kWarpsPerBlock) { return size_t(warps) * N * sizeof(float2); }

}  // namespace

int launch_learned_sweep(const SweepArgs& a, const void* wts, cudaStream_t st) {
  if (a.N > kMaxN || a.K > kMaxDegree) return LEMC_ERR_CAPACITY;
  const int blocks = (a.W + kWarpsPerBlock - 1) / kWarpsPerBlock;
  with_slots(a.N, [&](auto s) {
    learned_sweep_kernel<s.value><<<blocks, kWarpsPerBlock * 32, walker_smem(a.N), st>>>(
        a, static_cast<const __nv_bfloat16*>(wts));
  });
  return cudaPeekAtLastError() == cudaSuccess ? LEMC_OK : LEMC_ERR_CUDA;
}

}  // namespace lemc

using namespace lemc;

struct lemc_proposal {
  int N = 0, m = 0;
  float invR = 0.f;
  float* theta = nullptr;       // FP32 master weights
  float* am = nullptr;          // Adam moments
  float* av = nullptr;
  __nv_bfloat16* wts = nullptr; // BF16 weights the samplers read
  double* J = nullptr;          // ES objective accumulators
  int J_cap = 0;
  double* trace = nullptr;
  int trace_cap = 0;
  Sample* samples = nullptr;    // training samples ahead
  int samples_cap = 0;
  float* noise = nullptr;       // perturbation directions ahead
  int noise_cap = 0;            // of this many (step, pair)s
  uint64_t train_steps = 0;     // Adam steps taken (bias correction, Philox counters)
};

namespace {

int upload_params(lemc_proposal* p, const float* host) {
  if (cudaMemcpy(p->theta, host, sizeof(float) * kNParams, cudaMemcpyHostToDevice) != cudaSuccess)
    return LEMC_ERR_CUDA;
  to_bf16_kernel<<<(kNParams + 255) / 256, 256>>>(p->theta, p->wts);
  if (cudaMemset(p->am, 0, sizeof(float) * kNParams) != cudaSuccess ||
      cudaMemset(p->av, 0, sizeof(float) * kNParams) != cudaSuccess)
    return LEMC_ERR_CUDA;
  p->train_steps = 0;
  return cudaDeviceSynchronize() == cudaSuccess ? LEMC_OK : LEMC_ERR_CUDA;
}

}  // namespace

extern "C" int lemc_proposal_n_params(int* n) {
  if (!n) return LEMC_ERR_ARG;
  *n = kNParams;
  return LEMC_OK;
}

extern "C" int lemc_proposal_create(int particles, int inverse_filling, float init_sigma,
                                    uint64_t seed, lemc_proposal** out) {
  if (!out) return LEMC_ERR_ARG;
  *out = nullptr;
  if (particles < 2 || inverse_filling < 1 || !(init_sigma > 0.f)) return LEMC_ERR_ARG;
  if (particles > kMaxN) return LEMC_ERR_CAPACITY;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return LEMC_ERR_NODEVICE;
  }
  lemc_proposal* p = new lemc_proposal();
  p->N = particles;
  p->m = inverse_filling;
  p->invR = float(1.0 / std::sqrt(2.0 * inverse_filling * particles));
  bool ok = cudaMalloc(&p->theta, sizeof(float) * kNParams) == cudaSuccess &&
            cudaMalloc(&p->am, sizeof(float) * kNParams) == cudaSuccess &&
            cudaMalloc(&p->av, sizeof(float) * kNParams) == cudaSuccess &&
            cudaMalloc(&p->wts, sizeof(__nv_bfloat16) * kNParams) == cudaSuccess;
  if (!ok) {
    lemc_proposal_destroy(p);
    return LEMC_ERR_CUDA;
  }
  // start at the plain isotropic Gaussian step init_sigma: small random
  // hidden weights, output weights near zero, output bias (0, 0, log s, log s)
  std::mt19937_64 gen(seed);
  std::normal_distribution<float> nd(0.f, 1.f);
  std::vector<float> h(kNParams, 0.f);
  for (int k = kOffW1; k < kOffB1; ++k) h[k] = 0.7f * nd(gen);
  for (int k = kOffW2; k < kOffB2; ++k) h[k] = nd(gen) / std::sqrt(float(kIn));
  for (int k = kOffW3; k < kOffB3; ++k) h[k] = 1e-3f * nd(gen);
  h[kOffB3 + 2] = h[kOffB3 + 3] = std::log(init_sigma);
  const int st = upload_params(p, h.data());
  if (st != LEMC_OK) {
    lemc_proposal_destroy(p);
    return st;
  }
  *out = p;
  return LEMC_OK;
}

extern "C" int lemc_proposal_destroy(lemc_proposal* p) {
  if (!p) return LEMC_OK;
  cudaFree(p->theta);
  cudaFree(p->am);
  cudaFree(p->av);
  cudaFree(p->wts);
  cudaFree(p->J);
  cudaFree(p->trace);
  cudaFree(p->samples);
  cudaFree(p->noise);
  delete p;
  return LEMC_OK;
}

extern "C" int lemc_proposal_get_params(const lemc_proposal* p, float* host, int n) {
  if (!p || !host || n != kNParams) return LEMC_ERR_ARG;
  return cudaMemcpy(host, p->theta, sizeof(float) * kNParams, cudaMemcpyDeviceToHost) == cudaSuccess
             ? LEMC_OK
             : LEMC_ERR_CUDA;
}

extern "C" int lemc_proposal_set_params(lemc_proposal* p, const float* host, int n) {
  if (!p || !host || n != kNParams) return LEMC_ERR_ARG;
  return upload_params(p, host);
}

extern "C" int lemc_proposal_eval(const lemc_proposal* p, const float* host_xy, int n,
                                  const int32_t* particle, const float* eps, float* out) {
  if (!p || !host_xy || !particle || !eps || !out || n <= 0) return LEMC_ERR_ARG;
  for (int s = 0; s < n; ++s)
    if (particle[s] < 0 || particle[s] >= p->N) return LEMC_ERR_ARG;
  const int N = p->N;
  float2* d_cfg = nullptr;
  int32_t* d_i = nullptr;
  float *d_e = nullptr, *d_o = nullptr;
  int st = LEMC_OK;
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess && st == LEMC_OK) st = LEMC_ERR_CUDA;
  };
  ok(cudaMalloc(&d_cfg, sizeof(float2) * size_t(n) * N));
  ok(cudaMalloc(&d_i, sizeof(int32_t) * n));
  ok(cudaMalloc(&d_e, sizeof(float) * 2 * n));
  ok(cudaMalloc(&d_o, sizeof(float) * 8 * n));
  if (st == LEMC_OK) {
    ok(cudaMemcpy(d_cfg, host_xy, sizeof(float2) * size_t(n) * N, cudaMemcpyHostToDevice));
    ok(cudaMemcpy(d_i, particle, sizeof(int32_t) * n, cudaMemcpyHostToDevice));
    ok(cudaMemcpy(d_e, eps, sizeof(float) * 2 * n, cudaMemcpyHostToDevice));
  }
  if (st == LEMC_OK) {
    with_slots(N, [&](auto s) {
      learned_eval_kernel<s.value><<<(n + kWarpsPerBlock - 1) / kWarpsPerBlock, kWarpsPerBlock * 32,
                                     walker_smem(N)>>>(d_cfg, n, N, p->invR, float(p->m), d_i, d_e,
                                                       p->wts, d_o);
    });
    ok(cudaPeekAtLastError());
    ok(cudaDeviceSynchronize());
    ok(cudaMemcpy(out, d_o, sizeof(float) * 8 * n, cudaMemcpyDeviceToHost));
  }
  cudaFree(d_cfg);
  cudaFree(d_i);
  cudaFree(d_e);
  cudaFree(d_o);
  return st;
}

extern "C" int lemc_proposal_train(lemc_proposal* p, const void* configs, int n_cfg,
                                   const lemc_train_config* tc, double* trace) {
  if (!p || !configs || n_cfg < 1 || !tc) return LEMC_ERR_ARG;
  if (tc->steps < 1 || tc->batch < 1 || tc->pairs < 1 || !(tc->lr > 0.f) || !(tc->es_sigma > 0.f))
    return LEMC_ERR_ARG;
  const int N = p->N;
  // static shared memory of es_objective_kernel: parameters, phi scratch, partial sums
  const size_t smem_static = sizeof(float) * (kNParams + kTrainWarps * kH + 2 * kTrainWarps);
  const size_t smem_dyn = walker_smem(N, kTrainWarps);
  if (smem_static + smem_dyn > 227 * 1024) return LEMC_ERR_CAPACITY;
  if (smem_static + smem_dyn > 48 * 1024) {
    cudaError_t e = cudaSuccess;
    with_slots(N, [&](auto s) {
      e = cudaFuncSetAttribute(es_objective_kernel<s.value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(smem_dyn));
    });
    if (e != cudaSuccess) return LEMC_ERR_CUDA;
  }
  if (p->J_cap < 2 * tc->pairs) {
    cudaFree(p->J);
    p->J = nullptr;
    if (cudaMalloc(&p->J, sizeof(double) * 2 * tc->pairs) != cudaSuccess) return LEMC_ERR_CUDA;
    p->J_cap = 2 * tc->pairs;
  }
  if (p->trace_cap < tc->steps) {
    cudaFree(p->trace);
    p->trace = nullptr;
    p->trace_cap = 0;
    if (cudaMalloc(&p->trace, sizeof(double) * tc->steps) != cudaSuccess ||
        cudaMemset(p->trace, 0, sizeof(double) * tc->steps) != cudaSuccess)
      return LEMC_ERR_CUDA;
    p->trace_cap = tc->steps;
  }
  // the samples of several steps, or a part of one step's, at a time: 12 MB at most,
  // kept with the proposal like the directions' 10 MB
  const int64_t all = int64_t(tc->steps) * tc->batch;
  const int part = std::min(tc->batch, kMaxSamples);         // of one step
  const int ahead = std::max(1, std::min(tc->steps, kMaxSamples / tc->batch));  // steps
  const int cap = int(std::min<int64_t>(all, int64_t(ahead) * part));
  if (p->samples_cap < cap) {
    cudaFree(p->samples);
    p->samples = nullptr;
    p->samples_cap = 0;
    if (cudaMalloc(&p->samples, sizeof(Sample) * cap) != cudaSuccess) return LEMC_ERR_CUDA;
    p->samples_cap = cap;
  }
  // directions of as many steps, or none (each block forms its own) if one step has more
  const int dirs = std::min(tc->steps, kMaxDirections / tc->pairs);
  if (p->noise_cap < dirs * tc->pairs) {
    cudaFree(p->noise);
    p->noise = nullptr;
    p->noise_cap = 0;
    if (cudaMalloc(&p->noise, sizeof(float) * size_t(dirs) * tc->pairs * kNParams) != cudaSuccess)
      return LEMC_ERR_CUDA;
    p->noise_cap = dirs * tc->pairs;
  }
  const uint32_t k0 = uint32_t(tc->seed), k1 = uint32_t(tc->seed >> 32);
  const int perts = 2 * tc->pairs;
  const float2* cfgs = static_cast<const float2*>(configs);
  for (int s = 0; s < tc->steps; ++s) {
    const uint32_t step = uint32_t(p->train_steps);
    if (cudaMemsetAsync(p->J, 0, sizeof(double) * 2 * tc->pairs) != cudaSuccess) return LEMC_ERR_CUDA;
    const float* noise = nullptr;
    if (dirs > 0) {
      if (s % dirs == 0) {
        const int n = std::min(dirs, tc->steps - s);
        es_noise_kernel<<<(n * tc->pairs * kNParams + 255) / 256, 256>>>(step, n, tc->pairs, k0, k1,
                                                                         p->noise);
      }
      noise = p->noise + size_t(s % dirs) * tc->pairs * kNParams;
    }
    for (int64_t begin = 0; begin < tc->batch; begin += part) {
      const int first = int(begin);
      const int n = std::min(part, tc->batch - first);  // of this step in this launch
      const int rounds = (n + kTrainWarps - 1) / kTrainWarps;
      const dim3 grid(std::min(rounds, std::max(1, kTrainBlocks / perts)), perts);
      with_slots(N, [&](auto sl) {
        if (s % ahead == 0) {
          const int count = part < tc->batch ? n : std::min(ahead, tc->steps - s) * tc->batch;
          es_samples_kernel<sl.value><<<(count + kWarpsPerBlock - 1) / kWarpsPerBlock,
                                        kWarpsPerBlock * 32, walker_smem(N)>>>(
              cfgs, n_cfg, N, step, k0, k1, first, tc->batch, count, p->samples);
        }
        es_objective_kernel<sl.value><<<grid, kTrainWarps * 32, walker_smem(N, kTrainWarps)>>>(
            cfgs, n_cfg, N, p->invR, float(p->m), p->theta, tc->es_sigma, step, k0, k1, first, n,
            p->samples + size_t(s % ahead) * part, noise, p->J);
      });
    }
    // Entry s + step of the trace, where it has one: with step counted from the
    // weights' last reset, a first call's entry 2 s holds step s.
    const uint64_t at = uint64_t(s) + step;
    es_adam_kernel<<<(kNParams * kAdamLanes + 255) / 256, 256>>>(p->theta, p->am, p->av, p->wts, p->J,
                                                    tc->pairs, tc->batch, tc->es_sigma, tc->lr,
                                                    step, k0, k1, noise,
                                                    at < uint64_t(p->trace_cap) ? p->trace + at : nullptr);
    if (cudaPeekAtLastError() != cudaSuccess) return LEMC_ERR_CUDA;
    ++p->train_steps;
  }
  if (cudaDeviceSynchronize() != cudaSuccess) return LEMC_ERR_CUDA;
  if (trace &&
      cudaMemcpy(trace, p->trace, sizeof(double) * tc->steps, cudaMemcpyDeviceToHost) != cudaSuccess)
    return LEMC_ERR_CUDA;
  return LEMC_OK;
}

// Weights of a proposal for the samplers of lemc_ctx (device BF16 array).
const void* lemc_proposal_weights(const lemc_proposal* p) { return p ? p->wts : nullptr; }
int lemc_proposal_particles(const lemc_proposal* p) { return p ? p->N : 0; }
int lemc_proposal_filling(const lemc_proposal* p) { return p ? p->m : 0; }
