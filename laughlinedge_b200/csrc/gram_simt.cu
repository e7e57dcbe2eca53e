// FP64 accumulation of the weighted Gram matrices (SIMT, exact products).
//
//   G_h[a][b] += sum_w  W_h(w) * conj(v_a(w)) * v_b(w)
//
// for three weight planes h at once.  The FP32 inputs are widened to FP64
// before multiplying, so each product is exact and the only rounding is the
// FP64 summation.  This is the reference accumulation the tensor-core path is
// checked against, and the production path for LEMC_GRAM_FP64.
//
// Also here: the row sums of the reference estimator (LEMC_GUIDE_ROW),
// fg[a][b] = sum v_b/v_a, gg = sum |v_b/v_a|^2, and V-weighted sums, over the
// walkers guided by row a (reference em_spectrum.cu:99-115).
#include <cuda_runtime.h>

#include "lemc_internal.h"

namespace lemc {
namespace {

constexpr int kGramThreads = 256;
constexpr size_t kGramSmem = 40 * 1024;

// Tile shapes (rows a x rows b).  A block of 256 threads computes one tile of
// one walker range; a thread owns 2 x 2 outputs (24 FP64 sums), so a tile takes
// TA TB / 4 threads and the block holds NG = 1024 / (TA TB) groups that share
// each staged chunk of walkers, summed at the end.
//
// Bound: the FP64 pipe (64 FMA/cycle/SM; 65 % busy), with the shared-memory loads of the
// operands beside it.  A (pair, walker) costs 10 FMAs: 4 for conj(a) b, 6 for the three
// weighted sums (folding the weights into one operand first would cost 12).  The staged
// values are widened to FP64 once per chunk; widening inside the product loop, seven
// conversions for every 10 FMAs at a quarter of their rate, and one output per thread
// held the previous 16 x 16 form at 5 % of the pipe.  A thread stages a value's two
// components together (one 16-byte store instead of two of 8, half the index work: 2.96
// -> 2.77 ms for 526 states at 65536 walkers, and 2.70 with four walkers in flight).  4 x 2
// outputs a thread save a third of the loads but leave one block an SM, 2.91 ms.  The
// small shapes keep the padding of small sectors low and spread their walkers over more
// blocks.
//
// Measured (B200): Gram of 526 states (N=100, dL 0,2..16) at 65536 walkers 2.70 ms, their
// cross planes 8.3 ms (40.3 in the 16 x 16 form); 29 states (N=8, dL 1..6) at 4096
// walkers 21 us (101).
template <int TA, int TB>
struct Tile {
  static constexpr int TX = TB / 2, TY = TA / 2;  // threads: tx over b, ty over a
  static constexpr int TPG = TX * TY;
  static constexpr int NG = kGramThreads / TPG;
  static constexpr int CH = TA == 8 ? (TB == 8 ? 128 : TB == 16 ? 64 : 32) : (TB == 16 ? 64 : 32);
  static constexpr int SA = TA + 1, SB = TB + 1;  // double2 row strides per walker
  static constexpr int NF = (TA + TB) * CH / kGramThreads;  // staged values per thread
  static constexpr size_t kStage = sizeof(double2) * CH * (SA + SB) + sizeof(double) * 3 * CH;
  static constexpr size_t kReduce = NG > 1 ? sizeof(double) * (NG / 2) * TPG * 24 : 0;
  static_assert(NF * kGramThreads == (TA + TB) * CH && CH % 32 == 0 && CH % NG == 0, "tile shape");
  static_assert(kStage <= kGramSmem && kReduce <= kGramSmem, "tile shape");
};

// NW = 3: all three weight planes; NW = 1: only the first (the job's others are off)
template <int TA, int TB, int NW>
__device__ __forceinline__ void gram_tile(const float* __restrict__ V, int ldv,
                                          const float* __restrict__ rec_w, int ldw, int wbeg,
                                          int wend, const GramJob& jb, double* __restrict__ out,
                                          size_t plane, unsigned char* smem) {
  using T = Tile<TA, TB>;
  double2* sa = reinterpret_cast<double2*>(smem);      // [CH][SA]
  double2* sb = sa + T::CH * T::SA;                    // [CH][SB]
  double* wt = reinterpret_cast<double*>(sb + T::CH * T::SB);  // [3][CH]
  const int tid = threadIdx.x;
  const int g = tid / T::TPG, tg = tid % T::TPG;
  // 16 threads over b: a warp takes 8 of them by 4 over a, whose 16-byte loads read fewer
  // distinct rows than 16 by 2
  constexpr bool kSquare = T::TX == 16;
  const int tx = kSquare ? (tg & 7) + ((tg >> 5) & 1) * 8 : tg % T::TX;
  const int ty = kSquare ? ((tg >> 3) & 3) + (tg >> 6) * 4 : tg / T::TX;

  // staged element e = it * 256 + tid: walker e % CH of tile row e / CH, the rows of a
  // first (a warp reads 32 consecutive walkers of a row)
  float2 pf[T::NF];
  float pw[3] = {0.f, 0.f, 0.f};
  auto fetch = [&](int c0) {
#pragma unroll
    for (int it = 0; it < T::NF; ++it) {
      const int e = it * kGramThreads + tid;
      const int s = e % T::CH, q = e / T::CH;
      const bool isb = q >= TA;
      const int r = isb ? jb.b0 + q - TA : jb.a0 + q;
      const int dim = isb ? jb.Db : jb.Da;
      const float* v = V + (size_t)((isb ? jb.row_b : jb.row_a) + r) * ldv + c0 + s;
      const bool in = c0 + s < wend && r < dim;
      pf[it] = in ? make_float2(v[0], v[(size_t)dim * ldv]) : make_float2(0.f, 0.f);
    }
    if (tid < T::CH) {
      const int wi = c0 + tid;
      const float one = wi < wend ? rec_w[(size_t)LEMC_W_ONE * ldw + wi] : 0.f;
#pragma unroll
      for (int h = 0; h < NW; ++h) {
        const int pl = jb.plane[h];
        pw[h] = 0.f;
        if (wi < wend && pl >= 0) pw[h] = pl == LEMC_W_ONE ? one : one * rec_w[(size_t)pl * ldw + wi];
      }
    }
  };
  auto stage = [&]() {
#pragma unroll
    for (int it = 0; it < T::NF; ++it) {
      const int e = it * kGramThreads + tid;
      const int s = e % T::CH, q = e / T::CH;
      (q < TA ? sa[s * T::SA + q] : sb[s * T::SB + q - TA]) = make_double2(pf[it].x, pf[it].y);
    }
    if (tid < T::CH) {
#pragma unroll
      for (int h = 0; h < NW; ++h) wt[h * T::CH + tid] = double(pw[h]);
    }
  };

  double2 acc[NW][2][2];
#pragma unroll
  for (int h = 0; h < NW; ++h)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) acc[h][i][j] = make_double2(0.0, 0.0);

  fetch(wbeg);
  for (int c0 = wbeg; c0 < wend; c0 += T::CH) {
    __syncthreads();  // the previous chunk is consumed
    stage();
    __syncthreads();
    if (c0 + T::CH < wend) fetch(c0 + T::CH);  // lands while this chunk is summed
#pragma unroll 4
    for (int s = g; s < T::CH; s += T::NG) {
      double2 a[2], b[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[i] = sa[s * T::SA + ty + i * T::TY];
        b[i] = sb[s * T::SB + tx + i * T::TX];
      }
      double w[NW];
#pragma unroll
      for (int h = 0; h < NW; ++h) w[h] = wt[h * T::CH + s];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const double pr = a[i].x * b[j].x + a[i].y * b[j].y;  // conj(a) b
          const double pi = a[i].x * b[j].y - a[i].y * b[j].x;
#pragma unroll
          for (int h = 0; h < NW; ++h) {
            acc[h][i][j].x += w[h] * pr;
            acc[h][i][j].y += w[h] * pi;
          }
        }
    }
  }
  // fold the NG walker groups into group 0
  if constexpr (T::NG > 1) {
    double2* red = reinterpret_cast<double2*>(smem);
    constexpr int kV = NW * 4;
#pragma unroll
    for (int off = T::NG / 2; off > 0; off >>= 1) {
      __syncthreads();
      if (g >= off && g < 2 * off) {
#pragma unroll
        for (int v = 0; v < kV; ++v)
          red[v * (off * T::TPG) + (g - off) * T::TPG + tg] = acc[v >> 2][(v >> 1) & 1][v & 1];
      }
      __syncthreads();
      if (g < off) {
#pragma unroll
        for (int v = 0; v < kV; ++v) {
          const double2 o = red[v * (off * T::TPG) + g * T::TPG + tg];
          acc[v >> 2][(v >> 1) & 1][v & 1].x += o.x;
          acc[v >> 2][(v >> 1) & 1][v & 1].y += o.y;
        }
      }
    }
    if (g > 0) return;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int a = jb.a0 + ty + i * T::TY, b = jb.b0 + tx + j * T::TX;
      if (a >= jb.Da || b >= jb.Db) continue;
      const size_t o = 2 * ((size_t)jb.out + (size_t)a * jb.Db + b);
      const size_t ot = 2 * ((size_t)jb.mirror + (size_t)b * jb.Da + a);
#pragma unroll
      for (int h = 0; h < NW; ++h) {
        atomicAdd(out + o + 2 * plane * h, acc[h][i][j].x);
        atomicAdd(out + o + 2 * plane * h + 1, acc[h][i][j].y);
        if (jb.mirror >= 0) {  // the transposed block: conj of the same sum (real weights)
          atomicAdd(out + ot + 2 * plane * h, acc[h][i][j].x);
          atomicAdd(out + ot + 2 * plane * h + 1, -acc[h][i][j].y);
        }
      }
    }
}

__global__ void __launch_bounds__(kGramThreads, 2)
gram_simt_kernel(const float* __restrict__ V, int ldv, const float* __restrict__ rec_w, int ldw,
                 int W, int per, const GramJob* __restrict__ jobs, double* __restrict__ out0,
                 size_t plane0, double* __restrict__ out1, size_t plane1) {
  __shared__ __align__(16) unsigned char smem[kGramSmem];
  const GramJob jb = jobs[blockIdx.x];
  const int wbeg = blockIdx.y * per;
  const int wend = min(W, wbeg + per);
  double* out = jb.buf == 0 ? out0 : out1;
  const size_t plane = jb.buf == 0 ? plane0 : plane1;
  if (!out || wbeg >= wend) return;
  const bool one = jb.plane[1] < 0 && jb.plane[2] < 0;
#define LEMC_TILE(A, B)                                                                   \
  if (one)                                                                                \
    gram_tile<A, B, 1>(V, ldv, rec_w, ldw, wbeg, wend, jb, out, plane, smem);             \
  else                                                                                    \
    gram_tile<A, B, 3>(V, ldv, rec_w, ldw, wbeg, wend, jb, out, plane, smem);             \
  break
  switch (jb.ta * 64 + jb.tb) {
    case 8 * 64 + 8: LEMC_TILE(8, 8);
    case 8 * 64 + 16: LEMC_TILE(8, 16);
    case 8 * 64 + 32: LEMC_TILE(8, 32);
    case 16 * 64 + 16: LEMC_TILE(16, 16);
    case 16 * 64 + 32: LEMC_TILE(16, 32);
    case 32 * 64 + 32: LEMC_TILE(32, 32);
  }
#undef LEMC_TILE
}

// Row sums of the reference estimator.  Block (row a, column b); the threads
// run over the walkers guided by row a.  Accumulators per (a, b):
//   [0,1] sum v_b/v_a      [2] sum |v_b/v_a|^2
//   [3,4] sum r2 v_b/v_a   [5,6] sum r4 v_b/v_a
//   [7,8] sum cos v_b/v_a  [9,10] sum sin v_b/v_a   [11,12] sum U v_b/v_a
// (cos/sin of the first angular probe)
//
// Bound by latency: a row holds a few hundred walkers, so one block per (a, b)
// puts all D^2 sums in flight and a thread meets a handful of walkers.  Threads
// over walkers also read V along its contiguous axis (a thread per column read
// 32 rows, ldv apart, per warp load).  Measured (B200, 29 rows, 16384 walkers):
// 69 -> 12 us a launch.
constexpr int NROWACC = 13;
constexpr int kRowThreads = 256;

__global__ void __launch_bounds__(kRowThreads)
row_accumulate_kernel(const float* __restrict__ V, int ldv, const float* __restrict__ rec_w,
                      int ldw, const int32_t* __restrict__ row_first, int D,
                      const int32_t* __restrict__ row_re, const int32_t* __restrict__ row_im,
                      double* __restrict__ acc_out) {
  const int a = blockIdx.x, b = blockIdx.y;
  const int w0 = row_first[a], w1 = row_first[a + 1];
  double acc[NROWACC];
#pragma unroll
  for (int q = 0; q < NROWACC; ++q) acc[q] = 0.0;
  const size_t ra = row_re[a], ia = row_im[a], rb = row_re[b], ib = row_im[b];
  for (int w = w0 + threadIdx.x; w < w1; w += kRowThreads) {
    const double var = V[ra * ldv + w], vai = V[ia * ldv + w];
    const double vbr = V[rb * ldv + w], vbi = V[ib * ldv + w];
    const double den = var * var + vai * vai;
    // v_b / v_a = v_b conj(v_a) / |v_a|^2
    const double rr = (vbr * var + vbi * vai) / den;
    const double ri = (vbi * var - vbr * vai) / den;
    const double one = rec_w[(size_t)LEMC_W_ONE * ldw + w];
    const double h2 = rec_w[(size_t)LEMC_W_R2 * ldw + w];
    const double h4 = rec_w[(size_t)LEMC_W_R4 * ldw + w];
    const double hc = rec_w[(size_t)LEMC_W_PROBE0 * ldw + w];
    const double hs = rec_w[(size_t)(LEMC_W_PROBE0 + 1) * ldw + w];
    const double hu = rec_w[(size_t)LEMC_W_USER * ldw + w];
    acc[0] += one * rr;
    acc[1] += one * ri;
    acc[2] += one * (rr * rr + ri * ri);
    acc[3] += h2 * rr;
    acc[4] += h2 * ri;
    acc[5] += h4 * rr;
    acc[6] += h4 * ri;
    acc[7] += hc * rr;
    acc[8] += hc * ri;
    acc[9] += hs * rr;
    acc[10] += hs * ri;
    acc[11] += hu * rr;
    acc[12] += hu * ri;
  }
  __shared__ double red[kRowThreads / 32][NROWACC];
#pragma unroll
  for (int q = 0; q < NROWACC; ++q) {
    double v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < NROWACC) {
    double v = 0.0;
#pragma unroll
    for (int l = 0; l < kRowThreads / 32; ++l) v += red[l][threadIdx.x];
    acc_out[((size_t)a * D + b) * NROWACC + threadIdx.x] += v;
  }
}

}  // namespace

int launch_gram_simt(const float* V, int ldv, const float* rec_w, int ldw, int W, const GramJob* jobs,
                     int n_jobs, double* out0, size_t plane0, double* out1, size_t plane1,
                     cudaStream_t st) {
  if (n_jobs <= 0) return LEMC_OK;
  // Walker split: about sixteen blocks for each of the 2 x 148 resident slots, so
  // the last wave is a small share (cross planes of 526 states,
  // before the paired staging: 9.2 ms; with six blocks a slot 9.9 ms), in whole
  // 128-walker chunks; every split costs one FP64 atomic per output and plane.
  const long want = (16L * 2 * 148 + n_jobs - 1) / n_jobs;
  const int chunks = (W + 127) / 128;
  const int splits = int(want < 1 ? 1 : want > chunks ? chunks : want);
  const int per = (chunks + splits - 1) / splits * 128;
  const dim3 grid(n_jobs, (W + per - 1) / per);
  gram_simt_kernel<<<grid, kGramThreads, 0, st>>>(V, ldv, rec_w, ldw, W, per, jobs, out0, plane0,
                                                  out1, plane1);
  return cudaPeekAtLastError() == cudaSuccess ? LEMC_OK : LEMC_ERR_CUDA;
}

int launch_row_accumulate(const float* V, int ldv, const float* rec_w, int ldw, int W,
                          const int32_t* row_first, int n_rows, int D, const int32_t* row_re,
                          const int32_t* row_im, double* acc, cudaStream_t st) {
  if (n_rows <= 0 || D <= 0) return LEMC_OK;
  (void)W;
  const dim3 grid(n_rows, D);
  row_accumulate_kernel<<<grid, kRowThreads, 0, st>>>(V, ldv, rec_w, ldw, row_first, D, row_re, row_im,
                                              acc);
  return cudaPeekAtLastError() == cudaSuccess ? LEMC_OK : LEMC_ERR_CUDA;
}

}  // namespace lemc
