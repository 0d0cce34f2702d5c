// Coefficient estimation for a fixed frequency set, and its adjoint.
//
// With the identified set held fixed (no identification, no subtraction of
// other modes), Iterate's coefficient estimate (src/iterate.cc:146-171) is a
// linear map c = A x. For each given k0 with k1 = (a k0 + b) mod n, bin
// beta = floor(k1 B / n) and xi0 = k1/n - (beta + 1/2)/B:
//   c(k0) = s_k sum_t sum_r U_{t,r}[beta] e^{-2 pi i tau_{t,r} k1 / n},
//   s_k   = e^{-2 pi i c k0 / n} / (wf(xi0) T (1 + 2L)),
// where U_{t,r} are BinInTime's bins of row tau_{t,r} (q_t, q_t +- B 2^s):
//   U_tau[beta] = sum_{|t| <= p2} x[(a (tau + t) + c) mod n] wt(t)
//                 e^{2 pi i b (tau + t) / n} e^{-2 pi i t (2 beta + 1) / (2B)}.
// The adjoint dx = A^H g (g = dL/dc in torch's convention) is
//   G_{t,r}[beta] = sum_{k in beta} conj(s_k) g_k e^{2 pi i tau_{t,r} k1 / n},
//   H_{t,r}[m]    = sum_beta G_{t,r}[beta] e^{2 pi i beta m / B}   (inverse DFT),
//   dx[(a (tau + t) + c) mod n] += wt(t) e^{-2 pi i b (tau + t) / n}
//                                  e^{pi i t / B} H_{t,r}[t mod B]
// i.e. per-bin spreading over the rows, an inverse size-B DFT, unfolding to
// the window support and a windowed scatter-add at the permuted indices.
// All in FP64; the scatter-add uses FP64 atomics (rows overlap in x).
#include "common.cuh"
#include "launch.h"

namespace mpsft {

namespace {

__device__ inline int64_t RowOffset(int r, int64_t B) {
  if (r == 0) return 0;
  const int s = (r - 1) / 2;
  return (r & 1) ? (B << s) : -(B << s);
}

struct ModeSetup {
  int64_t k1;
  int beta;
  double2 s;  // e^{-2 pi i c k0 / n} / (wf T (1 + 2L))
};

// The mode's setup, by G neighbouring lanes of a warp (every lane calls). The two
// erf of WindowInFreq are evaluated by the even and the odd lanes, each one of them
// (FP64 runs at two lanes per clock, so a warp pays for an erf once per evaluation).
template <int G>
__device__ inline ModeSetup SetupMode(const SigIter &it, int32_t k0, int lane) {
  const int64_t n = it.n, B = it.bins;
  const ModN mod{uint32_t(n), it.n_inv};
  ModeSetup m;
  m.k1 = mod(int64_t(it.a) * k0 + it.b);
  m.beta = int(mod.quot(m.k1 * B));
  // k1/n - (beta + 1/2)/B from its exact numerator (|num| < 2^53)
  const double xi0 =
      double(2 * B * m.k1 - (2 * int64_t(m.beta) + 1) * n) * it.xi_scale;
  double wf;
  if constexpr (G == 1) {
    wf = WindowInFreq(it, xi0);
  } else {
    const double h = 0.5 * it.width;
    const double e = erf((xi0 + ((lane & 1) ? -h : h)) * it.erf_d);
    const double other = __shfl_xor_sync(0xffffffffu, e, 1);
    wf = 0.5 * ((lane & 1) ? other - e : e - other);
  }
  const double scale = 1.0 / (wf * double(it.trials * (1 + 2 * it.bits)));
  m.s = cscale(Phase64(it, -int64_t(it.c) * k0), scale);
  return m;
}

// forward: G lanes of a warp per mode, over the (trial, row) values of the mode's
// bin in ubuf (trials x rows x bins_cap), then a shuffle tree. A mode is some 250
// FP64 operations of setup and a dozen per row. Few modes: a warp each, in a block
// of its own, so that they spread over the SMs' FP64 pipes and no lane walks the
// rows one after another (200 modes, 25 rows: 25 us with a thread per mode, a call
// of 162 us; 150 us with a warp each). Many: a warp per mode evaluates the setup 32
// times over, and fewer lanes per mode are faster (LanesPerMode).
template <int G>
__global__ void __launch_bounds__(32) k_estimate(const SigIter *__restrict__ its,
                                                 const int32_t *k0s, int64_t m,
                                                 double2 *coef) {
  const SigIter &it = PdlEnterLoaded(its, 0);
  const int lane = threadIdx.x, sub = lane & (G - 1);
  constexpr int kModes = 32 / G;
  for (int64_t i0 = int64_t(blockIdx.x) * kModes; i0 < m;
       i0 += int64_t(gridDim.x) * kModes) {
    const int64_t i = i0 + lane / G;
    const bool live = i < m;
    const ModeSetup ms = SetupMode<G>(it, k0s[live ? i : m - 1], lane);
    double2 acc = make_double2(0.0, 0.0);
    for (int j = sub; j < it.trials * it.rows; j += G) {
      const int t = j / it.rows, r = j - t * it.rows;
      const int64_t tau = int64_t(it.q[t]) + RowOffset(r, it.bins);
      const double2 u = it.ubuf[size_t(j) * it.bins_cap + ms.beta];
      acc = cadd(acc, cmul(u, Phase64(it, -tau * ms.k1)));
    }
    // (lanes past the last mode take part in the shuffles)
    __syncwarp();
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
      acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if (live && sub == 0) coef[i] = cmul(acc, ms.s);
  }
}

// adjoint, step 1: G_rows (in the fold buffer, zeroed) += conj(s_k) g_k
// e^{2 pi i tau k1 / n}, stored conjugated for the forward FFT that follows
// (conj(DFT(conj(G_rows))) is the inverse DFT of G_rows). G lanes per mode over the
// rows, as k_estimate (200 modes: 29 us with a thread per mode; the adjoint's call
// went from 565 to 545 us with a warp each).
template <int G>
__global__ void __launch_bounds__(32) k_adjoint_spread(const SigIter *__restrict__ its,
                                                       const int32_t *k0s,
                                                       const double2 *g, int64_t m) {
  const SigIter &it = PdlEnterLoaded<false>(its, 0);
  const int lane = threadIdx.x, sub = lane & (G - 1);
  constexpr int kModes = 32 / G;
  double2 *rows = reinterpret_cast<double2 *>(it.fold);
  for (int64_t i0 = int64_t(blockIdx.x) * kModes; i0 < m;
       i0 += int64_t(gridDim.x) * kModes) {
    const int64_t i = i0 + lane / G;
    const bool live = i < m;
    const ModeSetup ms = SetupMode<G>(it, k0s[live ? i : m - 1], lane);
    if (live) {
      const double2 w = cmul(cconj(ms.s), g[i]);
      for (int j = sub; j < it.trials * it.rows; j += G) {
        const int t = j / it.rows, r = j - t * it.rows;
        const int64_t tau = int64_t(it.q[t]) + RowOffset(r, it.bins);
        const double2 v = cconj(cmul(w, Phase64(it, tau * ms.k1)));
        double2 *dst = rows + size_t(j) * it.bins_cap + ms.beta;
        atomicAdd(&dst->x, v.x);
        atomicAdd(&dst->y, v.y);
      }
    }
    __syncwarp();
  }
}

// adjoint, step 3: after ubuf = e^{2 pi i b tau / n} DFT(conj(G)) (the row
// transform with its row factors), conj(ubuf) = e^{-2 pi i b tau / n} H; one
// thread per (trial, row, t) scatters it, times the conjugate of the modulated
// window (wmod), into dx. Two FP64 atomics per sample at random positions; with
// a sincospi and a phase product per sample instead of wmod the kernel took
// 33 us at 401 bins and 25 rows, now 8 us.
__global__ void __launch_bounds__(256) k_adjoint_scatter(const SigIter *__restrict__ its,
                                                         double2 *dx) {
  const SigIter &it = PdlEnterLoaded(its, 0);
  const int tt = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y, t = blockIdx.z;
  if (tt >= it.p) return;
  const int B = it.bins;
  const int ts = tt - it.p2;  // t in [-p2, p2]
  const ModN mod{uint32_t(it.n), it.n_inv};
  const int64_t u = mod(int64_t(it.q[t]) + RowOffset(r, B) + ts);
  const uint32_t j = mod(int64_t(it.a) * u + it.c);
  // t mod B: -p2 = (B + 1)/2 mod B since p is an odd multiple of B
  const uint32_t m = (uint32_t(tt) + uint32_t(B + 1) / 2) % uint32_t(B);
  const double2 h = it.ubuf[(size_t(t) * it.rows + r) * it.bins_cap + m];
  double2 w = it.wmod[ts < 0 ? -ts : ts];
  if (ts < 0) w.y = -w.y;
  const double2 v = cconj(cmul(h, w));
  atomicAdd(&dx[j].x, v.x);
  atomicAdd(&dx[j].y, v.y);
}

// Lanes per mode (k_estimate, k_adjoint_spread): a warp while the modes leave the
// SMs room (two for each of their schedulers), then fewer lanes, which share out
// less but repeat the setup less often. Calls of the estimate at 401 bins, n = 2^18,
// one trial, with 32, 8 and 1 lanes: 500 modes 65, 65, 78 us; 1500 modes 76, 65, 77;
// 6000 modes 93, 78, 78; 24000 modes 203, 116, 102; 100000 modes 644, 265, 197 us.
int LanesPerMode(int64_t m) { return m <= 1024 ? 32 : (m <= 8192 ? 8 : 1); }

// Blocks of one warp, 32 / lanes modes each, up to 2^20, striding beyond.
unsigned ModeBlocks(int64_t m, int lanes) {
  const int64_t b = (m * lanes + 31) / 32;
  return unsigned(b < (int64_t(1) << 20) ? b : (int64_t(1) << 20));
}

}  // namespace

void LaunchEstimate(const SigIter *d_it, const int32_t *k0, int64_t m,
                    double2 *coef, cudaStream_t s) {
  if (m <= 0) return;
  const int lanes = LanesPerMode(m);
  const unsigned blocks = ModeBlocks(m, lanes);
  if (lanes == 32) {
    Launch(k_estimate<32>, blocks, 32, 0, s, d_it, k0, m, coef);
  } else if (lanes == 8) {
    Launch(k_estimate<8>, blocks, 32, 0, s, d_it, k0, m, coef);
  } else {
    Launch(k_estimate<1>, blocks, 32, 0, s, d_it, k0, m, coef);
  }
}

void LaunchAdjointSpread(const SigIter *d_it, const int32_t *k0, const double2 *g,
                         int64_t m, cudaStream_t s) {
  if (m <= 0) return;
  const int lanes = LanesPerMode(m);
  const unsigned blocks = ModeBlocks(m, lanes);
  if (lanes == 32) {
    Launch(k_adjoint_spread<32>, blocks, 32, 0, s, d_it, k0, g, m);
  } else if (lanes == 8) {
    Launch(k_adjoint_spread<8>, blocks, 32, 0, s, d_it, k0, g, m);
  } else {
    Launch(k_adjoint_spread<1>, blocks, 32, 0, s, d_it, k0, g, m);
  }
}

void LaunchAdjointScatter(const SigIter *d_it, int p, int rows, int trials, double2 *dx,
                          cudaStream_t s) {
  dim3 grid((p + 255) / 256, rows, trials);
  Launch(k_adjoint_scatter, grid, 256, 0, s, d_it, dx);
}

}  // namespace mpsft
