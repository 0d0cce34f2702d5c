// Window tables, FFT twiddles and Bluestein chirp tables.
//
// Window (src/window.cc:28-75): wt(t) = w * sinc(pi t w) * exp(-2 (pi t sigma_f)^2)
// with w = 1/(2 bins); wt(0) = w. The window is even, so only |t| in
// [0, p2] is stored. Computed in FP64 and also rounded to FP32.
//
// Bluestein (chirp-z) form of the size-B DFT X[k] = sum_j y[j] e^{-2 pi i jk/B}:
//   X[k] = chirp[k] * sum_j (y[j] chirp[j]) * conj(chirp[k - j]),
//   chirp[j] = e^{-pi i j^2 / B} with j^2 reduced mod 2B exactly,
// a circular convolution of length M = 2^ceil(log2(2B - 1)) done with the
// shared-memory FFT; chat = FFT_M of the conjugate chirp sequence, stored in
// bit-reversed order.
#include "fft.cuh"
#include "launch.h"

namespace mpsft {

namespace {

__global__ void k_twiddles(float2 *tw32, double2 *tw64) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= kTwiddleEntries) return;
  TwiddleAt(e, tw32, tw64);
}

// sin(x)/x with the reference's Taylor guard (src/sincos.cc:69-88).
__device__ double SincPi(double x) {
  const double t0 = 2.220446049250313080847e-16;  // DBL_EPSILON
  const double t2 = 1.4901161193847656e-08;       // sqrt(t0)
  const double tn = 1.220703125e-04;              // sqrt(t2)
  if (x < 0) x = -x;
  if (x >= tn) return sin(x) / x;
  double r = 1.0;
  if (x >= t0) {
    const double x2 = x * x;
    r -= x2 / 6.0;
    if (x >= t2) r += (x2 * x2) / 120.0;
  }
  return r;
}

// FP64 window at t = i >= 0, in the reference's evaluation order.
__device__ double Window64At(const SigIter &it, int i) {
  if (i == 0) return it.width;
  const double t = double(i);
  const double u = __dmul_rn(__dmul_rn(t, M_PI), it.sigma_f);
  return __dmul_rn(__dmul_rn(it.width, SincPi(__dmul_rn(__dmul_rn(t, M_PI), it.width))),
                   exp(__dmul_rn(__dmul_rn(-2.0, u), u)));
}

// FP64 window (the reference's evaluation order) into wt64 and, when
// present, the float-float copy wtff; with_fp32 also rounds it into wt32.
__global__ void k_window64(const SigIter *__restrict__ its, int with_fp32) {
  PdlEnter(its, kTraceWindow64);
  const SigIter &it = its[blockIdx.y];
  if (!it.active || it.tables_valid) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > it.p2) return;
  const double v = Window64At(it, i);
  it.wt64[i] = v;
  if (with_fp32) it.wt32[i] = float(v);
  if (it.wtff != nullptr) {
    const float h = __double2float_rn(v);
    it.wtff[i] = make_float2(h, __double2float_rn(v - double(h)));
  }
}

// The same window evaluated in FP32 for the FP32 binning (a few ulp; the
// FP64 tables are built beside it, off the binning's critical path).
__global__ void k_window32(const SigIter *__restrict__ its) {
  PdlEnter(its, kTraceWindow32);
  const SigIter &it = its[blockIdx.y];
  if (!it.active || it.tables_valid || it.force_fp64) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > it.p2) return;
  const float w = float(it.width);
  float v = w;
  if (i > 0) {
    const float t = float(i);
    const float y = t * w;  // sinc argument in units of pi
    const float u = t * float(M_PI * it.sigma_f);
    v = w * (sinpif(y) / (float(M_PI) * y)) * expf(-2.f * u * u);
  }
  it.wt32[i] = v;
}

// e^{2 pi i m / n} of a residue m in [0, n), reduced to half a turn first.
__device__ double2 UnitRoot64(int64_t m, int64_t n) {
  if (2 * m > n) m -= n;
  double s, c;
  sincospi(2.0 * (double(m) / double(n)), &s, &c);
  return make_double2(c, s);
}

// The modulated window of the FP64 binning, wmod[t] = wt(t) e^{2 pi i (b t/n -
// t/(2B))} for t in [0, p2], and the row factors row_fac = e^{2 pi i (b (q +
// off) mod n)/n}: the binning's phase at t of row q + off is
// e^{2 pi i b off / n} times wmod's, so one table serves every row.
//
// With t = r + f B the phase is that of r times e^{2 pi i (b f B mod n)/n}
// (-1)^f: one FP64 sincospi per r (its angle one exact integer over 2nB) and
// one per f instead of one per t. FP64 evaluations are what bounds this kernel
// (a sincospi is about 50 operations, the window twice that, on pipes of two
// lanes per clock), so a block covers only 8 r's and one signal's bins spread
// over every SM (501 bins, 18537 window points evaluated: 18 us with 32 r's in
// 16 blocks, 12.5 us with 8); the last block has the row factors. eval: the
// window itself is evaluated here (and stored in wt64 when present) unless
// the signal's tables stand, else read from wt64.
constexpr int kModCols = 8, kModThreads = 128;
constexpr int kModFolds = kFoldLanes * kMaxFoldsPerLane / 2 + 1;  // f = t / B
static_assert(kModCols + kModFolds <= kModThreads, "a thread per phase");

__global__ void __launch_bounds__(kModThreads)
    k_window_mod(const SigIter *__restrict__ its, int eval, int cond) {
  const SigIter &it = PdlEnterLoaded<false>(its, blockIdx.y, kTraceWindow64);
  __shared__ double2 zr[kModCols], zf[kModFolds];
  if (!it.active) return;
  if (cond ? !RedoFP64(it) : it.force_fp64) return;
  const int B = it.bins;
  const int r0 = blockIdx.x * kModCols;
  const int64_t n = it.n;
  const ModN mod{uint32_t(n), it.n_inv};
  const int64_t b = mod(it.b);
  const int tid = threadIdx.x;
  if (blockIdx.x == gridDim.x - 1) {
    const int rows = it.rows;
    for (int i = tid; i < it.trials * rows; i += kModThreads) {
      const int t = i / rows, row = i - t * rows;
      int64_t off = 0;
      if (row > 0) {
        off = int64_t(B) << ((row - 1) >> 1);
        if ((row & 1) == 0) off = -off;
      }
      it.row_fac[i] = UnitRoot64(mod(b * mod(int64_t(it.q[t]) + off)), n);
    }
    return;
  }
  if (r0 >= B) return;
  const int nf = it.p2 / B + 1;
  if (tid < kModCols) {
    const int64_t r = r0 + tid;
    const int64_t nB = n * B;
    int64_t num = 2 * B * int64_t(mod(b * r)) - r * n;  // over 2 n B turns
    if (num > nB) num -= 2 * nB;
    double s, c;
    sincospi(double(num) / double(nB), &s, &c);
    zr[tid] = make_double2(c, s);
  } else if (tid < kModCols + nf) {
    const int f = tid - kModCols;
    const double2 z = UnitRoot64(mod(b * mod(int64_t(f) * B)), n);
    zf[f] = (f & 1) ? make_double2(-z.x, -z.y) : z;
  }
  __syncthreads();
  const int r = r0 + (tid & (kModCols - 1));
  if (r < B) {
    const double2 z = zr[tid & (kModCols - 1)];
    for (int f = tid / kModCols; f < nf; f += kModThreads / kModCols) {
      const int t = r + f * B;
      if (t > it.p2) break;
      double w;
      if (eval && !it.tables_valid) {
        w = Window64At(it, t);
        if (it.wt64 != nullptr) it.wt64[t] = w;
      } else {
        w = it.wt64[t];
      }
      it.wmod[t] = cscale(cmul(z, zf[f]), w);
    }
  }
}

// ph_lo[l] = e^{2 pi i l / n} for l < 2^ph_k and ph_hi[h] = e^{2 pi i h 2^ph_k / n}
// for h <= (n - 1) >> ph_k, from exact integer phases.
__global__ void k_phase_tables(const SigIter *__restrict__ its) {
  PdlEnter();
  const SigIter &it = its[blockIdx.y];
  if (!it.ph_build) return;  // (tables shared with another signal, or cached)
  const int64_t n = it.n;
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  double s, c;
  if (i < (int64_t(1) << it.ph_k)) {
    sincospi(2.0 * (double(i) / double(n)), &s, &c);
    it.ph_lo[i] = make_double2(c, s);
  }
  if (i <= ((n - 1) >> it.ph_k)) {
    sincospi(2.0 * (double(i << it.ph_k) / double(n)), &s, &c);
    it.ph_hi[i] = make_double2(c, s);
  }
}

__device__ inline float2 *ChirpOf(const SigIter &it, float2 *) { return it.chirp32; }
__device__ inline double2 *ChirpOf(const SigIter &it, double2 *) { return it.chirp64; }
__device__ inline float2 *ChatOf(const SigIter &it, float2 *) { return it.chat32; }
__device__ inline double2 *ChatOf(const SigIter &it, double2 *) { return it.chat64; }

// cond: only signals with more near-tie bins than their list holds (whose
// iteration is redone in FP64) take part.
template <typename V>
__global__ void __launch_bounds__(512)
    k_bluestein_setup(const SigIter *__restrict__ its, const V *__restrict__ tw,
                      int cond) {
  PdlEnter(its, kTraceBluestein);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *a = reinterpret_cast<V *>(smem_raw);
  const SigIter &it = its[blockIdx.x];
  if (!it.active) return;
  // (tables_valid: the FP64 tables of a signal forced to FP64 in every
  // iteration; of another signal redone in FP64, its FP32 tables)
  if (cond ? (!RedoFP64(it) || (it.force_fp64 && it.tables_valid))
           : (it.force_fp64 || it.tables_valid)) {
    return;
  }
  const int B = it.bins, M = it.fft_m;
  V *chirp = ChirpOf(it, (V *)nullptr);
  V *chat = ChatOf(it, (V *)nullptr);
  const int64_t twoB = 2 * int64_t(B);
  for (int j = threadIdx.x; j < M; j += blockDim.x) {
    a[Pad(j)] = vmake2(0.0, 0.0, (V *)nullptr);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < B; j += blockDim.x) {
    const int64_t j2 = (int64_t(j) * j) % twoB;
    double s, c;
    sincospi(-double(j2) / double(B), &s, &c);
    chirp[j] = vmake2(c, s, (V *)nullptr);
    const V cc = vmake2(c, -s, (V *)nullptr);  // conj(chirp[j])
    a[Pad(j)] = cc;
    if (j > 0) a[Pad(M - j)] = cc;
  }
  // FP32 tables: the bins-grid unit roots of the near-tie phase steps
  if (!cond && sizeof(V) == sizeof(float2) && it.r2b64 != nullptr) {
    for (int r = threadIdx.x; r < twoB; r += blockDim.x) {
      double s, c;
      sincospi(-double(r) / double(B), &s, &c);
      it.r2b64[r] = make_double2(c, s);
    }
  }
  __syncthreads();
  // chat in bit-reversed order (the row transforms' forward output order)
  BlockFFTDif(a, M, it.fft_log2m, tw, false, int(threadIdx.x), int(blockDim.x));
  for (int j = threadIdx.x; j < M; j += blockDim.x) chat[j] = a[Pad(j)];
}

}  // namespace

void LaunchTwiddles(float2 *tw32, double2 *tw64, cudaStream_t s) {
  const int n = kTwiddleEntries;
  k_twiddles<<<(n + 255) / 256, 256, 0, s>>>(tw32, tw64);
}

void LaunchPhaseTables(const SigIter *d_its, int nsig, int64_t entries,
                       cudaStream_t s) {
  dim3 grid(unsigned((entries + 255) / 256), nsig);
  Launch(k_phase_tables, grid, 256, 0, s, d_its);
}

void LaunchWindow(const SigIter *d_its, int nsig, int max_p2, cudaStream_t s) {
  dim3 grid((max_p2 + 1 + 255) / 256, nsig);
  Launch(k_window64, grid, 256, 0, s, d_its, 1);
}

void LaunchWindowMod(const SigIter *d_its, int nsig, int max_bins, WindowSource window,
                     bool cond, cudaStream_t s) {
  dim3 grid((max_bins + kModCols - 1) / kModCols + 1, nsig);
  Launch(k_window_mod, grid, kModThreads, 0, s, d_its, window == kWindowNew ? 1 : 0,
         cond ? 1 : 0);
}

void LaunchWindow64(const SigIter *d_its, int nsig, int max_p2, cudaStream_t s) {
  dim3 grid((max_p2 + 1 + 255) / 256, nsig);
  Launch(k_window64, grid, 256, 0, s, d_its, 0);
}

void LaunchWindow32(const SigIter *d_its, int nsig, int max_p2, cudaStream_t s) {
  dim3 grid((max_p2 + 1 + 255) / 256, nsig);
  Launch(k_window32, grid, 256, 0, s, d_its);
}

void LaunchBluesteinSetup(const SigIter *d_its, int nsig, int max_m, bool fp64,
                          const float2 *tw32, const double2 *tw64,
                          cudaStream_t s, bool cond) {
  if (fp64) {
    const size_t sm = size_t(PadLen(max_m)) * sizeof(double2);
    AllowSmem(k_bluestein_setup<double2>, size_t(PadLen(kMaxFFT64)) * sizeof(double2));
    Launch(k_bluestein_setup<double2>, nsig, 512, sm, s, d_its, tw64, cond ? 1 : 0);
  } else {
    const size_t sm = size_t(PadLen(max_m)) * sizeof(float2);
    AllowSmem(k_bluestein_setup<float2>, size_t(PadLen(kMaxFFT)) * sizeof(float2));
    Launch(k_bluestein_setup<float2>, nsig, 512, sm, s, d_its, tw32, cond ? 1 : 0);
  }
}

}  // namespace mpsft

namespace mpsft {

namespace {

// Estimate of mean |x|^2: kEnergyParts blocks per signal, block b taking
// kEnergyBatch of the kEnergyBlocks runs, thread t sample t of each, then the
// block's fixed tree; energy[sig * kEnergyStride + b] = the block's share of
// the mean. A signal shorter than kEnergyBlocks samples is summed whole by
// block 0.
// Bound by memory latency (512 KB in runs of 2 KB, each on a page of its own):
// a thread's kEnergyBatch loads are issued together. One block with a load per
// round trip took 139 us cold, one block of 8 batches 45 us, 6 us now.
constexpr int kEnergyBatch = kEnergyBlocks / kEnergyParts;
template <typename TX>
__global__ void __launch_bounds__(256)
    k_energy_sample(const void *const *__restrict__ xs, const int64_t *__restrict__ ns,
                    double *__restrict__ energy, int per_block) {
  PdlEnter();
  __shared__ double red[256];
  const int sig = blockIdx.y;
  const TX *x = reinterpret_cast<const TX *>(xs[sig]);
  const int64_t n = ns[sig];
  const int64_t run = min(int64_t(per_block), n / kEnergyBlocks);
  float acc = 0.f;
  if (run > 0) {
    const int r0 = blockIdx.x * kEnergyBatch;
    for (int64_t i = threadIdx.x; i < run; i += blockDim.x) {
      TX v[kEnergyBatch];
#pragma unroll
      for (int u = 0; u < kEnergyBatch; ++u) {
        v[u] = x[n * (r0 + u) / kEnergyBlocks + i];
      }
#pragma unroll
      for (int u = 0; u < kEnergyBatch; ++u) {
        const float re = float(v[u].x), im = float(v[u].y);
        acc = fmaf(re, re, fmaf(im, im, acc));
      }
    }
  } else if (blockIdx.x == 0) {
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
      const TX v = x[i];
      const float re = float(v.x), im = float(v.y);
      acc = fmaf(re, re, fmaf(im, im, acc));
    }
  }
  red[threadIdx.x] = double(acc);
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    energy[size_t(sig) * kEnergyStride + blockIdx.x] =
        red[0] / double(run > 0 ? run * kEnergyBlocks : n);
  }
}

}  // namespace

void LaunchEnergy(const void *const *x, const int64_t *n, int nsig, bool c128,
                  double *energy, cudaStream_t s, int per_block) {
  const dim3 grid(kEnergyParts, nsig);
  if (c128) {
    Launch(k_energy_sample<double2>, grid, 256, 0, s, x, n, energy, per_block);
  } else {
    Launch(k_energy_sample<float2>, grid, 256, 0, s, x, n, energy, per_block);
  }
}

bool WindowKernelsLaunchable() {
  int n1 = 0, n2 = 0;
  const size_t sm32 = size_t(PadLen(kMaxFFT)) * sizeof(float2);
  const size_t sm64 = size_t(PadLen(kMaxFFT64)) * sizeof(double2);
  AllowSmem(k_bluestein_setup<float2>, sm32);
  AllowSmem(k_bluestein_setup<double2>, sm64);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n1, k_bluestein_setup<float2>, 512, sm32);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n2, k_bluestein_setup<double2>, 512, sm64);
  return n1 > 0 && n2 > 0;
}

}  // namespace mpsft
