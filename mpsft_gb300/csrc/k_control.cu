// Device-side iteration control of the recovery loop (Demo1::Run,
// src/demo1.cc:36-59), so that a whole solve runs as one CUDA graph whose
// iteration body sits under a conditional while node.
//
// k_plan (before each iteration, one warp per signal) computes what the
// reference computes on the host at the start of Iterate: the number of bins
// B = max(2 (k - found) + 1, min_bins), NumBits, the window scalars
// (src/window.cc:28-51, with explicitly rounded FP64 operations so that they
// equal the host's values bit for bit), the thresholds 3 sigma / sqrt(B) and
// sigma / sqrt(B), and takes the iteration's transform and q's from the draw
// table the host filled from the signal's RNG in the reference's order
// (with each trial's row phase e^{2 pi i (b q mod n)/n}, computed there).
// k_finish (after the merge) applies the stop rule: count the iteration, a
// stale one when nothing was found, stop after max_stale_iter stale ones (never
// reset), on a status, or at max_iter; then it sets the while condition to
// "some signal still has work and draws".
//
// Fixed bins: once 2 (k - found) + 1 <= min_bins, every later iteration of a
// signal has bins = min_bins (found never decreases). When every signal of a
// batch is there, the next iteration can be planned ahead ("ahead" plan,
// into a second descriptor array) and its gather/fold run while the current
// iteration decides; k_finish then drops the planned iteration of a signal
// that stopped.
#include <algorithm>

#include "common.cuh"
#include "launch.h"

namespace mpsft {

thread_local bool g_launch_pdl = false;

namespace {

__device__ int32_t NumBitsDev(int32_t n, int32_t bins) {
  if (n < bins) return 1;
  int32_t out = 0;
  while (n >= bins) {
    n >>= 1;
    ++out;
  }
  return out;
}

__device__ inline int32_t NextBins(const SolveCtl &c, int32_t found) {
  const int32_t bins = (c.k - found) * 2 + 1;
  return bins < c.min_bins ? c.min_bins : bins;
}

// One warp per signal. A new number of bins takes eight FP64 divisions and a
// square root (about 700 cycles each on this part's FP64 pipes, whatever the
// number of lanes): the divisions run in three stages, the independent ones of a
// stage on different lanes, without 128-bit divisions (one thread after the
// other: one recovery of 1000 modes 1.008x, 24 uneven ones 1.005x slower).
// What is read through the descriptors (the number of modes, the draws, the
// table cache's entries) is read by all lanes at once before anything is stored,
// a draw per lane, so that the kernel waits for memory three times and not for
// every trial again. Lane 0 stores the rest. (With k_finish, which does the same:
// 6 us less of every iteration of 24 signals, 2 to 3 us of one signal's; a solve
// of one signal 1117 -> 1081 us, of 24 signals 5611 -> 5494 us, of 24 uneven ones
// 23.9 -> 23.4 ms.)
//
// max_bins: signals needing more bins wait (the launch shapes of this body
// do not cover them). ahead = 1 plans iteration iter + 1 of a signal in the
// fixed-bins state while iteration iter runs (bins = min_bins; the flags,
// which iteration iter still uses, are cleared by its k_finish instead).
__global__ void k_plan(SolveCtl *__restrict__ ctl, SigIter *__restrict__ its,
                       int nsig, int32_t max_bins, int ahead) {
  PdlEnter(its, kTracePlan);
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= nsig) return;
  const SolveCtl c = ctl[i];
  SigIter &it = its[i];
  const int local = c.iter + ahead - c.draw_base;
  if (c.done || local >= c.draws_avail) {
    if (lane == 0) it.active = 0;
    return;
  }
  // a, b, c, a_inv, q_0 .. (lanes 0 .. 3 + trials) and re, im of every trial's
  // row phase (lanes 0 .. 2 trials - 1)
  const int32_t dv = lane < 4 + c.trials
                         ? c.draws[size_t(local) * c.draw_stride + lane] : 0;
  const double bv = lane < 2 * c.trials
                        ? c.draw_bq[size_t(local) * (c.draw_stride - 4) * 2 + lane] : 0.0;
  const int32_t bins = ahead ? c.min_bins : NextBins(c, *it.tab_count);
  if (bins > max_bins) {
    if (lane == 0) it.active = 0;
    return;
  }
  const bool cached = c.win_base != nullptr && !c.force_fp64;
  const int h = bins >> 1;
  const int64_t win_base = cached ? c.win_base[h] : 0;
  const int32_t win_valid = cached ? c.win_valid[h] : 0;
  // Everything that depends on the bins only (and on the signal's constants)
  // stays from the previous iteration when the bins repeat (most late
  // iterations).
  const bool same_bins = it.bins == bins;
  const double B = double(bins), n = double(it.n), sigma = c.sigma;
  double width = 0, sigma_f = 0, xi_scale = 0, sigma_t = 0, bin_thr = 0, sv_thr = 0;
  double erf_d = 0, folds = 0, wf_scale = 0;
  if (!same_bins) {
    // Window scalars in the reference's operation order, no contraction.
    const double sq = c.sqrt_c_delta;
    const double rb = __dsqrt_rn(B);
    // each lane one quotient of the stage (0, 1 or the rest)
    auto div3 = [lane](double n0, double d0, double n1, double d1, double n2, double d2,
                       double *q0, double *q1, double *q2) {
      const double q = __ddiv_rn(lane == 0 ? n0 : (lane == 1 ? n1 : n2),
                                 lane == 0 ? d0 : (lane == 1 ? d1 : d2));
      *q0 = __shfl_sync(0xffffffffu, q, 0);
      *q1 = __shfl_sync(0xffffffffu, q, 1);
      *q2 = __shfl_sync(0xffffffffu, q, 2);
    };
    div3(1.0, __dmul_rn(2.0, B), 0.5,
         __dmul_rn(__dmul_rn(__dmul_rn(B, 2.0), M_SQRT2), sq), 1.0,
         __dmul_rn(__dmul_rn(2.0, n), B), &width, &sigma_f, &xi_scale);
    div3(1.0, __dmul_rn(2.0 * M_PI, sigma_f), __dmul_rn(3.0, sigma), rb, sigma, rb,
         &sigma_t, &bin_thr, &sv_thr);
    const double tmp =
        __dadd_rn(__dmul_rn(__dmul_rn(2.0 * M_SQRT2, sigma_t), sq), 1.0);
    erf_d = __dmul_rn(M_SQRT2 * M_PI, sigma_t);
    double unused;
    div3(tmp, B, erf_d, __dmul_rn(__dmul_rn(4.0, n), B), 0.0, 1.0, &folds, &wf_scale,
         &unused);
  }
  const int32_t b = __shfl_sync(0xffffffffu, dv, 1);
  const uint64_t phi_b = PhiOf(b, it.n);
  const int32_t cc = __shfl_sync(0xffffffffu, dv, 2);
  const int32_t a_inv = __shfl_sync(0xffffffffu, dv, 3);
  if (lane >= 4 && lane < 4 + c.trials) it.q[lane - 4] = dv;
  if (lane < 2 * c.trials) {
    (lane & 1 ? it.bq_im : it.bq_re)[lane >> 1] = bv;
  }
  if (lane != 0) return;
  if (ahead && it.fold_alt != nullptr) {
    // the planned iteration folds (and stashes its samples) into the
    // buffers this one's row transforms and re-binning do not read
    void *f = it.fold;
    it.fold = it.fold_alt;
    it.fold_alt = f;
    unsigned char *st = it.stash;
    it.stash = it.stash_alt;
    it.stash_alt = st;
  }
  if (!same_bins) {
    int32_t f = int32_t(ceil(folds));
    if (f % 2 == 0) ++f;
    const int32_t bits = NumBitsDev(it.n, bins);
    it.bins = bins;
    it.bits = bits;
    it.rows = 1 + 2 * bits;
    it.folds = f;
    it.p = f * bins;
    it.p2 = (it.p - 1) / 2;
    it.width = width;
    it.sigma_f = sigma_f;
    it.erf_d = erf_d;
    it.psi = PsiOf(bins);
    it.wf_scale = float(wf_scale);
    it.xi_scale = xi_scale;
    it.bin_thr = bin_thr;
    it.sv_thr = sv_thr;
    SetThresholdCopies(&it);
    int l = 0;
    while ((1 << l) < 2 * bins - 1) ++l;
    it.fft_log2m = l;
    it.fft_m = 1 << l;
    if (!c.fp64_path) {
      it.eps_rel = float(c.margin * 5.9604644775390625e-08);  // margin * 2^-24
      it.eps_ms = float(c.margin * double(kEpsRms) * 5.9604644775390625e-08 *
                        0.70710678118654752);  // / sqrt(2)
    } else {
      it.eps_rel = 0.f;
      it.eps_ms = 0.f;
    }
  }
  it.a = dv;
  it.b = b;
  it.c = cc;
  it.a_inv = a_inv;
  it.trials = c.trials;
  it.phi_b = phi_b;
  it.win_thr = c.win_thr;
  it.force_fp64 = c.force_fp64;
  it.win_slot = -1;
  if (cached) {
    // tables from the context's cache: built already, or built now by the
    // one signal of the batch that claims the block
    const WinBlock wb = WinBlockOf(it.p2, bins, it.fft_m);
    unsigned char *blk = c.win_pool + win_base;
    it.wt32 = reinterpret_cast<float *>(blk);
    it.wt64 = reinterpret_cast<double *>(blk + wb.wt64);
    it.wtff = reinterpret_cast<float2 *>(blk + wb.wtff);
    it.chirp32 = reinterpret_cast<float2 *>(blk + wb.chirp32);
    it.chat32 = reinterpret_cast<float2 *>(blk + wb.chat32);
    it.r2b64 = reinterpret_cast<double2 *>(blk + wb.r2b64);
    const bool build = win_valid == 0 && atomicCAS(&c.win_claim[h], 0, 1) == 0;
    it.tables_valid = build ? 0 : 1;
    if (build) it.win_slot = h;
  } else {
    // (a signal is forced to FP64 throughout a solve or never)
    it.tables_valid = c.last_bins == bins ? 1 : 0;
  }
  if (!ahead) {
    it.flags[0] = 0;
    it.flags[1] = 0;
    it.flags[2] = 0;
  }
  it.active = 1;
}

// The while condition: some signal has work (not stopped, draws left) and
// its next iteration's bins lie in (cond_lo, cond_hi] (and, with
// exclude_fixed, exceed its min_bins). its_ahead (or null): the iteration
// planned ahead (pipelined body).
__global__ void __launch_bounds__(1024)
    k_finish(SolveCtl *__restrict__ ctl, SigIter *__restrict__ its, int nsig,
             cudaGraphConditionalHandle handle, int set_condition,
             int32_t cond_lo, int32_t cond_hi, SigIter *__restrict__ its_ahead,
             int exclude_fixed) {
  PdlEnter(its, kTraceFinish);
  int any = 0;
  for (int i = threadIdx.x; i < nsig; i += blockDim.x) {
    // everything read before anything is stored: two waits for memory, not one
    // at every counter
    const SolveCtl c = ctl[i];
    const SigIter &it = its[i];
    int32_t *const fl = it.flags;
    int32_t found = *it.tab_count;
    const int32_t progress = fl[0], near_ties = fl[2], spills = fl[4];
    int32_t bits = fl[1], max_found = fl[3];
    const int32_t active = it.active, bins = it.bins, win_slot = it.win_slot;
    const bool forced = it.force_fp64 != 0, f64 = c.fp64_path || forced;
    const int64_t gathers = BinGathers(it, f64), bytes = BinBytesOf(it, f64);
    const int64_t tab_cap = it.tab_cap;
    int32_t iter = c.iter, done = c.done;
    if (active) {
      // this iteration's spilled candidates, after all others (InsertSpills)
      if (spills > 0) {
        InsertSpills(it);
        found = *it.tab_count;
        bits = fl[1];
        max_found = fl[3];
      }
      SolveCtl &o = ctl[i];
      iter += 1;
      int32_t stale = c.stale, status = c.status;
      if (bits & kStatusCapacity) {
        status = kSolveCapacity;
      } else if (bits & kStatusNonFinite) {
        status = kSolveNonFinite;
      } else if (int64_t(max_found) * 2 > tab_cap) {
        status = kSolveCapacity;
      }
      if (!progress) stale += 1;
      if (status == 0 && stale < c.max_stale && iter >= c.max_iter) {
        status = kSolveIterCap;
      }
      if (status != 0 || stale >= c.max_stale) done = 1;
      o.iter = iter;
      o.near_ties = c.near_ties + near_ties;
      if (bits & kStatusUnresolved) o.unresolved = c.unresolved + 1;
      o.fp64_iters = c.fp64_iters + forced;
      o.gathers = c.gathers + gathers;
      o.bin_bytes = c.bin_bytes + bytes;
      o.stale = stale;
      o.status = status;
      o.done = done;
      o.last_bins = bins;
      // the tables this signal built are complete (every table kernel of
      // the iteration has run)
      if (win_slot >= 0) c.win_valid[win_slot] = 1;
      its[i].active = 0;
    }
    if (its_ahead != nullptr) {
      if (done) its_ahead[i].active = 0;
      fl[0] = 0;
      fl[1] = 0;
      fl[2] = 0;
    }
    if (!done && iter - c.draw_base < c.draws_avail) {
      const int32_t nb = NextBins(c, found);
      if (nb > cond_lo && nb <= cond_hi && !(exclude_fixed && nb <= c.min_bins)) {
        any = 1;
      }
    }
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0 && set_condition) {
    cudaGraphSetConditional(handle, any ? 1u : 0u);
  }
}

// Holds the stream for `ns` nanoseconds of the global timer (one thread;
// the wait always ends): in profiling runs, the host enqueues the timed
// binning launch and its events meanwhile, so that no host launch gap falls
// between the events.
__global__ void k_delay(unsigned long long ns) {
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  do {
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  } while (t - t0 < ns);
}

// dst[0..bytes) = src[0..bytes) with src in device-mapped pinned host memory, in
// words (CopySplit), the remainder bytewise.
__global__ void __launch_bounds__(256)
    k_copy_mapped(const unsigned char *__restrict__ src, unsigned char *__restrict__ dst,
                  size_t bytes) {
  PdlEnter();
  const size_t stride = size_t(gridDim.x) * blockDim.x;
  const size_t t0 = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const CopyWords cw =
      CopySplit(reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst), bytes);
  if (cw.width == 16) {
    const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
    uint4 *d4 = reinterpret_cast<uint4 *>(dst);
    for (size_t i = t0; i < cw.words; i += stride) d4[i] = s4[i];
  } else if (cw.width == 4) {
    const uint32_t *s1 = reinterpret_cast<const uint32_t *>(src);
    uint32_t *d1 = reinterpret_cast<uint32_t *>(dst);
    for (size_t i = t0; i < cw.words; i += stride) d1[i] = s1[i];
  }
  for (size_t i = cw.words * cw.width + t0; i < bytes; i += stride) dst[i] = src[i];
}

}  // namespace

void LaunchCopyMapped(const void *src_dev, void *dst, size_t bytes, cudaStream_t s) {
  if (bytes == 0) return;
  const size_t words = bytes / 16 + 1;
  const unsigned blocks = unsigned(std::min<size_t>(152, (words + 255) / 256));
  Launch(k_copy_mapped, blocks, 256, 0, s, static_cast<const unsigned char *>(src_dev),
                                       static_cast<unsigned char *>(dst), bytes);
}

void LaunchDelay(unsigned long long ns, cudaStream_t s) {
  k_delay<<<1, 1, 0, s>>>(ns);
}

void LaunchPlan(SolveCtl *ctl, SigIter *its, int nsig, int32_t max_bins,
                cudaStream_t s, bool ahead) {
  // a warp per signal and block: its FP64 operations get a scheduler
  Launch(k_plan, nsig, 32, 0, s, ctl, its, nsig, max_bins, ahead ? 1 : 0);
}

void LaunchFinish(SolveCtl *ctl, SigIter *its, int nsig,
                  cudaGraphConditionalHandle handle, bool set_condition,
                  int32_t cond_lo, int32_t cond_hi, cudaStream_t s,
                  SigIter *its_ahead, bool exclude_fixed) {
  Launch(k_finish, 1, 1024, 0, s, ctl, its, nsig, handle, set_condition ? 1 : 0,
                              cond_lo, cond_hi, its_ahead, exclude_fixed ? 1 : 0);
}

bool ControlKernelsLaunchable() {
  int a = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_finish, 1024, 0);
  return a > 0;
}

}  // namespace mpsft
