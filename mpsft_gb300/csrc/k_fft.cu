// Size-B forward DFT of every folded row (FFTPlan::Run of size B,
// src/base.cc:86-97, called at src/binner.cc:428 and 509-510), by Bluestein's
// chirp-z method over the shared-memory radix-2 FFT (any odd B, including
// large primes), followed by the row factor that the fold left out,
// e^{2 pi i (b q mod n)/n} (FP32) or e^{2 pi i (b (q + off) mod n)/n} (FP64).
// Output: complex128 bins in ubuf.
//
// One CTA per (row, trial, signal). FP32 path: the convolution runs in FP32
// (M <= 16384 points, 128 KB of shared memory); FP64 path: in FP64
// (M <= 8192). In solves and iterations the FP32 path writes complex64 bins
// (ubuf32) and keeps the FP64 pipes out of the epilogue (GB300 issues FP64
// at a small fraction of its FP32 rate, with long latencies): the row factor
// is applied as a float-float value, and each product is formed with exact
// FMA products and a two-sum, then rounded once to FP32.
#include <cooperative_groups.h>

#include <algorithm>

#include "fft.cuh"
#include "launch.h"

namespace mpsft {

namespace {

__device__ inline const float2 *ChirpOf(const SigIter &it, float2 *) { return it.chirp32; }
__device__ inline const double2 *ChirpOf(const SigIter &it, double2 *) { return it.chirp64; }
__device__ inline const float2 *ChatOf(const SigIter &it, float2 *) { return it.chat32; }
__device__ inline const double2 *ChatOf(const SigIter &it, double2 *) { return it.chat64; }

// y * (bh + bl) rounded to FP32 (bh + bl: a unit phase as float-float):
// the high products exactly (FMA residuals), a two-sum of the pair, then the
// residuals and the low-word products, one final rounding.
__device__ __forceinline__ float DotRound(float x0, float y0, float x1, float y1,
                                          float l0, float l1) {
  // x0 y0 + x1 y1 + (x0 l0 + x1 l1)
  const float p0 = __fmul_rn(x0, y0), e0 = fmaf(x0, y0, -p0);
  const float p1 = __fmul_rn(x1, y1), e1 = fmaf(x1, y1, -p1);
  const float s = __fadd_rn(p0, p1);
  const float bb = __fsub_rn(s, p0);
  const float es = __fadd_rn(__fsub_rn(p0, __fsub_rn(s, bb)), __fsub_rn(p1, bb));
  const float lo = __fadd_rn(__fadd_rn(es, __fadd_rn(e0, e1)),
                             fmaf(x0, l0, __fmul_rn(x1, l1)));
  return __fadd_rn(s, lo);
}
__device__ __forceinline__ float2 MulPhaseFF(float2 y, float2 bh, float2 bl) {
  return make_float2(DotRound(y.x, bh.x, -y.y, bh.y, bl.x, bl.y),
                     DotRound(y.x, bh.y, y.y, bh.x, bl.y, bl.x));
}

// cond: only signals whose iteration is redone in FP64 take part. The FP32
// transform also records the mean |U|^2 and the largest |U| of each row (for the
// near-tie bound; an FP64 square root per output and what goes with it were a
// seventh of the FP64 transform's operations).
//
// Rows per block: small transforms share a block, RowsPerBlock(M) rows side by
// side (M/8 threads each for the radix-8 passes), so that late iterations
// with few bins do not launch a block per tiny row.
constexpr int kRowFftThreads = 512;
constexpr int kRowsMax = 64;
__device__ __forceinline__ int RowsPerBlock(int M) {
  const int r = kRowFftThreads * 8 / M;
  return r < 1 ? 1 : (r > kRowsMax ? kRowsMax : r);
}

// FP64 operations bound the FP64 transform (fft.cuh, BlockConv): at 501 bins
// (M = 1024) and one row per SM 40 us (cold) with whole radix-2 stages, 37 us
// now; at 101 bins (M = 256) 27 and 18 us.
template <typename V>
__global__ void __launch_bounds__(kRowFftThreads)
    k_row_fft(const SigIter *__restrict__ its, int max_trials,
              const V *__restrict__ tw, int cond, int rpb_cap) {
  const SigIter &it = PdlEnterLoaded(its, blockIdx.z, kTraceRowFft);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned row_max_bits[kRowsMax];
  if (!it.active) return;
  if (cond ? !RedoFP64(it) : it.force_fp64) return;
  const int tr = blockIdx.y;
  const int B = it.bins, M = it.fft_m;
  const int rpb = min(RowsPerBlock(M), rpb_cap);
  const int row0 = blockIdx.x * rpb;
  if (row0 >= it.rows || tr >= it.trials) return;
  const int nth = kRowFftThreads / rpb;  // threads per row
  const int lr = threadIdx.x / nth, tid = threadIdx.x % nth;
  const int row = row0 + lr;
  const bool live = lr < rpb && row < it.rows;
  V *a = reinterpret_cast<V *>(smem_raw) + size_t(lr) * PadLen(M);
  const V *__restrict__ chirp = ChirpOf(it, (V *)nullptr);
  const V *__restrict__ chat = ChatOf(it, (V *)nullptr);
  if (threadIdx.x < kRowsMax) row_max_bits[threadIdx.x] = 0u;
  // the trial's row factor as float-float for the complex64 epilogue (read
  // after the transforms' barriers)
  __shared__ float2 bq_ff[2];
  const bool out32 = sizeof(V) == sizeof(float2) && it.ubuf32 != nullptr;
  if (out32 && threadIdx.x == 0) {
    const double br = it.bq_re[tr], bi = it.bq_im[tr];
    const float hr = __double2float_rn(br), hi = __double2float_rn(bi);
    bq_ff[0] = make_float2(hr, hi);
    bq_ff[1] = make_float2(__double2float_rn(br - double(hr)),
                           __double2float_rn(bi - double(hi)));
  }
  const int L = it.fft_log2m, half = M / 2;
  if constexpr (sizeof(V) == sizeof(double2)) {
    // element loops: up to 4 elements per thread with their loads issued
    // together; the first forward stage (span M/2, its upper inputs zero since
    // B <= M/2) is part of the fill
    if (live) {
      const V *__restrict__ src = reinterpret_cast<const V *>(it.fold) +
                                  (size_t(tr) * it.rows + row) * it.bins_cap;
      if (half == 0 && tid == 0) a[0] = vmul(src[0], __ldg(&chirp[0]));
      for (int j0 = tid; j0 < half; j0 += 4 * nth) {
        V v[4], w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + u * nth;
          v[u] = vmake2(0.0, 0.0, (V *)nullptr);
          if (j < B) {
            v[u] = vmul(src[j], __ldg(&chirp[j]));
            w[u] = Twiddle(tw, L, j, false);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + u * nth;
          if (j < half) {
            a[Pad(j)] = v[u];
            a[Pad(j + half)] = j < B ? vmul(v[u], w[u]) : v[u];
          }
        }
      }
    }
    __syncthreads();
    // forward DIF (bit-reversed out), product with chat (stored bit-reversed),
    // inverse DIT (natural out) but for its last stage; rows past the last run
    // the barriers only
    BlockConv(a, live ? M : 0, L > 0 ? L - 1 : 0, StagesPerPass(rpb * M), chat, tw, tid,
              nth);
  } else {
    // element loops: up to 8 elements per thread with their loads issued
    // together (a thread covers M / nth elements)
    if (live) {
      const V *__restrict__ src = reinterpret_cast<const V *>(it.fold) +
                                  (size_t(tr) * it.rows + row) * it.bins_cap;
      for (int j0 = tid; j0 < M; j0 += 8 * nth) {
        V v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int j = j0 + u * nth;
          if (j < M) {
            v[u] = j < B ? vmul(src[j], __ldg(&chirp[j]))
                         : vmake2(0.0, 0.0, (V *)nullptr);
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int j = j0 + u * nth;
          if (j < M) a[Pad(j)] = v[u];
        }
      }
    }
    __syncthreads();
    // forward DIF (bit-reversed out), product with chat (stored bit-reversed),
    // inverse DIT (natural out); rows past the last run the barriers only
    BlockFFTDif(a, live ? M : 0, it.fft_log2m, tw, false, tid, nth);
    if (live) {
      for (int j0 = tid; j0 < M; j0 += 8 * nth) {
        V w[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int j = j0 + u * nth;
          if (j < M) w[u] = __ldg(&chat[j]);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int j = j0 + u * nth;
          if (j < M) a[Pad(j)] = vmul(a[Pad(j)], w[u]);
        }
      }
    }
    __syncthreads();
    BlockFFTDit(a, live ? M : 0, it.fft_log2m, tw, true, tid, nth);
  }
  // output k of the inverse transform (FP64: the lower half of its last stage)
  auto conv_out = [&](int k) -> V {
    if (sizeof(V) == sizeof(float2) || half == 0) return a[Pad(k)];
    return vadd(a[Pad(k)], vmul(a[Pad(k + half)], Twiddle(tw, L, k, true)));
  };
  float ss = 0.f;  // this thread's share of the row's sum of |U|^2
  float mx = 0.f;  // and of its largest |U|
  if (live && out32) {
    // FP32 bins: exact power-of-two scale, float-float row factor
    const float inv_mf = 1.0f / float(M);
    const float2 bh = bq_ff[0], bl = bq_ff[1];
    float2 *dst = it.ubuf32 + (size_t(tr) * it.rows + row) * it.bins_cap;
    for (int k0 = tid; k0 < B; k0 += 8 * nth) {
      V w[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int k = k0 + u * nth;
        if (k < B) w[u] = __ldg(&chirp[k]);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int k = k0 + u * nth;
        if (k < B) {
          const V z = vmul(a[Pad(k)], w[u]);
          const float2 y = make_float2(float(z.x) * inv_mf, float(z.y) * inv_mf);
          dst[k] = MulPhaseFF(y, bh, bl);
          const float y2 = y.x * y.x + y.y * y.y;
          ss += y2;
          mx = fmaxf(mx, sqrtf(y2));
        }
      }
    }
  } else if (live) {
    // FP64 (row factor, power-of-two scale and all in FP64 operations, the
    // fewest: no magnitudes, which only the FP32 near-tie bound reads), or FP32
    // bins widened
    const double inv_m = 1.0 / double(M);
    const double2 f = sizeof(V) == sizeof(double2)
                          ? it.row_fac[tr * it.rows + row]
                          : make_double2(it.bq_re[tr], it.bq_im[tr]);
    const double2 bq = cscale(f, inv_m);
    double2 *dst = it.ubuf + (size_t(tr) * it.rows + row) * it.bins_cap;
    for (int k0 = tid; k0 < B; k0 += 8 * nth) {
      V w[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int k = k0 + u * nth;
        if (k < B) w[u] = __ldg(&chirp[k]);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int k = k0 + u * nth;
        if (k < B) {
          if constexpr (sizeof(V) == sizeof(double2)) {
            dst[k] = vmul(bq, vmul(conv_out(k), w[u]));
          } else {
            const double2 y = cscale(to_d2(vmul(conv_out(k), w[u])), inv_m);
            dst[k] = vmul(f, y);
            const double y2 = y.x * y.x + y.y * y.y;
            ss += float(y2);
            mx = fmaxf(mx, float(sqrt(y2)));
          }
        }
      }
    }
  }
  if constexpr (sizeof(V) == sizeof(float2)) {
    // the row's sum of |U|^2 in a fixed order: a shuffle tree over segments of
    // min(nth, 32) threads (a row's threads are consecutive, nth a power of
    // two), then the row's segments in order
    __shared__ float seg_ss[kRowFftThreads / 8];
    const int seg = nth < 32 ? nth : 32;
    for (int o = seg >> 1; o > 0; o >>= 1) {
      ss += __shfl_xor_sync(0xffffffffu, ss, o);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & (seg - 1)) == 0) {
      seg_ss[threadIdx.x / seg] = ss;
      // non-negative floats order like their bit patterns
      if (live) atomicMax(&row_max_bits[lr], __float_as_uint(mx));
    }
    __syncthreads();  // (rows past the last only reach the barriers)
    if (live && tid == 0 && it.row_max != nullptr) {
      it.row_max[tr * it.rows + row] = __uint_as_float(row_max_bits[lr]);
      const int nseg = nth / seg;
      float t = 0.f;
      for (int j = 0; j < nseg; ++j) t += seg_ss[lr * nseg + j];
      it.row_ms[tr * it.rows + row] = t / float(B);
    }
  }
}

// The row transform with one row over a cluster of C blocks, for launches of
// few rows (one signal's call), which a block per row leaves on a few SMs:
// there the FP64 transform is bound by those SMs' FP64 pipes and the FP32 one
// by the latency of its passes over a long row. Block c holds the c-th of C
// slices of the bit-reversed array, Ms = M / C elements. The first log2 C
// forward stages need no exchange: every block reads the row's samples and
// evaluates its own outputs of them (the upper half of the input is zero). The
// stages within a slice run as in k_row_fft; the last log2 C inverse stages read
// the C slices' element k through distributed shared memory, each block a C-th
// of the k, and only the outputs below M/2. A transform too small to split
// (M < kSplitMin C) runs whole on block 0.
// Cold, FP64, 31 rows of 501 bins (M = 1024): 37 us with a block per row, 21 us
// with 4; FP32, 29 rows of 8001 bins (M = 16384): 87 us and 33 us
// with 8 (31 rows of 501 bins: 15.5 and 13 us).
constexpr int kSplitThreads = 256;
constexpr int kSplitMin = 64;  // elements per slice at least

// Output j of the row's transform times the row factor: FP64 bins (f scaled by
// 1 / M), FP32 bins widened, or (solves and iterations) complex64 bins.
__device__ __forceinline__ void StoreBin(const SigIter &it, int tr, int row, int j, double2 y,
                                         float2, float2, double2 f) {
  it.ubuf[(size_t(tr) * it.rows + row) * it.bins_cap + j] = vmul(f, y);
}
__device__ __forceinline__ void StoreBin(const SigIter &it, int tr, int row, int j, float2 y,
                                         float2 bh, float2 bl, double2 f) {
  const size_t o = (size_t(tr) * it.rows + row) * it.bins_cap + j;
  if (it.ubuf32 != nullptr) {
    it.ubuf32[o] = MulPhaseFF(y, bh, bl);
  } else {
    it.ubuf[o] = cmul(f, make_double2(y.x, y.y));
  }
}

// One row of one block of the cluster: fill, local stages, exchange, epilogue;
// FP32 adds this thread's share to the sum and the maximum of |U|^2.
template <typename V, int C>
__device__ __forceinline__ void SplitRow(const SigIter &it, int tr, int row, int c,
                                         cooperative_groups::cluster_group cl, V *a,
                                         const V *__restrict__ tw, bool work, float *ss,
                                         float *mx) {
  constexpr int kLog = C == 8 ? 3 : (C == 4 ? 2 : (C == 2 ? 1 : 0));
  constexpr int H = C > 1 ? C / 2 : 1;  // slices of the lower half
  constexpr bool kF64 = sizeof(V) == sizeof(double2);
  const int B = it.bins, L = it.fft_log2m, M = it.fft_m, Ms = M / C;
  const int tid = threadIdx.x, lg = L - kLog;
  const V *__restrict__ chirp = ChirpOf(it, (V *)nullptr);
  if (work) {
    const V *__restrict__ src = reinterpret_cast<const V *>(it.fold) +
                                (size_t(tr) * it.rows + row) * it.bins_cap;
    for (int k = tid; k < Ms; k += kSplitThreads) {
      V v[H];
#pragma unroll
      for (int m = 0; m < H; ++m) {
        const int j = k + m * Ms;
        v[m] = vmake2(0.0, 0.0, (V *)nullptr);
        if (j < B) {
          v[m] = vmul(src[j], __ldg(&chirp[j]));
          if (C > 1 && (c & (C / 2))) v[m] = vmul(v[m], Twiddle(tw, L, j, false));
        }
      }
#pragma unroll
      for (int st = 1; st < kLog; ++st) {
        const int cnt = C >> (st + 1);
#pragma unroll
        for (int m = 0; m < H; ++m) {
          if (m < cnt) {
            if (c & cnt) {
              v[m] = vmul(vsub(v[m], v[m + cnt]), Twiddle(tw, L - st, k + m * Ms, false));
            } else {
              v[m] = vadd(v[m], v[m + cnt]);
            }
          }
        }
      }
      a[Pad(k)] = v[0];
    }
  }
  __syncthreads();
  // stages per pass: FP64 by its schedulers (StagesPerPass), FP32 three (fewer
  // barriers) unless that leaves less than two warps
  BlockConv(a, work ? Ms : 0, lg, kF64 ? StagesPerPass(Ms) : (Ms >= 512 ? 3 : 2),
            ChatOf(it, (V *)nullptr) + size_t(c) * Ms, tw, tid, kSplitThreads);
  cl.sync();  // every slice is done
  if (work) {
    const double2 f = kF64 ? cscale(it.row_fac[tr * it.rows + row], 1.0 / double(M))
                           : make_double2(it.bq_re[tr], it.bq_im[tr]);
    const float2 bh = make_float2(__double2float_rn(f.x), __double2float_rn(f.y));
    const float2 bl = make_float2(__double2float_rn(f.x - double(bh.x)),
                                  __double2float_rn(f.y - double(bh.y)));
    const float inv_m = 1.f / float(M);
    const V *part[C];
#pragma unroll
    for (int i = 0; i < C; ++i) part[i] = C > 1 ? cl.map_shared_rank(a, i) : a;
    const int k1 = (c + 1) * (Ms / C);
    for (int k = c * (Ms / C) + tid; k < k1; k += kSplitThreads) {
      V x[C];
#pragma unroll
      for (int i = 0; i < C; ++i) x[i] = part[i][Pad(k)];
#pragma unroll
      for (int s = 0; s < kLog; ++s) {
#pragma unroll
        for (int i = 0; i < C; ++i) {
          if ((i & (1 << s)) == 0) {
            const int e = k + (i & ((1 << s) - 1)) * Ms;
            const V v = vmul(x[i + (1 << s)], Twiddle(tw, lg + s + 1, e, true));
            const V u = x[i];
            x[i] = vadd(u, v);
            if (s + 1 < kLog) x[i + (1 << s)] = vsub(u, v);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const int j = k + i * Ms;
        if (j < B) {
          V y = vmul(x[i], __ldg(&chirp[j]));
          if constexpr (kF64) {
            StoreBin(it, tr, row, j, y, bh, bl, f);
          } else {
            y.x *= inv_m;  // (a power of two: exact)
            y.y *= inv_m;
            StoreBin(it, tr, row, j, y, bh, bl, f);
            const float y2 = y.x * y.x + y.y * y.y;
            *ss += y2;
            *mx = fmaxf(*mx, sqrtf(y2));
          }
        }
      }
    }
  }
}

template <typename V, int C>
__global__ void __launch_bounds__(kSplitThreads)
    k_row_fft_split(const SigIter *__restrict__ its, const V *__restrict__ tw, int cond) {
  const SigIter &it = PdlEnterLoaded(its, blockIdx.z, kTraceRowFft);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float part_ss[C], part_mx[C];  // block 0's: every block's share
  __shared__ float warp_ss[kSplitThreads / 32], warp_mx[kSplitThreads / 32];
  const int row = blockIdx.x / C, tr = blockIdx.y;
  // (the same for every block of a cluster)
  if (!it.active || tr >= it.trials || row >= it.rows) return;
  if (cond ? !RedoFP64(it) : it.force_fp64) return;
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int c = int(cl.block_rank());
  V *a = reinterpret_cast<V *>(smem_raw);
  float ss = 0.f, mx = 0.f;
  if (it.fft_m >= kSplitMin * C) {
    SplitRow<V, C>(it, tr, row, c, cl, a, tw, true, &ss, &mx);
  } else {
    SplitRow<V, 1>(it, tr, row, 0, cl, a, tw, c == 0, &ss, &mx);
  }
  if constexpr (sizeof(V) == sizeof(double2)) {
    cl.sync();  // no block reads another's slice any more
  } else {
    // the row's largest magnitude and sum of |U|^2 in a fixed order: a shuffle
    // tree, the warps in order, the blocks in order
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ss += __shfl_xor_sync(0xffffffffu, ss, o);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
      warp_ss[threadIdx.x >> 5] = ss;
      warp_mx[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kSplitThreads / 32; ++w) {
        ss += warp_ss[w];
        mx = fmaxf(mx, warp_mx[w]);
      }
      *cl.map_shared_rank(&part_ss[c], 0) = ss;
      *cl.map_shared_rank(&part_mx[c], 0) = mx;
    }
    cl.sync();  // the shares are in block 0, and no block reads another's slice any more
    if (c == 0 && threadIdx.x == 0 && it.row_max != nullptr) {
      for (int i = 1; i < C; ++i) {
        ss += part_ss[i];
        mx = fmaxf(mx, part_mx[i]);
      }
      it.row_max[tr * it.rows + row] = mx;
      it.row_ms[tr * it.rows + row] = ss / float(it.bins);
    }
  }
}

// Small bins (Bluestein size M <= kDirectMaxM, bins <= 63): the DFT as a
// direct sum X[k] = sum_j F[j] e^{-2 pi i j k / B}, two warps per row and one
// output per lane, with the unit roots of the bins grid in shared memory;
// then the same epilogue as the Bluestein kernel. Each sum runs as four
// interleaved FMA chains over j = u mod 4 (each with its own root index
// j k mod B), added pairwise at the end: a short dependency chain per term,
// and an FP32 error below that of the Bluestein transform it replaces (two
// 128-point transforms at B = 51).
// Its latency is what counts: the values' loads go out before the roots are
// evaluated, the row factor's FP64 conversions run beside the sums, and four steps
// of the chains are unrolled (51 bins, 2^16 samples: a call 36.3 -> 36.0 us).
constexpr int kDirectMaxM = 128;
constexpr int kDirectMaxBins = kDirectMaxM / 2;
constexpr int kDirectRowsPerBlock = 4;  // two warps per row

__global__ void __launch_bounds__(64 * kDirectRowsPerBlock)
    k_row_dft_small(const SigIter *__restrict__ its, int cond) {
  const SigIter &it = PdlEnterLoaded(its, blockIdx.z, kTraceRowFft);
  __shared__ float2 roots[kDirectMaxBins];
  __shared__ float2 rows[kDirectRowsPerBlock][kDirectMaxBins];
  __shared__ float wmax[2 * kDirectRowsPerBlock];
  __shared__ float wss[2 * kDirectRowsPerBlock];
  if (!it.active) return;
  if (cond ? !RedoFP64(it) : it.force_fp64) return;
  const int tr = blockIdx.y;
  const int B = it.bins;
  if (tr >= it.trials) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lr = warp >> 1;
  const int row = blockIdx.x * kDirectRowsPerBlock + lr;
  const bool live = row < it.rows;
  // (B <= 64: a value and a root per thread of the row, the value's load first)
  const int j0 = (warp & 1) * 32 + lane;
  float2 v0 = make_float2(0.f, 0.f);
  if (live && j0 < B) {
    v0 = (reinterpret_cast<const float2 *>(it.fold) +
          (size_t(tr) * it.rows + row) * it.bins_cap)[j0];
  }
  if (threadIdx.x < B) {
    float sn, cs;
    sincospif(-2.0f * float(int(threadIdx.x)) / float(B), &sn, &cs);
    roots[threadIdx.x] = make_float2(cs, sn);
  }
  if (live && j0 < B) rows[lr][j0] = v0;
  __syncthreads();
  const int k = (warp & 1) * 32 + lane;
  float mx = 0.f, ss = 0.f;
  if (live && k < B) {
    const float2 *f = rows[lr];
    float xr[4] = {0.f, 0.f, 0.f, 0.f}, xi[4] = {0.f, 0.f, 0.f, 0.f};
    int id[4];
    id[0] = 0;
    id[1] = k;
    id[2] = (2 * k) % B;
    id[3] = (3 * k) % B;
    const int step = (4 * k) % B;
    // (the row factor's FP64 conversions run beside the sum)
    const double br = it.bq_re[tr], bi = it.bq_im[tr];
    const float2 bh = make_float2(__double2float_rn(br), __double2float_rn(bi));
    const float2 bl = make_float2(__double2float_rn(br - double(bh.x)),
                                  __double2float_rn(bi - double(bh.y)));
    int j = 0;
#pragma unroll 4
    for (; j + 4 <= B; j += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 v = f[j + u], w = roots[id[u]];
        xr[u] = fmaf(v.x, w.x, xr[u]);
        xr[u] = fmaf(-v.y, w.y, xr[u]);
        xi[u] = fmaf(v.x, w.y, xi[u]);
        xi[u] = fmaf(v.y, w.x, xi[u]);
        id[u] += step;
        if (id[u] >= B) id[u] -= B;
      }
    }
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      if (j + u < B) {
        const float2 v = f[j + u], w = roots[id[u]];
        xr[u] = fmaf(v.x, w.x, xr[u]);
        xr[u] = fmaf(-v.y, w.y, xr[u]);
        xi[u] = fmaf(v.x, w.y, xi[u]);
        xi[u] = fmaf(v.y, w.x, xi[u]);
      }
    }
    const float2 y = make_float2((xr[0] + xr[1]) + (xr[2] + xr[3]),
                                 (xi[0] + xi[1]) + (xi[2] + xi[3]));
    const size_t o = (size_t(tr) * it.rows + row) * it.bins_cap + k;
    if (it.ubuf32 != nullptr) {
      it.ubuf32[o] = MulPhaseFF(y, bh, bl);
    } else {
      const double2 bq = make_double2(br, bi);
      it.ubuf[o] = cmul(bq, make_double2(y.x, y.y));
    }
    ss = y.x * y.x + y.y * y.y;
    mx = sqrtf(ss);
  }
  // the row's largest magnitude and mean |U|^2: each warp's (a fixed shuffle
  // tree), then the row's pair of warps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
  }
  if (lane == 0) {
    wmax[warp] = mx;
    wss[warp] = ss;
  }
  __syncthreads();
  if (live && (warp & 1) == 0 && lane == 0 && it.row_max != nullptr) {
    it.row_max[tr * it.rows + row] = fmaxf(wmax[warp], wmax[warp + 1]);
    it.row_ms[tr * it.rows + row] = (wss[warp] + wss[warp + 1]) / float(B);
  }
}

}  // namespace

// Shared memory of a block: one padded row of the largest transform, or the
// rows of smaller ones side by side (at most 4096 + 256 + 64 slots).
inline size_t RowFftSlots(int max_m) {
  const size_t one = size_t(PadLen(max_m));
  const size_t packed = size_t(kRowFftThreads) * 8 + kRowFftThreads / 2 + kRowsMax;
  return one > packed ? one : packed;
}

// Shared memory of a split row's block: a slice of the largest transform, or
// a whole one too small to split.
inline size_t SplitSlots(int max_m, int c) {
  return size_t(PadLen(std::max(max_m / c, kSplitMin * c)));
}

template <typename V, int C>
void LaunchRowSplit(const SigIter *d_its, dim3 grid, int max_m, const V *tw, cudaStream_t s,
                    bool cond) {
  const size_t sm = SplitSlots(max_m, C) * sizeof(V);
  constexpr int kMost = sizeof(V) == sizeof(double2) ? kMaxFFT64 : kMaxFFT;
  AllowSmem(k_row_fft_split<V, C>, SplitSlots(kMost, C) * sizeof(V));
  grid.x *= C;
  LaunchCluster(k_row_fft_split<V, C>, grid, kSplitThreads, sm, s, C, d_its, tw,
                cond ? 1 : 0);
}

// Rows over clusters of c blocks; false for c = 1.
template <typename V>
bool LaunchRowSplits(const SigIter *d_its, dim3 grid, int c, int max_m, const V *tw,
                     cudaStream_t s, bool cond) {
  if (c == 8) {
    LaunchRowSplit<V, 8>(d_its, grid, max_m, tw, s, cond);
  } else if (c == 4) {
    LaunchRowSplit<V, 4>(d_its, grid, max_m, tw, s, cond);
  } else if (c == 2) {
    LaunchRowSplit<V, 2>(d_its, grid, max_m, tw, s, cond);
  } else {
    return false;
  }
  return true;
}

void LaunchRowFFT(const SigIter *d_its, int nsig, int max_rows,
                  int max_trials, int max_m, bool fp64, const float2 *tw32,
                  const double2 *tw64, cudaStream_t s, bool cond, bool split32) {
  // rows per block: as many as the transform size allows, but no fewer
  // blocks than about two per SM (so that a single signal, or the FP64
  // pipes, still spread over the GPU); every transform of the launch has at
  // most max_m points, so at least rpb rows per block
  if (!fp64 && max_m <= kDirectMaxM) {
    dim3 g((max_rows + kDirectRowsPerBlock - 1) / kDirectRowsPerBlock, max_trials,
           nsig);
    Launch(k_row_dft_small, g, 64 * kDirectRowsPerBlock, 0, s, d_its, cond ? 1 : 0);
    return;
  }
  // so few rows that a block each does not fill the SMs: a row over a cluster,
  // slices of kSplitMin elements or more. FP64: as many blocks as leave an SM
  // to each (two blocks on one SM share its pipes and gain nothing); FP32: up to
  // two per SM
  const int64_t total = int64_t(max_rows) * max_trials * nsig;
  if (fp64 || split32) {
    int c = 8;
    while (c > 1 && (total * c > (fp64 ? 152 : 304) || max_m < kSplitMin * c)) c /= 2;
    const dim3 g(max_rows, max_trials, nsig);
    if (fp64 ? LaunchRowSplits(d_its, g, c, max_m, tw64, s, cond)
             : LaunchRowSplits(d_its, g, c, max_m, tw32, s, cond)) {
      return;
    }
  }
  // (a power of two, so that a row's threads are whole shuffle segments)
  int rpb_cap = 1;
  while (int64_t(rpb_cap) * 2 <= total / (2 * 152)) {
    rpb_cap *= 2;
  }
  const int rpb = std::max(
      1, std::min({kRowsMax, kRowFftThreads * 8 / std::max(1, max_m), rpb_cap}));
  dim3 grid((max_rows + rpb - 1) / rpb, max_trials, nsig);
  if (fp64) {
    const size_t sm = RowFftSlots(max_m) * sizeof(double2);
    AllowSmem(k_row_fft<double2>, RowFftSlots(kMaxFFT64) * sizeof(double2));
    Launch(k_row_fft<double2>, grid, kRowFftThreads, sm, s, d_its, max_trials, tw64,
                                                        cond ? 1 : 0, rpb_cap);
  } else {
    const size_t sm = RowFftSlots(max_m) * sizeof(float2);
    AllowSmem(k_row_fft<float2>, RowFftSlots(kMaxFFT) * sizeof(float2));
    Launch(k_row_fft<float2>, grid, kRowFftThreads, sm, s, d_its, max_trials, tw32,
                                                       cond ? 1 : 0, rpb_cap);
  }
}

bool FftKernelsLaunchable() {
  int n1 = 0, n2 = 0;
  const size_t sm32 = RowFftSlots(kMaxFFT) * sizeof(float2);
  const size_t sm64 = RowFftSlots(kMaxFFT64) * sizeof(double2);
  AllowSmem(k_row_fft<float2>, sm32);
  AllowSmem(k_row_fft<double2>, sm64);
  // split rows: the largest transform over the smallest cluster
  int n3 = 0;
  const size_t sms = SplitSlots(kMaxFFT64, 2) * sizeof(double2);
  AllowSmem(k_row_fft_split<double2, 2>, sms);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n3, k_row_fft_split<double2, 2>,
                                                kSplitThreads, sms);
  if (n3 == 0) return false;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n1, k_row_fft<float2>, 512, sm32);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n2, k_row_fft<double2>, 512, sm64);
  return n1 > 0 && n2 > 0;
}

}  // namespace mpsft
