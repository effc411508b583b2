// v12.cu — the sFFT v1/v2 exec pipeline on GB300.
//
//   k_comb      (v2) strided W-point gather + shared-memory FFT + |.|^2 +
//               top-num residues (computefourier-1.0-2.0.cc:48-82) -> sorted,
//               de-duplicated residue list of the samplings  (:491-503);
//               from 1024 points k_comb_a / _b / _select over many CTAs
//   k_fold      permuted-filter fold, one thread per (loop, bucket),
//               taps summed in increasing order                      (:222-261);
//               FP32: k_fold_split
//   k_bucket    per loop: B-point FFT in shared memory, |.|^2, top-num
//               bucket selection                                    (:270-324);
//               FP64 from 1024 points k_bucket_a / _b / _select
//   k_vote_*    integer voting of the n/B frequencies of each selected
//               bucket                                               (:91-184)
//   k_estimate* per candidate: value in each loop, lower median of the
//               real and imaginary parts separately                 (:340-419)
//
// All kernels take a slot index (blockIdx.y or .z) so that one launch serves a
// batch of signals sharing a plan.  FP64 instantiations reproduce the CPU
// definition bit for bit; FP32 ones accumulate in float.
#include <algorithm>
#include <functional>
#include <queue>
#include <cstdlib>
#include <tuple>
#include <mutex>
#include <map>
#include <cfloat>
#include <climits>

#include "common.cuh"
#include "engine.h"
#include "fft.cuh"

namespace sfft {

template <typename R> __device__ __forceinline__ c2_t<R> cvt_in(double2 v);
template <> __device__ __forceinline__ double2 cvt_in<double>(double2 v) { return v; }
template <> __device__ __forceinline__ float2 cvt_in<float>(double2 v) {
  return make_float2(__double2float_rn(v.x), __double2float_rn(v.y));
}
template <typename R> __device__ __forceinline__ c2_t<R> cvt_in(float2 v);
template <> __device__ __forceinline__ double2 cvt_in<double>(float2 v) {
  return make_double2((double)v.x, (double)v.y);
}
template <> __device__ __forceinline__ float2 cvt_in<float>(float2 v) { return v; }

__device__ __forceinline__ int dlog2(unsigned v) { return 31 - __clz(v); }

// ------------------------------------------------------------------ fold --

template <typename R, typename In>
__global__ void __launch_bounds__(256, 4) k_fold(V12Dev d) {
  const int slot = blockIdx.y;
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= d.xs_size) return;
  const long locsz = (long)d.L_loc * d.B_loc;
  int j, b, B, w;
  const c2_t<R> *taps;
  if (g < locsz) {
    j = (int)(g / d.B_loc);
    b = (int)(g & (d.B_loc - 1));
    B = d.B_loc;
    w = d.w_loc;
    taps = (const c2_t<R> *)d.taps_loc;
  } else {
    const long h = g - locsz;
    j = d.L_loc + (int)(h / d.B_est);
    b = (int)(h & (d.B_est - 1));
    B = d.B_est;
    w = d.w_est;
    taps = (const c2_t<R> *)d.taps_est;
  }
  const int *rp = d.rparams + (long)slot * d.rp_stride;
  const unsigned long long ai = (unsigned)rp[d.L + j];
  const unsigned long long mask = (unsigned long long)d.n - 1;
  const In *x = (const In *)d.inputs[slot];
  c2_t<R> acc;
  acc.x = 0;
  acc.y = 0;
  // Gathers issued 4 at a time, summed in increasing tap order.  Four blocks
  // an SM with 4 gathers each keep the FP64 pipes busier than two with 8,
  // which need 102 registers a thread (one signal of 2^13 points 14.9 ->
  // 12.9 us, of 2^20 24.8 -> 19.9, 64 of 2^16 234.5 -> 232.7).
  for (int t0 = b; t0 < w; t0 += 4 * B) {
    c2_t<R> xv[4], hv[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int t = t0 + u * B;
      if (t < w) {
        const unsigned long long idx = ((unsigned long long)t * ai) & mask;
        xv[u] = cvt_in<R>(__ldg(x + idx));
        hv[u] = __ldg(taps + t);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (t0 + u * B < w) acc = cadd<R>(acc, cmul<R>(xv[u], hv[u]));
  }
  ((c2_t<R> *)d.xs)[(long)slot * d.xs_size + g] = acc;
}

// FP32 form of the fold with each bucket's taps split over S adjacent
// lanes (tap m of the bucket goes to lane m mod S), the S partial sums
// combined by shuffles.  A signal then spans S times as many threads as
// buckets, so the GPU's resident threads work on about one signal at a
// time: that signal's input stays in L2 while all its loops gather from it,
// instead of several signals' inputs contending for L2 and being fetched
// from DRAM repeatedly.  The summation order differs from the reference's,
// which the FP32 form does not reproduce anyway.
template <typename In, int S, int U = 4>
__device__ __forceinline__ void fold_split_thread(const V12Dev &d, int slot, long gt) {
  const long g = gt / S;
  const int part = (int)(gt % S);
  const bool live = g < d.xs_size;
  const long locsz = (long)d.L_loc * d.B_loc;
  int j = 0, b = 0, B = 1, w = 0;
  const float2 *taps = nullptr;
  if (live) {
    if (g < locsz) {
      j = (int)(g / d.B_loc);
      b = (int)(g & (d.B_loc - 1));
      B = d.B_loc;
      w = d.w_loc;
      taps = (const float2 *)d.taps_loc;
    } else {
      const long h = g - locsz;
      j = d.L_loc + (int)(h / d.B_est);
      b = (int)(h & (d.B_est - 1));
      B = d.B_est;
      w = d.w_est;
      taps = (const float2 *)d.taps_est;
    }
  }
  float2 acc = make_float2(0.f, 0.f);
  if (live) {
    const int *rp = d.rparams + (long)slot * d.rp_stride;
    const unsigned ai = (unsigned)rp[d.L + j], mask = (unsigned)d.n - 1u;
    const In *x = (const In *)d.inputs[slot];
    const int step = S * B;
    for (int t0 = b + part * B; t0 < w; t0 += U * step) {  // U gathers in flight
      float2 xv[U], hv[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int t = t0 + u * step;
        if (t < w) {
          xv[u] = cvt_in<float>(__ldg(x + (((unsigned)t * ai) & mask)));
          hv[u] = __ldg(taps + t);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++)
        if (t0 + u * step < w) acc = cadd<float>(acc, cmul<float>(xv[u], hv[u]));
    }
  }
#pragma unroll
  for (int o = S / 2; o > 0; o >>= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
  }
  if (live && part == 0) ((float2 *)d.xs)[(long)slot * d.xs_size + g] = acc;
}

template <typename In, int S>
__global__ void __launch_bounds__(256) k_fold_split(V12Dev d) {
  fold_split_thread<In, S>(d, blockIdx.y, (long)blockIdx.x * blockDim.x + threadIdx.x);
}

// ------------------------------------------------------- one-CTA FFTs --

// FFT and selection keys of N points in one CTA.  FP32: block_fft16, keys
// recomputed from the values (two FMAs); FP64: one radix-4 butterfly per
// thread and stage (PER of them beyond 1024 threads), keys stored beside the
// values (a recomputed one costs three FP64 instructions).
template <typename R>
struct OneCta;

template <>
struct OneCta<float> {
  static constexpr int threads(int N) { return N / 16 < 128 ? 128 : N / 16; }
  static size_t bytes(int N) { return sizeof(float2) * (size_t)fft16_size(N); }
  float2 *buf;
  __device__ __forceinline__ OneCta(unsigned char *smem, int) : buf((float2 *)smem) {}
  template <int PER, typename Ld>
  __device__ __forceinline__ void fft(int N, const float2 *tw, Ld ld) {
    if (N >= 16) {
      block_fft16<float>(buf, N, dlog2(N), tw, ld);
    } else {
      for (int i = threadIdx.x; i < N; i += blockDim.x) buf[i] = ld(i);
      __syncthreads();
      block_fft<float, 1>(buf, N, dlog2(N), tw);
    }
  }
  __device__ __forceinline__ float2 at(int i) const { return buf[fft16_at(i)]; }
  __device__ __forceinline__ unsigned key(int i) const { return pkey(cabs2<float>(at(i))); }
};

template <>
struct OneCta<double> {
  static constexpr int threads(int N) { return N / 4 < 128 ? 128 : N / 4 > 1024 ? 1024 : N / 4; }
  static size_t bytes(int N) { return (sizeof(double2) + sizeof(unsigned long long)) * (size_t)N; }
  double2 *buf;
  unsigned long long *keys;
  __device__ __forceinline__ OneCta(unsigned char *smem, int N)
      : buf((double2 *)smem), keys((unsigned long long *)(buf + N)) {}
  template <int PER, typename Ld>
  __device__ __forceinline__ void fft(int N, const double2 *tw, Ld ld) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) buf[i] = ld(i);
    __syncthreads();
    block_fft<double, PER>(buf, N, dlog2(N), tw);
    for (int i = threadIdx.x; i < N; i += blockDim.x) keys[i] = pkey(cabs2<double>(buf[i]));
    __syncthreads();
  }
  __device__ __forceinline__ double2 at(int i) const { return buf[i]; }
  __device__ __forceinline__ unsigned long long key(int i) const { return keys[i]; }
};

// ------------------------------------------------------------------ comb --

// Residues of one comb sampling: one bit plane per sampling (plain stores,
// nothing to clear); a single sampling's residues are the list itself.
template <typename K, int S, typename KeyAt>
__device__ __forceinline__ void comb_select(const V12Dev &d, int c, int slot, KeyAt keyat, SelShared<K> &ss) {
  const int W = d.W, words = (W + 31) >> 5;
  const bool one = d.comb_loops == 1;
  block_select<K, S>(keyat, W, d.num, one ? d.comb_list + (long)slot * W : nullptr,
                  d.comb_bits + ((long)slot * d.comb_loops + c) * words, ss);
  if (one && threadIdx.x == 0) d.counters[slot * CNT_STRIDE + CNT_COMB] = d.num;
}

// The union of the samplings' planes as a bitmap (plane 0) and as a sorted
// list.
__device__ __forceinline__ void comb_list_block(const V12Dev &d, int slot) {
  __shared__ int scan[64];
  const int W = d.W;
  const int words = (W + 31) >> 5;
  unsigned *bits = d.comb_bits + (long)slot * d.comb_loops * words;
  const int C = (words + blockDim.x - 1) / blockDim.x;
  const int lo = min(words, (int)threadIdx.x * C), hi = min(words, lo + C);
  int cnt = 0;
  for (int i = lo; i < hi; i++) {
    unsigned v = __ldcg(bits + i);
    for (int c = 1; c < d.comb_loops; c++) v |= __ldcg(bits + (long)c * words + i);
    bits[i] = v;
    cnt += __popc(v);
  }
  int pre, dummy;
  int2 tot = block_exscan2(cnt, 0, pre, dummy, scan);
  int *list = d.comb_list + (long)slot * W;
  for (int i = lo; i < hi; i++) {
    unsigned v = bits[i];
    while (v) {
      int bpos = __ffs(v) - 1;
      list[pre++] = i * 32 + bpos;
      v &= v - 1;
    }
  }
  if (threadIdx.x == 0) d.counters[slot * CNT_STRIDE + CNT_COMB] = tot.x;
}

// With several samplings the last CTA of a slot to finish builds the list.
__device__ __forceinline__ void comb_last_list(const V12Dev &d, int slot) {
  if (d.comb_loops == 1) return;
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0)
    last = atomicAdd(&d.counters[slot * CNT_STRIDE + CNT_TICKET], 1) == d.comb_loops - 1;
  __syncthreads();
  if (last) {
    __threadfence();
    comb_list_block(d, slot);
  }
}

template <typename R, int PER, typename In>
__device__ __forceinline__ void comb_block(const V12Dev &d, int c, int slot, unsigned char *smem,
                                           SelShared<key_t<R>> &ss) {
  const int W = d.W;
  OneCta<R> f(smem, W);
  const int *rp = d.rparams + (long)slot * d.rp_stride;
  const long sigma = d.n / W;
  const In *x = (const In *)d.inputs[slot] + rp[2 * d.L + c];
  f.template fft<PER>(W, (const c2_t<R> *)d.tw_comb, [=](int i) { return cvt_in<R>(__ldg(x + i * sigma)); });
  comb_select<key_t<R>, 16>(d, c, slot, [&](int i) { return f.key(i); }, ss);
}

template <typename R, int PER, typename In>
__global__ void __launch_bounds__(1024) k_comb(V12Dev d) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SelShared<key_t<R>> ss;
  comb_block<R, PER, In>(d, blockIdx.x, blockIdx.y, smem, ss);
  comb_last_list(d, blockIdx.y);
}

// ---------------------------------------------------------------- voting --
//
// In location loop j, frequency f gets a vote iff its position p = f ai_j (mod
// n) lies in the range [J q - q / 2, + q) (mod n) of a selected bucket J
// (v2: and f mod W is a comb residue; computefourier-1.0-2.0.cc:91-116,
// :125-184), that is iff bucket ((p + q / 2) mod n) / q is selected.  No count
// is added to in global memory; one thread or block owns each frequency:
//
//   k_vote_residue  (v2) a block counts the n / W frequencies of one comb
//                   residue in shared memory, one step per (loop, selected
//                   bucket): the range of J holds the positions congruent to
//                   r ai (mod W), at most q / W + 1 of them.
//   k_vote_cands    (v2) one thread per comb candidate, one bit test per loop
//                   in the bitmap of selected buckets the selection leaves.
//   k_vote_ranges   (v1) one thread per position of the selected ranges, the
//                   same bit tests; the first loop that selected a frequency
//                   owns it.
//
// v2 takes the first form when its steps, 2 k (q / W + 1) per residue and
// loop, are fewer than the n / W bit tests of the second.  Frequencies that
// reach the threshold are collected per block: one returning atomic a warp
// on a signal's hit counter, about 2 ns each at one address, takes 200 us for
// four voted signals of n = 2^22, k = 500.  Kernel times: those signals, two
// atomics per vote 283 -> 48 us (bit tests with the block's hits: 225 us with
// warp atomics); 32 plain signals of n = 2^22, k = 100: 45 -> 27 us (bit
// tests: 46); 64 v1 signals of n = 2^16: 28 -> 18 us.
//
// The counts stay in score for diagnostics: (epoch << 8) | votes, so that
// counts of earlier executions need no clearing; v2 keeps them
// residue-major, frequency f = rep W + r at r (n / W) + rep, where a
// residue's counts are consecutive.

// The bitmaps of the location loops: in shared memory unless they are large.
constexpr int VOTE_SMEM = 32 * 1024;
__host__ __device__ __forceinline__ int vote_words(int B) { return (B + 31) >> 5; }
static size_t vote_smem(const V12Dev &d) {
  const size_t b = sizeof(unsigned) * (size_t)d.L_loc * vote_words(d.B_loc);
  return b <= VOTE_SMEM ? b : 0;
}
__device__ __forceinline__ const unsigned *vote_bits(const V12Dev &d, int slot, unsigned *smem) {
  const int words = d.L_loc * vote_words(d.B_loc);
  const unsigned *src = d.sel_bits + (long)slot * words;
  if (words * (int)sizeof(unsigned) > VOTE_SMEM) return src;
  for (int i = threadIdx.x; i < words; i += blockDim.x) smem[i] = src[i];
  __syncthreads();
  return smem;
}

// Hits of a block (v1, and v2 in the voted mode): places are taken within
// the block first, then one place range for all of them in the signal's list.
struct VoteHits {
  int n, base;
};
__device__ __forceinline__ void hits_begin(VoteHits &h) {  // a barrier follows before the first place
  if (threadIdx.x == 0) h.n = 0;
}
__device__ __forceinline__ void hits_place(const V12Dev &d, int slot, VoteHits &h) {
  __syncthreads();
  if (threadIdx.x == 0 && h.n) {
    int *cnt = d.counters + slot * CNT_STRIDE;
    h.base = atomicAdd(&cnt[CNT_HITS], h.n);
    atomicAdd(&cnt[CNT_VOTED], h.n);
    if (h.base + h.n > d.hit_cap) atomicOr(&cnt[CNT_ERR], ERR_HIT_OVERFLOW);
  }
  __syncthreads();
}
__device__ __forceinline__ void hits_store(const V12Dev &d, int slot, const VoteHits &h, int place, unsigned f) {
  if (h.base + place < d.hit_cap) d.hits[(long)slot * d.hit_cap + h.base + place] = (int)f;
}

__device__ __forceinline__ unsigned vote_in(const V12Dev &d, const unsigned *sb, int j, unsigned ai, unsigned f) {
  const unsigned mask = (unsigned)d.n - 1u, q = (unsigned)d.q_loc;
  const unsigned b = ((f * ai + (q >> 1)) & mask) >> dlog2(q);
  return (sb[j * vote_words(d.B_loc) + (int)(b >> 5)] >> (b & 31u)) & 1u;
}

// v2: the votes of comb candidates h0 + u blockDim + thread, u < U
// (candidates as in cand_freq: residue-major).
template <int U>
__device__ __forceinline__ void vote_cands(const V12Dev &d, int slot, long h0, const unsigned *sb, VoteHits &hits) {
  const int *rp = d.rparams + (long)slot * d.rp_stride;
  const unsigned ep = (unsigned)rp[2 * d.L + d.comb_loops];
  const int lw = dlog2((unsigned)d.W), lr = dlog2((unsigned)d.n) - lw;
  const long total = (long)d.counters[slot * CNT_STRIDE + CNT_COMB] << lr;
  const int *list = d.comb_list + (long)slot * d.W;
  unsigned *score = d.score + (long)slot * d.n;
  unsigned f[U], votes[U];
  if (d.voted) {
    hits_begin(hits);
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
    const long h = h0 + (long)u * blockDim.x + threadIdx.x;
    f[u] = h < total ? (((unsigned)h & ((1u << lr) - 1u)) << lw) | (unsigned)list[h >> lr] : 0u;
    votes[u] = 0;
  }
  for (int j = 0; j < d.L_loc; j++) {
    const unsigned ai = (unsigned)rp[d.L + j];
#pragma unroll
    for (int u = 0; u < U; u++) votes[u] += vote_in(d, sb, j, ai, f[u]);
  }
  int place[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    if (h0 + (long)u * blockDim.x + threadIdx.x >= total) votes[u] = 0;
    // residue f mod W, repetition f / W
    if (votes[u]) score[((f[u] & ((1u << lw) - 1u)) << lr) | (f[u] >> lw)] = (ep << 8) | votes[u];
    place[u] = d.voted && (int)votes[u] >= d.thresh ? atomicAdd(&hits.n, 1) : -1;
  }
  if (d.voted) {
    hits_place(d, slot, hits);
#pragma unroll
    for (int u = 0; u < U; u++)
      if (place[u] >= 0) hits_store(d, slot, hits, place[u], f[u]);
  }
}

template <int U>
__global__ void __launch_bounds__(256) k_vote_cands(V12Dev d) {
  extern __shared__ unsigned vb[];
  __shared__ VoteHits hits;
  const unsigned *sb = vote_bits(d, blockIdx.y, vb);
  vote_cands<U>(d, blockIdx.y, (long)blockIdx.x * 256 * U, sb, hits);
}

// v2, one comb residue per block; n / W byte counters in shared memory (a
// frequency gets at most one vote per loop, of at most 32).
__device__ __forceinline__ void vote_residue(const V12Dev &d, int slot, int ridx, unsigned *cw, VoteHits &hits) {
  const int *rp = d.rparams + (long)slot * d.rp_stride;
  const unsigned mask = (unsigned)d.n - 1u, wm = (unsigned)d.W - 1u, q = (unsigned)d.q_loc;
  const int lw = dlog2((unsigned)d.W), lr = dlog2((unsigned)d.n) - lw, words = (1 << lr) >> 2;
  const unsigned r = (unsigned)d.comb_list[(long)slot * d.W + ridx], ep = (unsigned)rp[2 * d.L + d.comb_loops];
  for (int i = threadIdx.x; i < words; i += blockDim.x) cw[i] = 0u;
  hits_begin(hits);
  __syncthreads();
  for (int j = 0; j < d.L_loc; j++) {
    const int *Js = d.J + ((long)slot * d.L + j) * d.num;
    const unsigned a = (unsigned)rp[j], c = (r * (unsigned)rp[d.L + j]) & wm;
    for (int t = threadIdx.x; t < d.num; t += blockDim.x) {
      const unsigned low = ((unsigned)Js[t] * q - (q >> 1)) & mask;
      for (unsigned k = (c - low) & wm; k < q; k += (unsigned)d.W) {
        const unsigned rep = (((low + k) * a) & mask) >> lw;
        atomicAdd(&cw[rep >> 2], 1u << (8 * (rep & 3u)));
      }
    }
  }
  __syncthreads();
  uint4 *score = (uint4 *)(d.score + (long)slot * d.n + ((long)r << lr));
  const unsigned tag = ep << 8;
  for (int i = threadIdx.x; i < words; i += blockDim.x) {
    const unsigned v = cw[i];
    if (!v) continue;
    score[i] = make_uint4(tag | (v & 255u), tag | ((v >> 8) & 255u), tag | ((v >> 16) & 255u), tag | (v >> 24));
    if (d.voted) {
      int c = 0;
#pragma unroll
      for (int b = 0; b < 4; b++) c += (int)((v >> (8 * b)) & 255u) >= d.thresh;
      if (c) atomicAdd(&hits.n, c);
    }
  }
  if (!d.voted) return;
  hits_place(d, slot, hits);
  if (!hits.n) return;
  __syncthreads();  // every thread has read n
  if (threadIdx.x == 0) hits.n = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < words; i += blockDim.x) {
    const unsigned v = cw[i];
#pragma unroll
    for (int b = 0; b < 4; b++)
      if (v && (int)((v >> (8 * b)) & 255u) >= d.thresh)
        hits_store(d, slot, hits, atomicAdd(&hits.n, 1), ((unsigned)(4 * i + b) << lw) | r);
  }
}

__global__ void __launch_bounds__(256) k_vote_residue(V12Dev d) {
  extern __shared__ unsigned cw[];
  __shared__ VoteHits hits;
  const int slot = blockIdx.y;
  if ((int)blockIdx.x >= d.counters[slot * CNT_STRIDE + CNT_COMB]) return;
  vote_residue(d, slot, blockIdx.x, cw, hits);
}

// Whether v2's votes go by residue (see above): fewer steps than bit tests,
// and the counters fit (n / W of 4 .. 32768).
__host__ __device__ __forceinline__ bool vote_by_residue(const V12Dev &d) {
  const long R = d.n / d.W;
  return R >= 4 && R <= 32768 && (long)d.num * (d.q_loc / d.W + 1) < R;
}

// v1: VOTE_V positions of one loop's selected ranges per thread.
constexpr int VOTE_V = 4;

__global__ void __launch_bounds__(256) k_vote_ranges(V12Dev d, int per_loop_blocks) {
  extern __shared__ unsigned vb[];
  __shared__ VoteHits hits;
  hits_begin(hits);
  const int slot = blockIdx.y;
  const unsigned *sb = vote_bits(d, slot, vb);
  __syncthreads();
  const int q = d.q_loc, lq = dlog2(q);
  const int j = blockIdx.x / per_loop_blocks, tile = blockIdx.x - j * per_loop_blocks;
  const long per_loop = (long)d.num << lq, g0 = (long)tile * (256 * VOTE_V) + threadIdx.x;
  const int *Js = d.J + ((long)slot * d.L + j) * d.num;
  const int *rp = d.rparams + (long)slot * d.rp_stride;
  const unsigned mask = (unsigned)d.n - 1u, tag = (unsigned)rp[2 * d.L + d.comb_loops] << 8;
  unsigned f[VOTE_V];
  int place[VOTE_V];
#pragma unroll
  for (int v = 0; v < VOTE_V; v++) {
    const long g = g0 + 256 * v;
    place[v] = -1;
    f[v] = 0;
    if (g < per_loop) {
      const unsigned e = (unsigned)g, J = (unsigned)Js[e >> lq];
      const unsigned p = (J * (unsigned)q - (unsigned)(q >> 1) + (e & (unsigned)(q - 1))) & mask;
      f[v] = (p * (unsigned)rp[j]) & mask;
      unsigned before = 0, votes = 1;
      for (int t = 0; t < j; t++) before |= vote_in(d, sb, t, (unsigned)rp[d.L + t], f[v]);
      for (int t = j + 1; t < d.L_loc; t++) votes += vote_in(d, sb, t, (unsigned)rp[d.L + t], f[v]);
      if (!before) {
        d.score[(long)slot * d.n + f[v]] = tag | votes;
        if ((int)votes >= d.thresh) place[v] = atomicAdd(&hits.n, 1);
      }
    }
  }
  hits_place(d, slot, hits);
#pragma unroll
  for (int v = 0; v < VOTE_V; v++)
    if (place[v] >= 0) hits_store(d, slot, hits, place[v], f[v]);
}

// ---------------------------------------------------------------- bucket --

// Place of bucket i in a loop's x_samp: (i mod T) * G + i / T in the grouped
// layout (xs_perm = log2 G).
__device__ __forceinline__ int xs_place(int i, int lg, int lt) {
  return lg ? ((i & ((1 << lt) - 1)) << lg) | (i >> lt) : i;
}

struct LoopSpan {
  int B;
  long off;
  bool loc;
};
__device__ __forceinline__ LoopSpan loop_span(const V12Dev &d, int j) {
  LoopSpan l;
  l.loc = j < d.L_loc;
  l.B = l.loc ? d.B_loc : d.B_est;
  l.off = l.loc ? (long)j * d.B_loc : (long)d.L_loc * d.B_loc + (long)(j - d.L_loc) * d.B_est;
  return l;
}

// The bitmap of loop j's selected buckets (location loops only).
__device__ __forceinline__ unsigned *sel_plane(const V12Dev &d, int slot, int j) {
  return j < d.L_loc ? d.sel_bits + ((long)slot * d.L_loc + j) * vote_words(d.B_loc) : nullptr;
}

template <typename R, int PER>
__device__ __forceinline__ void bucket_block(const V12Dev &d, int j, int slot, unsigned char *smem,
                                             SelShared<key_t<R>> &ss) {
  const LoopSpan l = loop_span(d, j);
  const int B = l.B;
  OneCta<R> f(smem, B);
  c2_t<R> *xs = (c2_t<R> *)d.xs + (long)slot * d.xs_size + l.off;
  f.template fft<PER>(B, (const c2_t<R> *)(l.loc ? d.tw_loc : d.tw_est), [=](int i) { return xs[i]; });
  float2 *xs32 = d.xs32 ? (float2 *)d.xs32 + (long)slot * d.xs_size + l.off : nullptr;
  const int lg = d.xs_perm, lt = dlog2(B) - lg, gm = (1 << lg) - 1;
#pragma unroll 4
  for (int p = threadIdx.x; p < B; p += blockDim.x) {  // in the order of the places: coalesced
    const c2_t<R> v = f.at(lg ? ((p & gm) << lt) | (p >> lg) : p);
    xs[p] = v;
    if (xs32) xs32[p] = make_float2((float)v.x, (float)v.y);
  }
  block_select<key_t<R>, 16>([&](int i) { return f.key(i); }, B, d.num, d.J + ((long)slot * d.L + j) * d.num,
                         sel_plane(d, slot, j), ss);
}

template <typename R, int PER>
__global__ void __launch_bounds__(1024) k_bucket(V12Dev d) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SelShared<key_t<R>> ss;
  bucket_block<R, PER>(d, blockIdx.x, blockIdx.y, smem, ss);
}

// ------------------------------------------------ FFTs over many CTAs --
//
// Bucket and comb FFTs as two launches of fft_tile and one of the selection
// (which reads the keys the second launch leaves).

// First launch: stages 1 .. M1 of every loop's array, xs -> xs_tmp.
template <typename R>
__global__ void __launch_bounds__(1024) k_bucket_a(V12Dev d, int elems, int nloc, int nest) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int x = blockIdx.x, slot = blockIdx.y;
  const int j = x < d.L_loc * nloc ? x / nloc : d.L_loc + (x - d.L_loc * nloc) / nest;
  const int tile = x < d.L_loc * nloc ? x % nloc : (x - d.L_loc * nloc) % nest;
  const LoopSpan l = loop_span(d, j);
  const int M = l.B / fft_m2(l.B), lc = fft_lc(elems, M, l.B);
  const c2_t<R> *src = (const c2_t<R> *)d.xs + (long)slot * d.xs_size + l.off;
  c2_t<R> *dst = (c2_t<R> *)d.xs_tmp + (long)slot * d.xs_size + l.off;
  fft_tile<R>((c2_t<R> *)smem, M, lc, 1, l.B, tile << lc, dlog2(l.B) & 1,
              (const c2_t<R> *)(l.loc ? d.tw_loc : d.tw_est), [=](int i) { return src[i]; },
              [=](int i, c2_t<R> v) { dst[i] = v; });
}

// Second launch: the remaining stages, xs_tmp -> xs (in its layout), the
// FP32 copy and the selection keys.
template <typename R>
__global__ void __launch_bounds__(1024) k_bucket_b(V12Dev d, int elems, int nloc, int nest) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int x = blockIdx.x, slot = blockIdx.y;
  const int j = x < d.L_loc * nloc ? x / nloc : d.L_loc + (x - d.L_loc * nloc) / nest;
  const int tile = x < d.L_loc * nloc ? x % nloc : (x - d.L_loc * nloc) % nest;
  const LoopSpan l = loop_span(d, j);
  const int M = fft_m2(l.B), lc = fft_lc(elems, M, l.B);
  const long at = (long)slot * d.xs_size + l.off;
  const c2_t<R> *src = (const c2_t<R> *)d.xs_tmp + at;
  c2_t<R> *dst = (c2_t<R> *)d.xs + at;
  float2 *dst32 = d.xs32 ? (float2 *)d.xs32 + at : nullptr;
  key_t<R> *pw = (key_t<R> *)d.pw + at;
  const int lg = d.xs_perm, lt = dlog2(l.B) - lg;
  fft_tile<R>((c2_t<R> *)smem, M, lc, l.B / M, l.B, tile << lc, false,
              (const c2_t<R> *)(l.loc ? d.tw_loc : d.tw_est), [=](int i) { return src[i]; },
              [=](int i, c2_t<R> v) {
                const int p = xs_place(i, lg, lt);
                dst[p] = v;
                if (dst32) dst32[p] = make_float2((float)v.x, (float)v.y);
                pw[i] = pkey(cabs2<R>(v));
              });
}

// Selection of loop j from its keys: S of them per thread (S = 0: any number).
template <typename R, int S>
__global__ void __launch_bounds__(1024) k_bucket_select(V12Dev d) {
  using K = key_t<R>;
  __shared__ SelShared<K> ss;
  const int j = blockIdx.x, slot = blockIdx.y;
  const LoopSpan l = loop_span(d, j);
  const K *pw = (const K *)d.pw + (long)slot * d.xs_size + l.off;
  block_select<K, S>([=](int i) { return pw[i]; }, l.B, d.num, d.J + ((long)slot * d.L + j) * d.num,
                     sel_plane(d, slot, j), ss);
}

template <typename R, typename In>
__global__ void __launch_bounds__(1024) k_comb_a(V12Dev d, int elems) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int c = blockIdx.y, slot = blockIdx.z, W = d.W;
  const int M = W / fft_m2(W), lc = fft_lc(elems, M, W);
  const int *rp = d.rparams + (long)slot * d.rp_stride;
  const long sigma = d.n / W;
  const In *x = (const In *)d.inputs[slot] + rp[2 * d.L + c];
  c2_t<R> *dst = (c2_t<R> *)d.comb_tmp + ((long)slot * d.comb_loops + c) * W;
  fft_tile<R>((c2_t<R> *)smem, M, lc, 1, W, (int)blockIdx.x << lc, dlog2(W) & 1, (const c2_t<R> *)d.tw_comb,
              [=](int i) { return cvt_in<R>(__ldg(x + i * sigma)); }, [=](int i, c2_t<R> v) { dst[i] = v; });
}

template <typename R>
__global__ void __launch_bounds__(1024) k_comb_b(V12Dev d, int elems) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int c = blockIdx.y, slot = blockIdx.z, W = d.W;
  const int M = fft_m2(W), lc = fft_lc(elems, M, W);
  const c2_t<R> *src = (const c2_t<R> *)d.comb_tmp + ((long)slot * d.comb_loops + c) * W;
  key_t<R> *pw = (key_t<R> *)d.comb_pw + ((long)slot * d.comb_loops + c) * W;
  fft_tile<R>((c2_t<R> *)smem, M, lc, W / M, W, (int)blockIdx.x << lc, false, (const c2_t<R> *)d.tw_comb,
              [=](int i) { return src[i]; }, [=](int i, c2_t<R> v) { pw[i] = pkey(cabs2<R>(v)); });
}

template <typename R, int S>
__global__ void __launch_bounds__(1024) k_comb_select(V12Dev d) {
  using K = key_t<R>;
  __shared__ SelShared<K> ss;
  const int c = blockIdx.x, slot = blockIdx.y, W = d.W;
  const K *pw = (const K *)d.comb_pw + ((long)slot * d.comb_loops + c) * W;
  comb_select<K, S>(d, c, slot, [=](int i) { return pw[i]; }, ss);
  comb_last_list(d, slot);
}

// One Stockham stage over `narr` arrays of N points per slot (plan-time
// transforms of up to 2^30 points).
template <typename R>
__global__ void __launch_bounds__(256) k_fft_stage(const c2_t<R> *src, c2_t<R> *dst, int N, int Ns, int radix,
                                                   long arr_stride, int narr, long slot_stride,
                                                   const c2_t<R> *tw) {
  const int slot = blockIdx.y;
  const int per = N / radix;
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long)narr * per) return;
  const int arr = (int)(g / per), j = (int)(g - (long)arr * per);
  const long base = (long)slot * slot_stride + (long)arr * arr_stride;
  stockham_stage<R>(src + base, dst + base, N, Ns, radix, j, tw);
}

// FFT of `narr` arrays per slot held at a (ping) with b as scratch; the
// result ends in a.  Stage sequence of block_fft.
template <typename R>
static cudaError_t global_fft(c2_t<R> *a, c2_t<R> *b, int N, int narr, long arr_stride, long slot_stride,
                              int nslots, const c2_t<R> *tw, cudaStream_t s) {
  int logN = 0;
  while ((1 << logN) < N) logN++;
  c2_t<R> *src = a, *dst = b;
  int Ns = 1, launches = 0;
  auto stage = [&](int radix) -> cudaError_t {
    const long work = (long)narr * (N / radix);
    dim3 grid((unsigned)((work + 255) / 256), nslots);
    k_fft_stage<R><<<grid, 256, 0, s>>>(src, dst, N, Ns, radix, arr_stride, narr, slot_stride, tw);
    launches++;
    c2_t<R> *t = src;
    src = dst;
    dst = t;
    return cudaGetLastError();
  };
  cudaError_t e;
  if (logN & 1) {
    if ((e = stage(2))) return e;
    Ns = 2;
  }
  while (Ns < N) {
    if ((e = stage(4))) return e;
    Ns *= 4;
  }
  note_launches(launches);
  if (src != a) {  // odd number of stages: bring the result home
    for (int sl = 0; sl < nslots; sl++) {
      if ((e = cudaMemcpyAsync(a + sl * slot_stride, src + sl * slot_stride,
                               sizeof(c2_t<R>) * ((narr - 1) * arr_stride + N), cudaMemcpyDeviceToDevice, s)))
        return e;
    }
  }
  return cudaSuccess;
}

// -------------------------------------------------------------- estimate --

// Knuth's merge-exchange sorting network (TAOCP vol. 3, 5.2.2, Algorithm M)
// for N elements, generated at compile time; used through Cswap so that
// every comparator's indices are constants (the values stay in registers).
template <int N>
struct SortNet {
  static constexpr int count() {
    if (N < 2) return 0;
    int t = 0;
    while ((1 << t) < N) t++;
    int c = 0;
    for (int p = 1 << (t - 1); p > 0; p >>= 1) {
      int q = 1 << (t - 1), r = 0, dd = p;
      for (;;) {
        for (int i = 0; i + dd < N; i++)
          if ((i & p) == r) c++;
        if (q == p) break;
        dd = q - p;
        q >>= 1;
        r = p;
      }
    }
    return c;
  }
  static constexpr int C = count();
  int a[C > 0 ? C : 1], b[C > 0 ? C : 1];
  constexpr SortNet() : a(), b() {
    if (N < 2) return;
    int t = 0;
    while ((1 << t) < N) t++;
    int c = 0;
    for (int p = 1 << (t - 1); p > 0; p >>= 1) {
      int q = 1 << (t - 1), r = 0, dd = p;
      for (;;) {
        for (int i = 0; i + dd < N; i++)
          if ((i & p) == r) {
            a[c] = i;
            b[c] = i + dd;
            c++;
          }
        if (q == p) break;
        dd = q - p;
        q >>= 1;
        r = p;
      }
    }
  }
};

template <int N> struct NetOf { static constexpr SortNet<N> net{}; };

template <int N, int c, int C>
struct Cswap {
  static __device__ __forceinline__ void run(float (&v)[N]) {
    constexpr int i = NetOf<N>::net.a[c], j = NetOf<N>::net.b[c];
    const float x = v[i], y = v[j];
    v[i] = fminf(x, y);
    v[j] = fmaxf(x, y);
    Cswap<N, c + 1, C>::run(v);
  }
};
template <int N, int C>
struct Cswap<N, C, C> {
  static __device__ __forceinline__ void run(float (&)[N]) {}
};

template <int N>
__device__ __forceinline__ void sort_net(float (&v)[N]) {
  Cswap<N, 0, SortNet<N>::C>::run(v);
}

// Parberry's pairwise sorting network on P = 2^t wires (I. Parberry, "The
// pairwise sorting network", Parallel Processing Letters 2(2-3), 1992):
// calls f(i, j), i < j, for its comparators in order.  Its first half sorts
// pairs, then quadruples, ... of a bitonic-free layout; its second half
// merges with comparators (b - d a, b).
template <typename F>
constexpr void pairwise_net(int P, F &&f) {
  int a = 1;
  for (; a < P; a *= 2) {
    int b = a, c = 0;
    while (b < P) {
      f(b - a, b);
      b++;
      c = (c + 1) % a;
      if (c == 0) b += a;
    }
  }
  a /= 4;
  for (int e = 1; a > 0; a /= 2, e = 2 * e + 1) {
    for (int d = e; d > 0; d /= 2) {
      int b = (d + 1) * a, c = 0;
      while (b < P) {
        f(b - d * a, b);
        b++;
        c = (c + 1) % a;
        if (c == 0) b += a;
      }
    }
  }
}

constexpr int pow2_ceil(int n) {
  int p = 1;
  while (p < n) p *= 2;
  return p;
}

// A selection network for element M of N values: the pairwise network on
// P = pow2_ceil(N) wires restricted to the N wires [s, s + N) -- with -inf
// below s and +inf from s + N on, a comparator touching an outside wire
// moves nothing, so the inside comparators sort any N values -- then
// pruned to output M by backward liveness: a comparator whose outputs are
// both dead is dropped, one with a single live output keeps only its min
// or its max.  The offset s with the fewest min/max operations is chosen
// at compile time (lower median of 20: 125 operations, against 143 for
// the pruned merge-exchange network).  Comparator kinds: 1 both outputs,
// 2 min only, 3 max only.
template <int N, int M>
struct SelNet {
  static constexpr int P = pow2_ceil(N);
  static constexpr int FULL = [] {
    int c = 0;
    pairwise_net(P, [&](int, int) { c++; });
    return c;
  }();
  int C = 0, ops = 0;
  signed char a[FULL > 0 ? FULL : 1] = {}, b[FULL > 0 ? FULL : 1] = {}, kind[FULL > 0 ? FULL : 1] = {};
  // the network at offset s, pruned: fills a, b, kind, C; returns its operation count
  constexpr int build(int s) {
    int fa[FULL > 0 ? FULL : 1] = {}, fb[FULL > 0 ? FULL : 1] = {};
    int n = 0;
    pairwise_net(P, [&](int i, int j) {
      if (i >= s && j < s + N) {
        fa[n] = i - s;
        fb[n] = j - s;
        n++;
      }
    });
    bool live[N] = {};
    live[M] = true;
    signed char k[FULL > 0 ? FULL : 1] = {};
    int cnt = 0, o = 0;
    for (int c = n - 1; c >= 0; c--) {
      const bool li = live[fa[c]], lj = live[fb[c]];
      k[c] = li && lj ? 1 : li ? 2 : lj ? 3 : 0;
      if (li || lj) {
        live[fa[c]] = live[fb[c]] = true;
        cnt++;
        o += (li && lj) ? 2 : 1;
      }
    }
    C = 0;
    for (int c = 0; c < n; c++)
      if (k[c]) {
        a[C] = (signed char)fa[c];
        b[C] = (signed char)fb[c];
        kind[C] = k[c];
        C++;
      }
    ops = o;
    return o;
  }
  constexpr SelNet() {
    if (N < 2) return;
    int best = -1, bs = 0;
    for (int s = 0; s + N <= P; s++) {
      const int o = build(s);
      if (best < 0 || o < best) {
        best = o;
        bs = s;
      }
    }
    build(bs);
  }
};
template <int N, int M> struct SelOf { static constexpr SelNet<N, M> net{}; };

template <int N, int M, int c, int C>
struct Cmed {
  static __device__ __forceinline__ void run(float (&v)[N]) {
    constexpr int i = SelOf<N, M>::net.a[c], j = SelOf<N, M>::net.b[c];
    constexpr int k = SelOf<N, M>::net.kind[c];
    if constexpr (k == 1) {
      const float x = v[i], y = v[j];
      v[i] = fminf(x, y);
      v[j] = fmaxf(x, y);
    } else if constexpr (k == 2) {
      v[i] = fminf(v[i], v[j]);
    } else {
      v[j] = fmaxf(v[i], v[j]);
    }
    Cmed<N, M, c + 1, C>::run(v);
  }
};
template <int N, int M, int C>
struct Cmed<N, M, C, C> {
  static __device__ __forceinline__ void run(float (&)[N]) {}
};

// Element M of v in sorted order (v is overwritten).
template <int N, int M>
__device__ __forceinline__ float select_net(float (&v)[N]) {
  Cmed<N, M, 0, SelOf<N, M>::net.C>::run(v);
  return v[M];
}

// Lower median of v[0..Lr): the pruned network when Lr == LN is known at
// compile time, else a full sort (v is overwritten).
template <int LN, bool EXACT>
__device__ __forceinline__ float lower_median(float (&v)[LN], int Lr) {
  if constexpr (EXACT) {
    return select_net<LN, (LN - 1) / 2>(v);
  } else {
    sort_net(v);
    const int m = (Lr - 1) >> 1;
    float r = 0;
#pragma unroll
    for (int j = 0; j < LN; j++)
      if (j == m) r = v[j];
    return r;
  }
}

__device__ __forceinline__ long long okey(double v) {
  long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

struct Slot {
  int q, B, lq;
  long off;
};

__device__ __forceinline__ Slot loop_slot(const V12Dev &d, int j) {
  const bool loc = j < d.L_loc;
  Slot s;
  s.q = loc ? d.q_loc : d.q_est;
  s.B = loc ? d.B_loc : d.B_est;
  s.lq = dlog2(s.q);
  s.off = loc ? (long)j * d.B_loc : (long)d.L_loc * d.B_loc + (long)(j - d.L_loc) * d.B_est;
  return s;
}

// bucket and window index of frequency f in loop j
// (computefourier-1.0-2.0.cc:370-378)
__device__ __forceinline__ void bucket_of(const V12Dev &d, const Slot &s, unsigned f, unsigned long long ai,
                                          int &hashed, int &m) {
  // n is a power of two below 2^32: the product's low bits suffice
  const unsigned p = (f * (unsigned)ai) & ((unsigned)d.n - 1u);
  hashed = (int)(p >> s.lq);
  int dist = (int)(p & (s.q - 1));
  if (dist > (s.q >> 1)) {
    hashed = (hashed + 1) & (s.B - 1);
    dist -= s.q;
  }
  m = dist + ((s.q - 1) >> 1);
}

// FP32 value x_samp[bucket] / filter.freq[dist] with the reference's sign
// (conjugate, computefourier-1.0-2.0.cc:383-398), via g = conj(h)/|h|^2.
// scale receives (|a| + |b|)(|g.x| + |g.y|), a bound on the terms summed.
__device__ __forceinline__ void value32(const V12Dev &d, const float2 *xs, const float2 *win_loc,
                                        const float2 *win_est, int j, unsigned f, unsigned long long ai, float &re,
                                        float &im, float &scale) {
  const Slot s = loop_slot(d, j);
  int hashed, m;
  bucket_of(d, s, f, ai, hashed, m);
  const float2 v = xs[s.off + hashed];
  const float2 g = __ldg((j < d.L_loc ? win_loc : win_est) + m);
  re = v.x * g.x + v.y * g.y;
  im = v.x * g.y - v.y * g.x;
  scale = (fabsf(v.x) + fabsf(v.y)) * (fabsf(g.x) + fabsf(g.y));
}

// a / b, correctly rounded, from y = RN(1 / b) (0: not available): a quotient
// estimate corrected to within an ulp and then by Markstein's theorem (P.
// Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990: for q within an ulp of a / b and y
// = RN(1 / b), RN(q + RN(a - b q) y) = RN(a / b), the remainder being exact).
// Five FP64 instructions instead of the IEEE division's dozen and its branch.
// b is a window's c^2 + d^2 with an exponent of +-100 (checked where y is
// formed); a's is checked here, so that no step under- or overflows.
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const unsigned e = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu;
  if (e - 223u > 1600u || __double2hiint(y) == 0) return __ddiv_rn(a, b);
  double q = __dmul_rn(a, y);
  q = __fma_rn(__fma_rn(-q, b, a), y, q);
  return __fma_rn(__fma_rn(-q, b, a), y, q);
}

// FP64 value, the reference's exact operation sequence:
// ((a c + b d) / (c^2 + d^2), (a d - b c) / (c^2 + d^2)); wp: (c, d), (c^2 +
// d^2, its reciprocal)
__device__ __forceinline__ double2 exact_value(double2 v, const double2 *wp) {
  const double2 h = __ldg(wp), den = __ldg(wp + 1);
  using A = Ar<double>;
  return make_double2(div_by(A::add(A::mul(v.x, h.x), A::mul(v.y, h.y)), den.x, den.y),
                      div_by(A::sub(A::mul(v.x, h.y), A::mul(v.y, h.x)), den.x, den.y));
}

__device__ __forceinline__ double2 value64(const V12Dev &d, const double2 *xs, int j, unsigned f,
                                           unsigned long long ai) {
  const Slot s = loop_slot(d, j);
  int hashed, m;
  bucket_of(d, s, f, ai, hashed, m);
  const double2 v = xs[s.off + hashed];
  return exact_value(v, (const double2 *)(j < d.L_loc ? d.win_loc : d.win_est) + 2 * m);
}

// Lower medians of the real and imaginary parts of the L values v of lanes 0
// .. L - 1 (the element of rank (L - 1) / 2, ties in lane order); every lane
// of the warp calls and receives them.
__device__ __forceinline__ double2 warp_median64(double2 v, int L) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, m = (L - 1) >> 1;
  const long long kx = okey(v.x), ky = okey(v.y);
  int rx = 0, ry = 0;
  for (int j = 0; j < L; j++) {
    const long long a = __shfl_sync(FULL, kx, j), b = __shfl_sync(FULL, ky, j);
    rx += a < kx || (a == kx && j < lane);
    ry += b < ky || (b == ky && j < lane);
  }
  const int sx = __ffs(__ballot_sync(FULL, lane < L && rx == m)) - 1;
  const int sy = __ffs(__ballot_sync(FULL, lane < L && ry == m)) - 1;
  return make_double2(__shfl_sync(FULL, v.x, sx), __shfl_sync(FULL, v.y, sy));
}

// The exact estimate of frequency f by one warp, one loop per lane.
__device__ __forceinline__ double2 warp_estimate64(const V12Dev &d, const double2 *xs, const int *rp, unsigned f) {
  const int lane = threadIdx.x & 31;
  double2 v = make_double2(0.0, 0.0);
  if (lane < d.L) v = value64(d, xs, lane, f, (unsigned)rp[d.L + lane]);
  return warp_median64(v, d.L);
}

// Number of candidates of a slot: v1 hits, v2 every comb candidate (or,
// in the opt-in voted mode, v2 hits).
__device__ __forceinline__ long cand_total(const V12Dev &d, int slot) {
  const int *cnt = d.counters + slot * CNT_STRIDE;
  if (d.version == 0 || d.voted) return min(cnt[CNT_HITS], d.hit_cap);
  return (long)cnt[CNT_COMB] << (dlog2((unsigned)d.n) - dlog2((unsigned)d.W));  // n / W repetitions each
}

// Frequency of candidate h (< cand_total) of a slot.  v2 candidates are
// numbered residue-major, h = residue index * (n / W) + repetition, so the
// lanes of a warp share a comb residue: for each loop their window index
// (which depends on the residue only when the window length n / B divides
// W) is one broadcast load.  The output is a set; its order is free.
__device__ __forceinline__ unsigned cand_freq(const V12Dev &d, int slot, long h) {
  if (d.version == 0 || d.voted) return (unsigned)d.hits[(long)slot * d.hit_cap + h];
  const int lw = dlog2((unsigned)d.W), lr = dlog2((unsigned)d.n) - lw;
  const unsigned hu = (unsigned)h;
  return ((hu & ((1u << lr) - 1u)) << lw) + (unsigned)d.comb_list[(long)slot * d.W + (hu >> lr)];
}

// Publishes a slot's output count (and the overflow flag).
__device__ __forceinline__ void publish_count(const V12Dev &d, int slot, long total) {
  int *cnt = d.counters + slot * CNT_STRIDE;
  const int c = (int)min(total, (long)d.out_cap);
  cnt[CNT_OUT] = c;
  if (d.out_count) d.out_count[slot] = c;
  if (total > d.out_cap) atomicOr(&cnt[CNT_ERR], ERR_OUT_OVERFLOW);
}

// Candidate h of a slot; false when h is past the end.  Thread h == 0
// publishes the count.
__device__ __forceinline__ bool candidate(const V12Dev &d, int slot, long h, unsigned &f) {
  const long total = cand_total(d, slot);
  if (h == 0) publish_count(d, slot, total);
  if (h >= total || h >= d.out_cap) return false;
  f = cand_freq(d, slot, h);
  return true;
}

// Picks the lower-median element of v[0..Lr): FP32 approximations whose
// exact values lie within +-e[j] of v[j].  Returns its index if it is
// provably the exact lower median -- exactly m = (Lr-1)/2 intervals lie
// wholly below its interval and Lr-1-m wholly above -- else -1.
// Per-element bounds matter on clean signals: most candidates' values are
// tiny, and a bound taken from the largest value of the loop set (a tone's)
// would swallow their differences.
template <int LN, bool EXACT>
__device__ __forceinline__ int proven_median(const float (&v)[LN], const float (&e)[LN], int Lr) {
  float s[LN];
#pragma unroll
  for (int j = 0; j < LN; j++) s[j] = v[j];
  const int m = (Lr - 1) >> 1;
  const float med = lower_median<LN, EXACT>(s, Lr);
  int idx = -1;
  float em = 0.f;
#pragma unroll
  for (int j = LN - 1; j >= 0; j--)
    if (j < Lr && v[j] == med) {
      idx = j;
      em = e[j];
    }
  int below = 0, above = 0;
#pragma unroll
  for (int j = 0; j < LN; j++) {
    if (j < Lr && j != idx) {
      below += (v[j] + e[j] < med - em);
      above += (v[j] - e[j] > med + em);
    }
  }
  return (below == m && above == Lr - 1 - m) ? idx : -1;
}

// Resident 128-thread blocks per SM the estimation kernels are compiled
// for (registers per thread = 65536 / (128 * blocks); some loop counts spill
// up to 32 bytes, ptxas: FP32 19, 20 and 22, FP64 from 18 on).
constexpr int est32_blocks(int LN) { return LN <= 18 ? 8 : LN <= 24 ? 6 : 5; }
constexpr int est64_blocks(int LN) { return LN <= 14 ? 6 : LN <= 20 ? 5 : 4; }

// One FP32 candidate h (< the slot's total) by random bucket lookups.
template <int LN, bool EXACT>
__device__ __forceinline__ void est32_candidate(const V12Dev &d, int slot, long h) {
  const float2 *wl = (const float2 *)d.win_loc, *we = (const float2 *)d.win_est;
  const int Lr = EXACT ? LN : d.L;
  const int *rp = d.rparams + (long)slot * d.rp_stride;
  const float2 *xs = (const float2 *)d.xs + (long)slot * d.xs_size;
  const unsigned f = cand_freq(d, slot, h);
  float re[LN], im[LN];
#pragma unroll
  for (int j = 0; j < LN; j++) {
    if (EXACT || j < Lr) {
      float sc;
      value32(d, xs, wl, we, j, f, (unsigned)rp[d.L + j], re[j], im[j], sc);
    } else {
      re[j] = INFINITY;
      im[j] = INFINITY;
    }
  }
  const float mre = lower_median<LN, EXACT>(re, Lr), mim = lower_median<LN, EXACT>(im, Lr);
  const long o = (long)slot * d.out_stride + h;
  d.out_idx[o] = (int)f;
  ((float2 *)d.out_val)[o] = make_float2(mre, mim);
}

// FP32 form of the same plans: values and medians in FP32, one candidate per
// thread.  Blocks belong to one signal each and step through its candidates;
// a queue per signal that blocks moved between cost each of them an atomic
// round trip per signal once the candidates were gone (four voted signals of
// n = 2^22, k = 500: 18.6 -> 12 us).
template <int LN, bool EXACT>
__global__ void __launch_bounds__(128, est32_blocks(LN)) k_estimate32(V12Dev d) {
  const int slot = blockIdx.y;
  const long all = cand_total(d, slot), total = min(all, (long)d.out_cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) publish_count(d, slot, all);
  for (long h = (long)blockIdx.x * 128 + threadIdx.x; h < total; h += (long)gridDim.x * 128)
    est32_candidate<LN, EXACT>(d, slot, h);
}

// FP64 form, bit-exact, of v1, voted v2 and the v2 plans without the grouped
// layout.  Few candidates (a v1 signal has about as many as tones): one warp
// each, one loop per lane -- a candidate's L divisions then cost one lane's
// chain instead of L of them, and no FP32 selection is needed.  Many: one
// thread each; the median element is chosen on FP32 copies with a rigorous
// error bound, then only that element is divided in FP64 (the reference's
// exact operation sequence); what is not provable (ties, near-ties) is done
// by the warp.  A warp's candidate holds an FP64 pipe for about 24
// instructions of 64 to 76 cycles, 0.8 us; EST64_WARP of them per
// sub-partition take as long as the other form's start-to-end latency (34 to
// 60 us).  Kernel times, one thread per candidate taken from a queue per signal
// -> now: one v1 signal of 2^13 points 60 -> 5.4 us, of 2^24 points 37 -> 8
// us; 64 signals of 2^16 points 61 -> 14 us.
constexpr int EST64_WARP = 24;

template <int LN, bool EXACT>
__global__ void __launch_bounds__(128, est64_blocks(LN)) k_estimate64(V12Dev d, int warp_max) {
  const int slot = blockIdx.y, lane = threadIdx.x & 31;
  const long all = cand_total(d, slot), total = min(all, (long)d.out_cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) publish_count(d, slot, all);
  const int *rp = d.rparams + (long)slot * d.rp_stride;
  const double2 *xs = (const double2 *)d.xs + (long)slot * d.xs_size;
  const long o = (long)slot * d.out_stride;
  if (total <= warp_max) {
    for (long h = (long)blockIdx.x * 4 + (threadIdx.x >> 5); h < total; h += (long)gridDim.x * 4) {
      const unsigned f = cand_freq(d, slot, h);
      const double2 v = warp_estimate64(d, xs, rp, f);
      if (lane == 0) {
        d.out_idx[o + h] = (int)f;
        ((double2 *)d.out_val)[o + h] = v;
      }
    }
    return;
  }
  const float2 *wl = (const float2 *)d.win32_loc, *we = (const float2 *)d.win32_est;
  const float2 *xs32 = (const float2 *)d.xs32 + (long)slot * d.xs_size;
  const int Lr = EXACT ? LN : d.L;
  for (long h0 = (long)blockIdx.x * 128; h0 < total; h0 += (long)gridDim.x * 128) {
    const long h = h0 + threadIdx.x;
    const bool live = h < total;
    const unsigned f = live ? cand_freq(d, slot, h) : 0u;
    float re[LN], im[LN], eb[LN];
#pragma unroll
    for (int j = 0; j < LN; j++) {
      if (EXACT || j < Lr) {
        float sc;
        value32(d, xs32, wl, we, j, f, (unsigned)rp[d.L + j], re[j], im[j], sc);
        // |exact - approx| <= 2^-22 * scale: each FP32 operand carries one
        // rounding (2^-24 relative), plus two products and a sum; the
        // bound below has a 4x margin, which also covers the rounding of
        // the comparisons in proven_median.
        eb[j] = sc * 0x1p-20f + 1e-30f;
      } else {
        re[j] = INFINITY;
        im[j] = INFINITY;
        eb[j] = 0.f;
      }
    }
    const int ir = proven_median<LN, EXACT>(re, eb, Lr);
    const int ii = proven_median<LN, EXACT>(im, eb, Lr);
    double2 res = make_double2(0.0, 0.0);
    const bool proven = ir >= 0 && ii >= 0;
    if (live && proven) {
      res.x = value64(d, xs, ir, f, (unsigned)rp[d.L + ir]).x;
      res.y = value64(d, xs, ii, f, (unsigned)rp[d.L + ii]).y;
    }
    for (unsigned m = __ballot_sync(0xffffffffu, live && !proven); m; m &= m - 1u) {
      const int src = __ffs(m) - 1;
      const double2 v = warp_estimate64(d, xs, rp, __shfl_sync(0xffffffffu, f, src));
      if (lane == src) {
        res = v;
        atomicAdd(&d.counters[slot * CNT_STRIDE + CNT_EXACT], 1);
      }
    }
    if (live) {
      d.out_idx[o + h] = (int)f;
      ((double2 *)d.out_val)[o + h] = res;
    }
  }
}

// ------------------------------------------- estimate by comb residue --
//
// Plain v2 estimates every comb candidate f = rep * W + r (r a comb residue,
// rep < R = n / W).  When W is a multiple of q = n / B, loop j hashes f to
//   p = f ai mod n = (r ai mod n) + W (rep ai mod R)     (mod n)
// so the window index p mod q -- and the bucket's rounding carry -- depend
// on r only, and the bucket is b = c0 + (W / q) (rep ai mod R) (mod B)
// (computefourier-1.0-2.0.cc:370-378).  ai is odd, so rep -> rep ai mod R
// is a bijection: the R candidates of a residue read R distinct buckets,
// and a group of G = R / S of them with the same rep mod S reads the G
// buckets congruent to one value mod T = B / G.  The bucket kernel stores
// each loop's buckets grouped that way (xs_perm), which makes a group's
// buckets G consecutive entries.
//
// One CTA estimates EC_THREADS candidates (whole groups): one thread per
// (group, loop) computes that pair's table entry and issues one bulk
// asynchronous copy (cp.async.bulk, completion counted in bytes on an
// mbarrier that also counts the table writers' arrivals) of the group's
// bucket run into shared memory; each thread waits on the mbarrier, then
// reads its candidate's value of every loop from shared memory -- lanes i
// of a warp read entries (rot + i ai) mod G, distinct mod 16, so without
// bank conflicts -- and takes the lower medians.  Several CTAs per SM
// overlap one CTA's copies with the others' arithmetic.  Output positions:
// residue by residue, see ec_place.

// Candidates, and threads, per CTA.  A CTA waits for its copies, then
// computes; many small CTAs an SM keep some of them computing.  32 FP32
// signals of 2^22 points, k = 100, by threads x CTAs per SM: 256 x 4 353 us,
// 128 x 8 348, 128 x 9 (56 registers) 330, 128 x 10 (48) 356, 64 x 16 384,
// 64 x 18 370; 8 FP64 signals: 256 x 4 180, 128 x 7 167, 128 x 8 166,
// 128 x 9 179, 64 x 16 171 (before ec_place interleaved their stores, which
// costs 2 and 6 us of that).  All of these are at L = 20 loops; other loop
// counts take the same shape unmeasured, and in FP64 its 64 registers spill 16
// to 190 bytes at L = 10 .. 13 and from 20 on (none at the four 256-thread
// CTAs of before).  Groups are at most this long (xs_perm_of).
constexpr int EC_THREADS = EC_GROUP_MAX;
constexpr int EC_MAXL = 32;
constexpr long EC_WAIT_POLLS = 1L << 22;

struct EcVal {   // one (group, loop): entry i of the group reads byte (rot + i ai) mod 8 G of its run
  unsigned rot;
  unsigned ai;
  float gx, gy;  // FP32 window value conj(h) / |h|^2
};

// Shared state of one item of NTH candidates (groups of G >= 32).
template <int NTH>
struct EcShared {
  EcVal v[(NTH / 32) * EC_MAXL];
  int res[NTH / 32], grp[NTH / 32];
  unsigned long long bar;
};

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_test(unsigned long long *bar, unsigned parity) {
  unsigned done;
  asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
               : "=r"(done)
               : "r"(smem_u32(bar)), "r"(parity)
               : "memory");
  return done != 0;
}

// at most EC_WAIT_POLLS polls (each may suspend the thread for a bounded time)
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long *bar, unsigned parity) {
  for (long i = 0; i < EC_WAIT_POLLS; i++)
    if (mbar_test(bar, parity)) return true;
  return false;
}

// Bulk copy global -> this CTA's shared memory, completion counted in bytes
// on `bar` (16-byte aligned addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// The output lists a residue's R candidates as if groups were of min(R, 2
// EC_GROUP_MAX): position (grp' , i') holds rep = grp' + i' S'.  Where R is
// larger than a group, two neighbouring groups interleave in one such stretch:
// unit v of a residue is the group grp = v / 2 + (v odd ? S / 2 : 0), and its
// candidate i stands at 2 i + (v odd) of the pair's places.
__device__ __forceinline__ int ec_group(unsigned v, int lr, int lg) {
  const int p = lr > lg;
  return (int)((v >> p) + ((v & (unsigned)p) << (lr - lg - p)));
}
__device__ __forceinline__ long ec_place(long hb, int i, int lr, int lg) {  // hb: first position of unit v's run
  const int p = lr > lg;
  return (hb & ~((1L << (lg + p)) - 1)) + ((i << p) | ((int)(hb >> lg) & p));
}

// Staging of candidates [h0, h0 + NTH) of a slot (total: the slot's candidate
// count, a multiple of G, so a group is wholly live or wholly past the end;
// nothing is done when h0 >= total): one thread per (group, loop) writes the group's
// table entry for that loop and issues one bulk copy of the group's run of
// FP32 bucket values (xsrc) into seg (L * NTH float2); then every thread
// waits.  Every thread of a block of NTH threads calls it.  The mbarrier in
// sh is initialised here; a caller that stages another item with the same
// sh invalidates it first, after a block barrier.  srcmw (optional)
// receives each (group, loop)'s run start and window index.  SAME_LAUNCH: the
// bucket values were stored by this launch (the caller acquired them), not by
// an earlier one.  Returns the live groups, or -1 if the wait timed out.
template <int NTH, bool SAME_LAUNCH>
__device__ __forceinline__ int ec_stage(const V12Dev &d, int slot, long h0, long total, float2 *seg,
                                        EcShared<NTH> &sh, const float2 *xsrc, const float2 *wl, const float2 *we,
                                        int2 *srcmw) {
  const int L = d.L, lg = d.xs_perm, G = 1 << lg, units = NTH >> lg;
  const int lw = dlog2((unsigned)d.W), lr = dlog2((unsigned)d.n) - lw;  // R = n / W = 2^lr repetitions
  // One thread per (group, loop).  Its loads come first and do not wait for
  // the slot's candidate count (a residue past the last one reads the list's
  // unused end), and every division is a shift: this chain -- list entry,
  // copy -- is what a CTA's arithmetic waits for (32 FP32 signals of 2^22
  // points, k = 100: 359 us before, 349 so).
  int j = 0, u = 0, src = 0, mw = 0, rot = 0, res = 0, grp = 0;
  unsigned ai = 0;
  const bool unit = threadIdx.x < units * L;
  if (unit) {
    u = threadIdx.x / L;
    j = threadIdx.x - u * L;
    const unsigned h = (unsigned)h0 + ((unsigned)u << lg), ridx = h >> lr;
    res = d.comb_list[(long)slot * d.W + min(ridx, (unsigned)d.W - 1u)];
    grp = ec_group((h & ((1u << lr) - 1u)) >> lg, lr, lg);
    ai = (unsigned)d.rparams[(long)slot * d.rp_stride + L + j];
  }
  const int live = (int)min((long)units, (total - h0) >> lg);
  if (live <= 0) return 0;
  const bool tab = unit && u < live;
  float2 g = make_float2(0.f, 0.f);
  if (tab) {
    if (j == 0) {
      sh.res[u] = res;
      sh.grp[u] = grp;
    }
    const Slot s = loop_slot(d, j);
    const unsigned mask = (unsigned)d.n - 1u;
    const unsigned p0 = ((unsigned)res * ai) & mask;
    unsigned c0 = p0 >> s.lq;
    int dist = (int)(p0 & (unsigned)(s.q - 1));
    if (dist > (s.q >> 1)) {
      c0++;
      dist -= s.q;
    }
    mw = dist + ((s.q - 1) >> 1);
    const unsigned beta = (c0 + (((unsigned)grp * ai) << (lw - s.lq))) & ((unsigned)s.B - 1u);
    const int lt = dlog2((unsigned)s.B) - lg;
    src = (int)s.off + (int)((beta & ((1u << lt) - 1u)) << lg);
    rot = (int)(beta >> lt);
    g = __ldg((j < d.L_loc ? wl : we) + mw);
  }
  // the barrier completes once the byte count is announced, every (group,
  // loop) thread has written its table entry and issued its copy (release),
  // and all copied bytes have landed
  if (threadIdx.x == 0) {
    mbar_init(&sh.bar, 1 + live * L);
    mbar_expect(&sh.bar, (unsigned)(live * L * G * sizeof(float2)));
  }
  __syncthreads();
  if (tab) {
    // the copy is issued before the window value is used, so the two loads
    // overlap (the buffer's previous contents were read through the generic
    // proxy; the bucket values of the same launch were stored through it, and
    // a copy does not follow the acquire of those without a fence of its own)
    if constexpr (SAME_LAUNCH)
      asm volatile("fence.proxy.async;" ::: "memory");
    else
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    bulk_load(seg + j * NTH + (u << lg), xsrc + (long)slot * d.xs_size + src, (unsigned)(G * sizeof(float2)),
              &sh.bar);
    sh.v[u * L + j] = EcVal{8u * (unsigned)rot, 8u * ai, g.x, g.y};
    if (srcmw) srcmw[u * L + j] = make_int2(src, mw);
    mbar_arrive(&sh.bar);
  }
  // every thread waits (bounded) on its own
  if (!mbar_wait_bounded(&sh.bar, 0)) {
    atomicOr(&d.counters[slot * CNT_STRIDE + CNT_ERR], ERR_WAIT_TIMEOUT);
    mbar_wait_bounded(&sh.bar, 0);  // copies still in flight land before the block moves on
    return -1;
  }
  return live;
}

// The staging area's start in dynamic shared memory: runs of 8 G bytes at
// multiples of 8 G, so that a run's base and an offset within it combine by OR
// (one logic operation with the modulus).
constexpr int EC_ALIGN = 8 * EC_GROUP_MAX;  // bytes of the longest run
__device__ __forceinline__ float2 *ec_area(void *dyn) {
  return (float2 *)((unsigned char *)dyn + (-smem_u32(dyn) & (EC_ALIGN - 1u)));
}

// Value of loop j (a constant after unrolling) of candidate i: base is the
// shared address of the group's run of loop 0.
template <int NTH>
__device__ __forceinline__ float2 ec_at(unsigned base, const EcVal &t, int i, unsigned mask, int j) {
  const unsigned a = (((t.rot + (unsigned)i * t.ai) & mask) | base) + (unsigned)(j * NTH * (int)sizeof(float2));
  float2 x;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x.x), "=f"(x.y) : "r"(a));
  return x;
}

// The L FP32 values of candidate i of staged group u (see ec_stage):
// x_samp[bucket] / filter.freq[dist] with the reference's sign.
template <int LN, bool EXACT, int NTH>
__device__ __forceinline__ void ec32_values(const V12Dev &d, const float2 *seg, const EcShared<NTH> &sh, int u,
                                            int i, float (&re)[LN], float (&im)[LN]) {
  const int L = d.L, lg = d.xs_perm, G = 1 << lg;
  const int Lr = EXACT ? LN : L;
  const EcVal *tv = sh.v + u * L;
  const unsigned base = smem_u32(seg + (u << lg)), mask = 8u * (unsigned)(G - 1);
#pragma unroll
  for (int j = 0; j < LN; j++) {
    if (EXACT || j < Lr) {
      const EcVal t = tv[j];
      const float2 x = ec_at<NTH>(base, t, i, mask, j);
      re[j] = x.x * t.gx + x.y * t.gy;
      im[j] = x.x * t.gy - x.y * t.gx;
    } else {
      re[j] = INFINITY;
      im[j] = INFINITY;
    }
  }
}

// Lower medians of the values and the output entry of candidate i of
// group (res, grp).
template <int LN, bool EXACT>
__device__ __forceinline__ void ec32_finish(const V12Dev &d, int slot, long h0, int res, int grp, int i,
                                            float (&re)[LN], float (&im)[LN]) {
  const int Lr = EXACT ? LN : d.L;
  const float mre = lower_median<LN, EXACT>(re, Lr), mim = lower_median<LN, EXACT>(im, Lr);
  const int lg = d.xs_perm, lw = dlog2((unsigned)d.W), lr = dlog2((unsigned)d.n) - lw, ls = lr - lg;  // S = 2^ls
  const long o = (long)slot * d.out_stride + ec_place(h0 + threadIdx.x - i, i, lr, lg);
  d.out_idx[o] = (int)((((unsigned)grp + ((unsigned)i << ls)) << lw) + (unsigned)res);
  ((float2 *)d.out_val)[o] = make_float2(mre, mim);
}

// FP32 estimates of a staged item's live groups (see ec_stage).
template <int LN, bool EXACT, int NTH>
__device__ __forceinline__ void ec32_compute(const V12Dev &d, int slot, long h0, int live, const float2 *seg,
                                             const EcShared<NTH> &sh) {
  const int lg = d.xs_perm, G = 1 << lg;
  const int u = threadIdx.x >> lg, i = threadIdx.x & (G - 1);
  if (u >= live) return;  // also after a timeout (live < 0)
  float re[LN], im[LN];
  ec32_values<LN, EXACT, NTH>(d, seg, sh, u, i, re, im);
  ec32_finish<LN, EXACT>(d, slot, h0, sh.res[u], sh.grp[u], i, re, im);
}

// One item staged, waited for and estimated in FP32.
template <int LN, bool EXACT, int NTH, bool SAME_LAUNCH = false>
__device__ __forceinline__ void ec32_block(const V12Dev &d, int slot, long h0, long total, float2 *seg,
                                           EcShared<NTH> &sh) {
  const int live = ec_stage<NTH, SAME_LAUNCH>(d, slot, h0, total, seg, sh, (const float2 *)d.xs,
                                              (const float2 *)d.win_loc, (const float2 *)d.win_est, nullptr);
  ec32_compute<LN, EXACT, NTH>(d, slot, h0, live, seg, sh);
}

// Exact FP64 value of loop j of a staged candidate: the reference's
// operation sequence on the FP64 bucket value and window.
__device__ __forceinline__ double2 ec_exact64(const V12Dev &d, const EcVal &t, int2 sm, const double2 *xs, int i,
                                             int G, int j) {
  const int idx = (int)((t.rot + (unsigned)i * t.ai) >> 3) & (G - 1);
  return exact_value(xs[sm.x + idx], (const double2 *)(j < d.L_loc ? d.win_loc : d.win_est) + 2 * sm.y);
}

// Index of the lower-median element of a component, chosen on FP32 values and
// proven, or unproven (returned in `proven`).  key[j]: the value of loop j
// with its five lowest bits replaced by j, so that the median carries its
// index and no two keys tie.  |exact value - key| <= 2^-22 s + 2^-18 |v| <=
// 1.1 2^-18 s with s = (|a| + |b|)(|g.x| + |g.y|) (each FP32 operand carries
// one rounding, plus two products and a sum; then the five bits); e = 2^-17 s
// + 1e-30 leaves room for the rounding of the test itself.  The median's
// element is proven when no other interval meets its own, |key - med| > e +
// e_med for all others: then exactly as many exact values lie below it as
// keys do.  With w = (e + e_med) - |key - med|, sum(w + |w|) over all loops
// equals the median's own term if no other w is positive (adding zeros is
// exact).  A positive w of at most 2^-24 of the median's own term may vanish in
// the sum's rounding; an overlap of the intervals that small is far within the
// part of e (0.45 of it) that the bound above leaves unused.  An infinite or
// NaN key, or an infinite e of another loop, makes the sum differ or NaN; where
// the median's own e is infinite (values near FLT_MAX, whose scale overflows
// before they do) every term is, so the own term must be finite.
// This runs on the FMA pipe; the median networks have the ALU.
constexpr float EC_ERR = 0x1p-17f;
__device__ __forceinline__ float ec_key(float v, int j) { return __int_as_float((__float_as_int(v) & ~31) | j); }
__device__ __forceinline__ float ec_scale(float2 x, const EcVal &t) {
  return __fmul_rn(__fadd_rn(fabsf(x.x), fabsf(x.y)), __fadd_rn(fabsf(t.gx), fabsf(t.gy)));
}

template <int LN, bool EXACT, int NTH>
__device__ __forceinline__ int ec_proven(const float (&key)[LN], int Lr, const EcVal *tv, unsigned base, int i,
                                         unsigned mask, bool &proven) {
  float s[LN];
#pragma unroll
  for (int j = 0; j < LN; j++) s[j] = key[j];
  const float med = lower_median<LN, EXACT>(s, Lr);
  const int idx = min(__float_as_int(med) & 31, Lr - 1);
  const float em = __fmaf_rn(ec_scale(ec_at<NTH>(base, tv[idx], i, mask, idx), tv[idx]), EC_ERR, 1e-30f);
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < LN; j++) {
    if (EXACT || j < Lr) {
      const EcVal t = tv[j];
      const float e = __fmaf_rn(ec_scale(ec_at<NTH>(base, t, i, mask, j), t), EC_ERR, em);
      const float w = __fadd_rn(e, -fabsf(__fadd_rn(key[j], -med)));
      sum = __fadd_rn(sum, __fadd_rn(w, fabsf(w)));
    }
  }
  const float own = __fmaf_rn(ec_scale(ec_at<NTH>(base, tv[idx], i, mask, idx), tv[idx]), EC_ERR, em);
  proven = sum == __fadd_rn(own, own) && own < INFINITY;
  return idx;
}

// FP64 estimates of the staged candidates, bit-exact: the lower-median
// element of each component is chosen on the staged FP32 copy and proven
// (ec_proven), then divided exactly in FP64; what is not provable is done by
// the warp, one loop per lane (by one thread it took 20 us, which a single
// signal waited for: 31 -> 10 us at one signal of 2^20 points, 310 -> 265 us
// at 8 of 2^22).  There, the proof by sums instead of counts, the corrected
// quotient instead of IEEE division and 1024 threads per SM instead of 768
// took it from 262 to 184 us, the shorter staging chain to 178.
template <int LN, bool EXACT, int NTH>
__device__ __forceinline__ void ec64_block(const V12Dev &d, int slot, long h0, long total, float2 *seg,
                                           EcShared<NTH> &sh, int2 *srcmw) {
  const int live = ec_stage<NTH, false>(d, slot, h0, total, seg, sh, (const float2 *)d.xs32,
                                        (const float2 *)d.win32_loc, (const float2 *)d.win32_est, srcmw);
  const int L = d.L, lg = d.xs_perm, G = 1 << lg;
  const int u = threadIdx.x >> lg, i = threadIdx.x & (G - 1);
  if (u >= live) return;
  const int Lr = EXACT ? LN : L;
  const EcVal *tv = sh.v + u * L;
  const int2 *sm = srcmw + u * L;
  const unsigned base = smem_u32(seg + (u << lg)), mask = 8u * (unsigned)(G - 1);
  const double2 *xs = (const double2 *)d.xs + (long)slot * d.xs_size;
  // One component at a time (fewer live registers, more resident warps).
  // The real part's exact value is computed unconditionally, at a valid
  // index, so that its loads and FP64 work overlap the imaginary part's
  // selection.
  float v[LN];
#pragma unroll
  for (int j = 0; j < LN; j++) {
    v[j] = INFINITY;
    if (EXACT || j < Lr) {
      const EcVal t = tv[j];
      const float2 x = ec_at<NTH>(base, t, i, mask, j);
      v[j] = ec_key(x.x * t.gx + x.y * t.gy, j);
    }
  }
  bool pr, pi;
  const int ir = ec_proven<LN, EXACT, NTH>(v, Lr, tv, base, i, mask, pr);
  const double xre = ec_exact64(d, tv[ir], sm[ir], xs, i, G, ir).x;
#pragma unroll
  for (int j = 0; j < LN; j++) {
    if (EXACT || j < Lr) {
      const EcVal t = tv[j];
      const float2 x = ec_at<NTH>(base, t, i, mask, j);
      v[j] = ec_key(x.x * t.gy - x.y * t.gx, j);
    }
  }
  const int ii = ec_proven<LN, EXACT, NTH>(v, Lr, tv, base, i, mask, pi);
  double2 res = make_double2(xre, 0.0);
  const bool proven = pr && pi;
  if (proven) res.y = ec_exact64(d, tv[ii], sm[ii], xs, i, G, ii).y;
  // a warp's candidates belong to one group (G >= 32): u, tv and sm are its
  for (unsigned m = __ballot_sync(0xffffffffu, !proven); m; m &= m - 1u) {
    const int src = __ffs(m) - 1, lane = threadIdx.x & 31, is = __shfl_sync(0xffffffffu, i, src);
    double2 x = make_double2(0.0, 0.0);
    if (lane < L) x = ec_exact64(d, tv[lane], sm[lane], xs, is, G, lane);
    x = warp_median64(x, L);
    if (lane == src) {
      res = x;
      atomicAdd(&d.counters[slot * CNT_STRIDE + CNT_EXACT], 1);
    }
  }
  const int lw = dlog2((unsigned)d.W), lr = dlog2((unsigned)d.n) - lw, ls = lr - lg;
  const long o = (long)slot * d.out_stride + ec_place(h0 + threadIdx.x - i, i, lr, lg);
  d.out_idx[o] = (int)((((unsigned)sh.grp[u] + ((unsigned)i << ls)) << lw) + (unsigned)sh.res[u]);
  ((double2 *)d.out_val)[o] = res;
}

__device__ __forceinline__ long ec_total(const V12Dev &d, int slot) {
  return min((long)d.counters[slot * CNT_STRIDE + CNT_COMB] << (dlog2((unsigned)d.n) - dlog2((unsigned)d.W)),
             (long)d.out_cap);
}

template <int LN, bool EXACT>
__global__ void __launch_bounds__(EC_THREADS, 9) k_estimate_comb32(V12Dev d) {
  extern __shared__ __align__(128) float2 seg[];   // [loop][EC_THREADS]
  __shared__ EcShared<EC_THREADS> sh;
  const int slot = blockIdx.y;
  if (blockIdx.x == 0 && threadIdx.x == 0) publish_count(d, slot, cand_total(d, slot));
  const long total = ec_total(d, slot), h0 = (long)blockIdx.x * EC_THREADS;
  ec32_block<LN, EXACT, EC_THREADS>(d, slot, h0, total, ec_area(seg), sh);
}

template <int LN, bool EXACT>
__global__ void __launch_bounds__(EC_THREADS, 8) k_estimate_comb64(V12Dev d) {
  extern __shared__ __align__(128) float2 seg64[];   // [loop][EC_THREADS]
  __shared__ EcShared<EC_THREADS> sh;
  __shared__ int2 srcmw[(EC_THREADS / 32) * EC_MAXL];
  const int slot = blockIdx.y;
  if (blockIdx.x == 0 && threadIdx.x == 0) publish_count(d, slot, cand_total(d, slot));
  const long total = ec_total(d, slot), h0 = (long)blockIdx.x * EC_THREADS;
  ec64_block<LN, EXACT, EC_THREADS>(d, slot, h0, total, ec_area(seg64), sh, srcmw);
}

// ---------------------------------------------------------------- scatter --

// 16 stores of 16 bytes per thread: 64 KB a block.
constexpr int CLEAR_PER = 16;

__global__ void __launch_bounds__(256) k_clear_dense(void *const *dense, int n) {
  double2 *o = (double2 *)dense[blockIdx.y];
  const long i0 = (long)blockIdx.x * (256 * CLEAR_PER) + threadIdx.x;
#pragma unroll
  for (int u = 0; u < CLEAR_PER; u++)
    if (i0 + 256 * u < n) __stcs(o + i0 + 256 * u, make_double2(0.0, 0.0));  // L2 stays the transform's
}

template <typename R>
__global__ void k_scatter_dense(const int *out_idx, const c2_t<R> *out_val, const int *counters,
                                int out_cap, void *const *dense) {
  const int slot = blockIdx.y;
  const long h = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int cnt = counters[slot * CNT_STRIDE + CNT_OUT];
  if (h >= cnt) return;
  const long o = (long)slot * out_cap + h;
  const c2_t<R> v = out_val[o];
  ((double2 *)dense[slot])[out_idx[o]] = make_double2((double)v.x, (double)v.y);
}

// ---------------------------------------------------------------- launch --

int v12_max_fft(int prec) { return prec == PREC_FP64 ? 8192 : 16384; }

// Butterflies per thread and radix-4 stage of an FP64 one-CTA FFT.
static int one_cta_per(int N) { return std::max(1, N / 4 / 1024); }

// Threads of a selection over N keys: eight per thread, more beyond 8192 keys.
static int select_threads(int N) { return std::min(1024, std::max(128, N / 8)); }

template <typename R, typename In>
static cudaError_t launch_comb(const V12Dev &d, int nslots, cudaStream_t s) {
  cudaError_t e;
  if (d.comb_pw) {
    const int W = d.W, m2 = fft_m2(W);
    const FftShape f = fft_shape2(W, W, sizeof(c2_t<R>));
    const size_t sa = sizeof(c2_t<R>) * f.elems[0], sb = sizeof(c2_t<R>) * f.elems[1];
    if ((e = set_smem(k_comb_a<R, In>, sa)) || (e = set_smem(k_comb_b<R>, sb))) return e;
    k_comb_a<R, In><<<dim3(fft_ctas(f.elems[0], W / m2, W), d.comb_loops, nslots), f.elems[0] / 4, sa, s>>>(
        d, f.elems[0]);
    k_comb_b<R><<<dim3(fft_ctas(f.elems[1], m2, W), d.comb_loops, nslots), f.elems[1] / 4, sb, s>>>(d, f.elems[1]);
    const dim3 grid(d.comb_loops, nslots);
    const int T = select_threads(W);
    if (W <= 8 * 1024)
      k_comb_select<R, 8><<<grid, T, 0, s>>>(d);
    else if (W <= 16 * 1024)
      k_comb_select<R, 16><<<grid, T, 0, s>>>(d);
    else
      k_comb_select<R, 0><<<grid, T, 0, s>>>(d);
    note_launches(3);
    return cudaGetLastError();
  }
  const int T = OneCta<R>::threads(d.W);
  const size_t sm = OneCta<R>::bytes(d.W);
  dim3 grid(d.comb_loops, nslots);
#define SFFT_COMB(P)                                             \
  case P:                                                        \
    if ((e = set_smem(k_comb<R, P, In>, sm))) return e;          \
    k_comb<R, P, In><<<grid, T, sm, s>>>(d);                     \
    break;
  if constexpr (sizeof(R) == 4) {
    switch (1) { SFFT_COMB(1) }
  } else {
    switch (one_cta_per(d.W)) {
      SFFT_COMB(1)
      SFFT_COMB(2)
      default:
        return cudaErrorInvalidValue;
    }
  }
#undef SFFT_COMB
  note_launches(1);
  return cudaGetLastError();
}

template <typename R>
static cudaError_t launch_bucket(const V12Dev &d, int nslots, cudaStream_t s) {
  cudaError_t e;
  const int Bmax = d.B_loc > d.B_est ? d.B_loc : d.B_est;
  if (d.pw) {
    const FftShape f = fft_shape2(d.B_loc, d.B_est, sizeof(c2_t<R>));
    const size_t sa = sizeof(c2_t<R>) * f.elems[0], sb = sizeof(c2_t<R>) * f.elems[1];
    if ((e = set_smem(k_bucket_a<R>, sa)) || (e = set_smem(k_bucket_b<R>, sb))) return e;
    const int ml = fft_m2(d.B_loc), me = fft_m2(d.B_est);
    const int al = fft_ctas(f.elems[0], d.B_loc / ml, d.B_loc), ae = fft_ctas(f.elems[0], d.B_est / me, d.B_est);
    const int bl = fft_ctas(f.elems[1], ml, d.B_loc), be = fft_ctas(f.elems[1], me, d.B_est);
    k_bucket_a<R><<<dim3(d.L_loc * al + d.L_est * ae, nslots), f.elems[0] / 4, sa, s>>>(d, f.elems[0], al, ae);
    k_bucket_b<R><<<dim3(d.L_loc * bl + d.L_est * be, nslots), f.elems[1] / 4, sb, s>>>(d, f.elems[1], bl, be);
    const dim3 grid(d.L, nslots);
    const int T = select_threads(Bmax);
    if (Bmax <= 8 * 1024)
      k_bucket_select<R, 8><<<grid, T, 0, s>>>(d);
    else if (Bmax <= 16 * 1024)
      k_bucket_select<R, 16><<<grid, T, 0, s>>>(d);
    else
      k_bucket_select<R, 0><<<grid, T, 0, s>>>(d);
    note_launches(2);  // the third is counted with the stage kernels
    return cudaGetLastError();
  }
  const int T = OneCta<R>::threads(Bmax);
  const size_t sm = OneCta<R>::bytes(Bmax);
  dim3 grid(d.L, nslots);
#define SFFT_BUCKET(P)                                        \
  case P:                                                     \
    if ((e = set_smem(k_bucket<R, P>, sm))) return e;         \
    k_bucket<R, P><<<grid, T, sm, s>>>(d);                    \
    break;
  if constexpr (sizeof(R) == 4) {
    switch (1) { SFFT_BUCKET(1) }
  } else {
    switch (one_cta_per(Bmax)) {
      SFFT_BUCKET(1)
      SFFT_BUCKET(2)
      default:
        return cudaErrorInvalidValue;
    }
  }
#undef SFFT_BUCKET
  return cudaGetLastError();
}

template <int LN, bool EX>
struct k_estimate32_k {
  static cudaError_t go(int nslots, cudaStream_t s, const V12Dev &d, int nsm) {
    const int most = std::max(1, nsm * est32_blocks(LN) / nslots);
    const int blocks = (int)std::min<long>(most, ((long)d.out_cap + 127) / 128);
    k_estimate32<LN, EX><<<dim3(std::max(1, blocks), nslots), 128, 0, s>>>(d);
    return cudaSuccess;
  }
};
template <int LN, bool EX>
struct k_estimate64_k {
  static cudaError_t go(int nslots, cudaStream_t s, const V12Dev &d, int nsm) {
    // blocks of four warps: the resident ones shared out over the slots, at
    // most one warp per candidate
    const int most = std::max(1, nsm * est64_blocks(LN) / nslots);
    const int blocks = (int)std::min<long>(most, ((long)d.out_cap + 3) / 4);
    k_estimate64<LN, EX><<<dim3(std::max(1, blocks), nslots), 128, 0, s>>>(d, EST64_WARP * 4 * nsm / nslots);
    return cudaSuccess;
  }
};

template <template <int, bool> class KS>
static cudaError_t dispatch_estimate(const V12Dev &d, int nslots, int nsm, cudaStream_t s) {
  cudaError_t e;
  switch (d.L) {
#define SFFT_L(v)                                             \
  case v:                                                     \
    if ((e = KS<v, true>::go(nslots, s, d, nsm))) return e; \
    break;
    SFFT_L(8) SFFT_L(9) SFFT_L(10) SFFT_L(11) SFFT_L(12) SFFT_L(13) SFFT_L(14) SFFT_L(15) SFFT_L(16)
    SFFT_L(17) SFFT_L(18) SFFT_L(19) SFFT_L(20) SFFT_L(21) SFFT_L(22) SFFT_L(23) SFFT_L(24)
#undef SFFT_L
    default:
      if (d.L > 32) return cudaErrorInvalidValue;
      if ((e = KS<32, false>::go(nslots, s, d, nsm))) return e;
  }
  return cudaGetLastError();
}

// Multiprocessor count of the current device (cached per device).
static int sm_count() {
  static int cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
  if (!cache[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 152;
    cache[dev] = v;
  }
  return cache[dev];
}

// Estimation by comb residue (xs_perm set, FP32): one CTA per EC_THREADS
// candidates, up to min(W, comb_loops * 2k) residues of n / W candidates.
template <int LN, bool EX>
struct EcK32 {
  static cudaError_t go(int nslots, cudaStream_t s, const V12Dev &d, int) {
    const long cmax = std::min<long>(d.W, (long)d.comb_loops * d.num);
    const long cands = std::min<long>(cmax * (d.n / d.W), (long)d.out_cap);
    const size_t sm = sizeof(float2) * EC_THREADS * d.L + EC_ALIGN;
    cudaError_t e;
    if ((e = set_smem(k_estimate_comb32<LN, EX>, sm))) return e;
    dim3 g((unsigned)((cands + EC_THREADS - 1) / EC_THREADS), nslots);
    k_estimate_comb32<LN, EX><<<g, EC_THREADS, sm, s>>>(d);
    return cudaSuccess;
  }
};

template <int LN, bool EX>
struct EcK64 {
  static cudaError_t go(int nslots, cudaStream_t s, const V12Dev &d, int) {
    const long cmax = std::min<long>(d.W, (long)d.comb_loops * d.num);
    const long cands = std::min<long>(cmax * (d.n / d.W), (long)d.out_cap);
    const size_t sm = sizeof(float2) * EC_THREADS * d.L + EC_ALIGN;
    cudaError_t e;
    if ((e = set_smem(k_estimate_comb64<LN, EX>, sm))) return e;
    dim3 g((unsigned)((cands + EC_THREADS - 1) / EC_THREADS), nslots);
    k_estimate_comb64<LN, EX><<<g, EC_THREADS, sm, s>>>(d);
    return cudaSuccess;
  }
};

template <typename R>
static cudaError_t launch_estimate(const V12Dev &d, int nslots, cudaStream_t s) {
  if (sizeof(R) == 4 && d.xs_perm) return dispatch_estimate<EcK32>(d, nslots, 0, s);
  if (sizeof(R) == 8 && d.xs_perm) return dispatch_estimate<EcK64>(d, nslots, 0, s);
  if (sizeof(R) == 8) return dispatch_estimate<k_estimate64_k>(d, nslots, sm_count(), s);
  return dispatch_estimate<k_estimate32_k>(d, nslots, sm_count(), s);
}

template <typename R, typename In>
static cudaError_t run_typed(const V12Dev &d, int nslots, cudaStream_t s, StageEvents *se, cudaEvent_t input_read) {
  cudaError_t e;
  mark(se, s);
  if (d.version == 1) {
    if ((e = launch_comb<R, In>(d, nslots, s))) return e;
  }
  mark(se, s);
  if (sizeof(R) == 4) {
    constexpr int S = 4;
    dim3 fg((unsigned)((d.xs_size * S + 255) / 256), nslots);
    k_fold_split<In, S><<<fg, 256, 0, s>>>(d);
  } else {
    // FP64: a bucket's taps are one chain of instructions that each hold an
    // FP64 pipe, so few buckets go out in blocks of two warps, over as many
    // SMs as there are; from four warps to a pipe on the block's size decides
    // nothing (one signal of 2^13 points 17.5 us in blocks of eight warps, 12.0 in
    // blocks of two; of 2^20 points 19.4 and 13.9)
    const int T = d.xs_size * nslots <= (long)sm_count() * 4 * 4 * 32 ? 64 : 256;
    dim3 fg((unsigned)((d.xs_size + T - 1) / T), nslots);
    k_fold<R, In><<<fg, T, 0, s>>>(d);
  }
  if ((e = cudaGetLastError())) return e;
  mark(se, s);
  if (input_read && (e = cudaEventRecord(input_read, s))) return e;
  if ((e = launch_bucket<R>(d, nslots, s))) return e;
  {
    const size_t sm = vote_smem(d);
    const long residues = d.version ? std::min<long>(d.W, (long)d.comb_loops * d.num) : 0;
    const long cands = d.version ? residues * (d.n / d.W) : 0;
    if (d.version == 0) {
      const int blocks = (int)(((long)d.num * d.q_loc + 256 * VOTE_V - 1) / (256 * VOTE_V));
      k_vote_ranges<<<dim3((unsigned)(blocks * d.L_loc), nslots), 256, sm, s>>>(d, blocks);
    } else if (vote_by_residue(d)) {
      k_vote_residue<<<dim3((unsigned)residues, nslots), 256, d.n / d.W, s>>>(d);
    } else if (cands * nslots >= (long)sm_count() * 4 * 8 * 256) {
      // eight candidates per thread where that still gives every SM four blocks
      k_vote_cands<8><<<dim3((unsigned)((cands + 2047) / 2048), nslots), 256, sm, s>>>(d);
    } else {
      k_vote_cands<1><<<dim3((unsigned)((cands + 255) / 256), nslots), 256, sm, s>>>(d);
    }
    if ((e = cudaGetLastError())) return e;
    note_launches(1);
  }
  mark(se, s);
  if ((e = launch_estimate<R>(d, nslots, s))) return e;
  mark(se, s);
  note_launches(3);
  return cudaSuccess;
}

// ------------------------------------------------- persistent executor --
//
// sfft_exec_many over plans of different (n, k) as one kernel launch.  Each
// CTA (PT threads, one per SM) takes items from a global queue in list
// order.  An item is one block's worth of one stage of one signal -- a comb
// sampling, a chunk of the fold, the comb residue list, one loop's bucket
// FFT and selection, a chunk of the voting, a chunk of the estimation --
// and runs the same device code as the stage kernels.  Before it starts, its
// CTA waits (bounded) until the signal's counters show the stages it reads
// complete; after it ends, the CTA bumps the counter of its own stage.  The
// list is ordered so that every item's dependencies come earlier: a CTA only
// waits for items that CTAs already took, and those wait only for earlier
// items, so the queue always progresses, whatever the number of resident
// CTAs.  A wait that runs out flags the signal (ERR_WAIT_TIMEOUT) and the
// item is skipped, so the kernel always ends.

constexpr int PT = 1024;                 // threads of the executor's CTA
constexpr int PERSIST_VOTES = 8;         // candidates per thread of a voting item
constexpr long PERSIST_POLLS = 1L << 24;  // polls of a dependency (with back-off)

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits until *p >= target.  Bounded; gives up at once when another wait of
// the run has already run out (*abort), so a fault costs one time limit.
__device__ __forceinline__ bool persist_wait(const int *p, int target, int *abort) {
  for (long i = 0; i < PERSIST_POLLS; i++) {
    if (ld_acquire(p) >= target) return true;
    if ((i & 255) == 255 && *(volatile int *)abort) return false;
    __nanosleep(64);
  }
  atomicExch(abort, 1);
  return false;
}

__device__ __forceinline__ void mbar_inval(unsigned long long *bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <int LN, bool EX>
__device__ __forceinline__ void persist_est(const V12Dev &d, const PersistGroup &g, int slot, int idx, float2 *seg,
                                            EcShared<PT> &ecsh) {
  if (g.est_comb) {
    const long total = ec_total(d, slot), h0 = (long)idx * PT;
    if (h0 < total) ec32_block<LN, EX, PT, true>(d, slot, h0, total, seg, ecsh);
    __syncthreads();  // the item's mbarrier is no longer read
    if (threadIdx.x == 0 && h0 < total) mbar_inval(&ecsh.bar);
  } else {
    const long total = min(cand_total(d, slot), (long)d.out_cap);
    for (int c = 0; c < g.est_chunks; c++) {
      const long h = ((long)idx * g.est_chunks + c) * PT + threadIdx.x;
      if (h < total) est32_candidate<LN, EX>(d, slot, h);
    }
  }
}

__device__ __noinline__ void persist_est_any(const V12Dev &d, const PersistGroup &g, int slot, int idx, float2 *seg,
                                             EcShared<PT> &ecsh) {
  switch (d.L) {
#define SFFT_PL(v)                                       \
  case v:                                                \
    persist_est<v, true>(d, g, slot, idx, seg, ecsh);    \
    break;
    SFFT_PL(8) SFFT_PL(9) SFFT_PL(10) SFFT_PL(11) SFFT_PL(12) SFFT_PL(13) SFFT_PL(14) SFFT_PL(15) SFFT_PL(16)
    SFFT_PL(17) SFFT_PL(18) SFFT_PL(19) SFFT_PL(20) SFFT_PL(21) SFFT_PL(22) SFFT_PL(23) SFFT_PL(24)
#undef SFFT_PL
    default:
      persist_est<32, false>(d, g, slot, idx, seg, ecsh);
  }
}

template <typename In>
__global__ void __launch_bounds__(PT, 1) k_persist32(PersistProg p) {
  extern __shared__ __align__(128) unsigned char psmem[];
  __shared__ PersistGroup sg;      // the plan of the current item
  __shared__ EcShared<PT> ecsh;
  __shared__ SelShared<unsigned> ss;
  __shared__ VoteHits hits;
  __shared__ PersistItem sitem;
  __shared__ int s_ok;
  int *head = p.state, *abort = p.state + 1, *dep = p.state + 2;
  int cached = -1;
  for (;;) {
    if (threadIdx.x == 0) {
      const int it = atomicAdd(head, 1);
      sitem = it < p.nitems ? p.items[it] : PersistItem{-1, -1, 0, 0};
    }
    __syncthreads();
    const PersistItem w = sitem;
    if (w.kind < 0) break;
    if (w.group != cached) {
      const int *src = (const int *)(p.groups + w.group);
      int *dst = (int *)&sg;
      for (int i = threadIdx.x; i < (int)(sizeof(PersistGroup) / sizeof(int)); i += PT) dst[i] = src[i];
      cached = w.group;
      __syncthreads();
    }
    const V12Dev &d = sg.d;
    int *sdep = dep + 4 * (sg.gslot0 + w.slot);
    if (threadIdx.x == 0) {
      bool ok = !*(volatile int *)abort;
      if (ok && w.kind == PK_LIST)
        ok = persist_wait(sdep + 0, d.comb_loops, abort);
      else if (ok && w.kind == PK_BUCKET)
        ok = persist_wait(sdep + 1, sg.nfold, abort);
      else if (ok && (w.kind == PK_VOTE || w.kind == PK_EST))
        ok = persist_wait(sdep + 2, d.L, abort) && persist_wait(sdep + 3, 1, abort);
      if (!ok) atomicOr(&d.counters[w.slot * CNT_STRIDE + CNT_ERR], ERR_WAIT_TIMEOUT);
      s_ok = ok;
    }
    __syncthreads();
    if (s_ok) {
      switch (w.kind) {
        case PK_COMB:
          comb_block<float, 1, In>(d, w.idx, w.slot, psmem, ss);
          break;
        case PK_FOLD:
          for (int c = 0; c < sg.fold_chunks; c++)
            fold_split_thread<In, 4>(d, w.slot, ((long)w.idx * sg.fold_chunks + c) * PT + threadIdx.x);
          break;
        case PK_LIST:
          comb_list_block(d, w.slot);
          break;
        case PK_BUCKET:
          bucket_block<float, 1>(d, w.idx, w.slot, psmem, ss);
          break;
        case PK_VOTE:
          vote_cands<PERSIST_VOTES>(d, w.slot, (long)w.idx * PT * PERSIST_VOTES, vote_bits(d, w.slot, (unsigned *)psmem),
                                    hits);
          break;
        default:  // PK_EST
          if (w.idx == 0 && threadIdx.x == 0) publish_count(d, w.slot, cand_total(d, w.slot));
          persist_est_any(d, sg, w.slot, w.idx, ec_area(psmem), ecsh);
      }
    }
    __syncthreads();  // the item's writes precede its completion count
    if (threadIdx.x == 0) {
      const int k = w.kind == PK_COMB ? 0 : w.kind == PK_FOLD ? 1 : w.kind == PK_BUCKET ? 2 : w.kind == PK_LIST ? 3 : -1;
      if (k >= 0) {
        __threadfence();
        atomicAdd(sdep + k, 1);
      }
    }
  }
}

bool persist_eligible(const V12Dev &d) {
  const int mx = v12_max_fft(PREC_FP32);
  return d.version == 1 && !d.voted && d.prec == PREC_FP32 && !d.large_buckets && !d.large_comb && d.L <= 32 &&
         d.W >= 32 && d.W <= mx && d.B_loc <= mx && d.B_est <= mx && d.comb_loops <= 64;
}

void persist_shape(PersistGroup &g) {
  V12Dev &d = g.d;
  if (d.xs_perm && d.L > 24) d.xs_perm = 0;  // the comb-residue items hold L x PT values in shared memory
  g.fold_chunks = 8;
  g.nfold = (int)((d.xs_size * 4 + (long)PT * g.fold_chunks - 1) / ((long)PT * g.fold_chunks));
  const long cands = std::min<long>(std::min<long>(d.W, (long)d.comb_loops * d.num) * (d.n / d.W), (long)d.out_cap);
  g.nvote = (int)((cands + (long)PT * PERSIST_VOTES - 1) / ((long)PT * PERSIST_VOTES));
  g.est_comb = d.xs_perm != 0;
  g.est_chunks = g.est_comb ? 1 : 4;
  g.nest = (int)((cands + (long)PT * g.est_chunks - 1) / ((long)PT * g.est_chunks));
}

size_t persist_smem(const PersistGroup *groups, int ngroups) {
  size_t m = 0;
  for (int i = 0; i < ngroups; i++) {
    const V12Dev &d = groups[i].d;
    m = std::max(m, OneCta<float>::bytes(std::max(d.W, std::max(d.B_loc, d.B_est))));
    m = std::max(m, vote_smem(d));
    if (groups[i].est_comb) m = std::max(m, sizeof(float2) * (size_t)PT * d.L + EC_ALIGN);
  }
  return m;
}

// The queue order comes from a simulation of the executor on `workers`
// CTAs: every item gets a rough duration, becomes ready when the stages it
// reads are complete, and a free CTA takes the ready item of the
// highest-ranked signal (signals ranked by decreasing work), later stages
// first.  The items in simulated start order form the queue: an item starts
// only after its dependencies finished, so they precede it in the queue,
// and the order keeps CTAs off dependency waits as far as the durations
// are right.
void persist_items(const PersistGroup *groups, int ngroups, std::vector<PersistItem> &items, int workers) {
  struct Sig {
    int g, s;
    double work;
  };
  std::vector<Sig> sigs;
  for (int g = 0; g < ngroups; g++)
    for (int s = 0; s < groups[g].slots; s++)
      sigs.push_back({g, s, (double)groups[g].d.xs_size * groups[g].d.L + (double)groups[g].nest * PT});
  std::stable_sort(sigs.begin(), sigs.end(), [](const Sig &a, const Sig &b) { return a.work > b.work; });
  // durations (microseconds of one CTA, rough)
  auto dur = [&](const PersistGroup &G, int kind) -> double {
    const V12Dev &d = G.d;
    switch (kind) {
      case PK_COMB: return 2.0 + d.W / 2048.0;
      case PK_FOLD: {
        const double taps = (double)PT * G.fold_chunks / 4.0 * ((double)d.w_loc / d.B_loc + (double)d.w_est / d.B_est) / 2;
        return 1.0 + taps / 700.0;
      }
      case PK_LIST: return 1.0;
      case PK_BUCKET: return 2.0 + std::max(d.B_loc, d.B_est) / 2048.0;
      case PK_VOTE: return 1.0 + (double)PERSIST_VOTES * d.L_loc / 8.0;
      default: return 1.0 + (double)PT * G.est_chunks * d.L / 4000.0;
    }
  };
  const int nsig = (int)sigs.size();
  // per signal: items per stage, remaining counts, completion times
  struct St {
    int comb_left, fold_left, bucket_left, list_left;
    double comb_done, fold_done, bucket_done, list_done;
    bool list_q, bucket_q, tail_q;
  };
  std::vector<St> st(nsig);
  struct Ready {
    double t;
    int rank, kind, idx;
  };
  // ready items: ordered by (rank, later kind first, idx) among those ready by now
  auto cmp = [](const Ready &a, const Ready &b) {
    if (a.rank != b.rank) return a.rank > b.rank;
    if (a.kind != b.kind) return a.kind < b.kind;
    return a.idx > b.idx;
  };
  std::priority_queue<Ready, std::vector<Ready>, decltype(cmp)> ready(cmp);
  auto later = [](const Ready &a, const Ready &b) { return a.t > b.t; };
  std::priority_queue<Ready, std::vector<Ready>, decltype(later)> pending(later);  // not ready yet
  for (int r = 0; r < nsig; r++) {
    const PersistGroup &G = groups[sigs[r].g];
    st[r] = {G.d.comb_loops, G.nfold, G.d.L, 1, 0, 0, 0, 0, false, false, false};
    for (int c = 0; c < G.d.comb_loops; c++) ready.push({0.0, r, PK_COMB, c});
    for (int i = 0; i < G.nfold; i++) ready.push({0.0, r, PK_FOLD, i});
  }
  std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
  for (int w = 0; w < std::max(1, workers); w++) free_at.push(0.0);
  items.clear();
  auto release = [&](int r, double t) {  // newly ready stages of signal r at time t
    St &x = st[r];
    const PersistGroup &G = groups[sigs[r].g];
    if (!x.list_q && x.comb_left == 0) {
      x.list_q = true;
      pending.push({t, r, PK_LIST, 0});
    }
    if (!x.bucket_q && x.fold_left == 0) {
      x.bucket_q = true;
      for (int j = 0; j < G.d.L; j++) pending.push({t, r, PK_BUCKET, j});
    }
    if (!x.tail_q && x.bucket_left == 0 && x.list_left == 0) {
      x.tail_q = true;
      for (int i = 0; i < G.nvote; i++) pending.push({t, r, PK_VOTE, i});
      for (int i = 0; i < G.nest; i++) pending.push({t, r, PK_EST, i});
    }
  };
  while (!ready.empty() || !pending.empty()) {
    double t = free_at.top();
    free_at.pop();
    while (!pending.empty() && pending.top().t <= t) {
      ready.push(pending.top());
      pending.pop();
    }
    if (ready.empty()) {  // idle until the next item becomes ready
      t = pending.top().t;
      while (!pending.empty() && pending.top().t <= t) {
        ready.push(pending.top());
        pending.pop();
      }
    }
    const Ready it = ready.top();
    ready.pop();
    const int g = sigs[it.rank].g, sl = sigs[it.rank].s;
    const double end = t + dur(groups[g], it.kind);
    items.push_back({it.kind, g, sl, it.idx});
    free_at.push(end);
    St &x = st[it.rank];
    // completion bookkeeping (dependents become ready when the last item of a stage ends)
    if (it.kind == PK_COMB) {
      x.comb_done = std::max(x.comb_done, end);
      if (--x.comb_left == 0) release(it.rank, x.comb_done);
    } else if (it.kind == PK_FOLD) {
      x.fold_done = std::max(x.fold_done, end);
      if (--x.fold_left == 0) release(it.rank, x.fold_done);
    } else if (it.kind == PK_BUCKET) {
      x.bucket_done = std::max(x.bucket_done, end);
      if (--x.bucket_left == 0) release(it.rank, std::max(x.bucket_done, x.list_done));
    } else if (it.kind == PK_LIST) {
      x.list_done = end;
      if (--x.list_left == 0) release(it.rank, std::max(x.bucket_done, x.list_done));
    }
  }
}

cudaError_t persist_run(const PersistProg &p, cudaStream_t s) {
  cudaError_t e;
  if ((e = cudaMemsetAsync(p.state, 0, sizeof(int) * (2 + 4 * (size_t)p.nslots_total), s))) return e;
  const int grid = sm_count();
  // always opted in: with the kernel's static shared memory, 32-48 KB of
  // dynamic shared memory would exceed the default limit
  const size_t sm = std::max<size_t>(p.smem, 40 * 1024);
  if (p.in_type == IN_C128) {
    if ((e = set_smem(k_persist32<double2>, sm))) return e;
    k_persist32<double2><<<grid, PT, sm, s>>>(p);
  } else {
    if ((e = set_smem(k_persist32<float2>, sm))) return e;
    k_persist32<float2><<<grid, PT, sm, s>>>(p);
  }
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t global_fft_c128(void *a, void *b, int N, int narr, long arr_stride, long slot_stride, int nslots,
                            const void *tw, cudaStream_t s) {
  return global_fft<double>((double2 *)a, (double2 *)b, N, narr, arr_stride, slot_stride, nslots, (const double2 *)tw,
                            s);
}

cudaError_t v12_run(const V12Dev &d, int nslots, cudaStream_t s, StageEvents *se, cudaEvent_t input_read) {
  if (d.prec == PREC_FP64)
    return d.in_type == IN_C128 ? run_typed<double, double2>(d, nslots, s, se, input_read)
                                : run_typed<double, float2>(d, nslots, s, se, input_read);
  return d.in_type == IN_C128 ? run_typed<float, double2>(d, nslots, s, se, input_read)
                              : run_typed<float, float2>(d, nslots, s, se, input_read);
}

// ------------------------------------------------------------------ setup --

// The draws and input pointers of a launch captured in a graph, read from
// page-locked host memory when the graph runs, and the cleared counters: one
// node where two copies and a memset were three (24 uneven signals, 15
// branches: 340 -> 321 us a pass).  A direct launch keeps the copies: with its
// draws as kernel arguments it was no faster (four voted signals of n = 2^22,
// k = 500: 207 -> 210 us).
__global__ void __launch_bounds__(256) k_setup_staged(const int *h_rp, const void *const *h_in, int nrp, int *rp, int nin,
                                                      const void **in, int ncnt, int *cnt) {
  for (int i = threadIdx.x; i < nrp; i += 256) rp[i] = h_rp[i];
  for (int i = threadIdx.x; i < nin; i += 256) in[i] = h_in[i];
  for (int i = threadIdx.x; i < ncnt; i += 256) cnt[i] = 0;
}

// From pageable memory, which the runtime stages before it returns.
cudaError_t setup_slots(const int *h_rp, int rp_stride, const void *const *h_in, int num, int *rp, const void **in,
                        int *cnt, cudaStream_t s) {
  cudaError_t e;
  if ((e = cudaMemcpyAsync(rp, h_rp, sizeof(int) * (size_t)rp_stride * num, cudaMemcpyHostToDevice, s)) ||
      (e = cudaMemcpyAsync(in, h_in, sizeof(void *) * (size_t)num, cudaMemcpyHostToDevice, s)))
    return e;
  return cnt ? cudaMemsetAsync(cnt, 0, sizeof(int) * CNT_STRIDE * (size_t)num, s) : cudaSuccess;
}

cudaError_t setup_slots_staged(const int *h_rp, int rp_stride, const void *const *h_in, int num, int *rp,
                               const void **in, int *cnt, cudaStream_t s) {
  k_setup_staged<<<1, 256, 0, s>>>(h_rp, h_in, rp_stride * num, rp, num, in, CNT_STRIDE * num, cnt);
  note_launches(1);
  return cudaGetLastError();
}

__global__ void k_copy_ints(const int *src, int *dst, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) dst[i] = src[i];
}

cudaError_t copy_ints(const int *src, int *dst, int count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  k_copy_ints<<<(count + 255) / 256, 256, 0, s>>>(src, dst, count);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t clear_dense(void *const *dense, int n, int nslots, cudaStream_t s) {
  k_clear_dense<<<dim3((unsigned)((n + 256L * CLEAR_PER - 1) / (256L * CLEAR_PER)), nslots), 256, 0, s>>>(dense, n);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t scatter_dense(const int *out_idx, const void *out_val, int prec, const int *counters,
                          int out_cap, void *const *dense, int nslots, cudaStream_t s) {
  dim3 grid((out_cap + 255) / 256, nslots);
  if (prec == PREC_FP64)
    k_scatter_dense<double><<<grid, 256, 0, s>>>(out_idx, (const double2 *)out_val, counters, out_cap, dense);
  else
    k_scatter_dense<float><<<grid, 256, 0, s>>>(out_idx, (const float2 *)out_val, counters, out_cap, dense);
  note_launches(1);
  return cudaGetLastError();
}

}  // namespace sfft

namespace {

template <int N>
int copy_median_network(int *dst, long cap) {
  constexpr const sfft::SelNet<N, (N - 1) / 2> &net = sfft::SelOf<N, (N - 1) / 2>::net;
  if (!dst || cap < 3L * net.C) return -1;
  for (int c = 0; c < net.C; c++) {
    dst[3 * c] = net.a[c];
    dst[3 * c + 1] = net.b[c];
    dst[3 * c + 2] = net.kind[c];
  }
  return net.C;
}

}  // namespace

extern "C" int sfft_debug_median_network(int n, int *dst, long cap) {
  switch (n) {
#define SFFT_MN(v) \
  case v:          \
    return copy_median_network<v>(dst, cap);
    SFFT_MN(8) SFFT_MN(9) SFFT_MN(10) SFFT_MN(11) SFFT_MN(12) SFFT_MN(13) SFFT_MN(14) SFFT_MN(15) SFFT_MN(16)
    SFFT_MN(17) SFFT_MN(18) SFFT_MN(19) SFFT_MN(20) SFFT_MN(21) SFFT_MN(22) SFFT_MN(23) SFFT_MN(24)
#undef SFFT_MN
    default:
      return -1;
  }
}
