// v3.cu — the sFFT v3 ("exactly sparse") exec path on GB300.
//
//   k_v3_first   the first half of the Mansour comb FFTs on the gathered
//                samples (computefourier-3.0.cc:96-127), and the folds of the
//                contiguous (:130-212) and the permuted (:215-297) Gaussian
//                filter, each for both time shifts.
//   k_v3_second  the second half of the Mansour FFTs and the Gaussian bucket
//                FFTs.
//   k_v3_peel    one thread-block cluster (8 or 16 CTAs) per signal runs
//                alternate_fft's estimate / peel rounds (:784-1088):
//                bucket estimation spread over the cluster, subtraction of
//                recovered tones with FP64 atomics, and the bucket-count
//                fixpoint test, with a bounded number of rounds.
// The result map is a per-signal open-addressing table in global memory.
// FP64 throughout: the phase-slope frequency decode needs phase accuracy
// below pi/n.  On GB300 a warp's FP64 instruction holds its sub-partition's
// FP64 pipe for 64 to 76 cycles, with one lane active or 32, so these kernels
// take about as long as their longest chain of FP64 instructions: folds and
// FFTs are spread over many CTAs, and the phases go through integer
// arithmetic and a table (phase.cuh).
#include <cooperative_groups.h>

#include "common.cuh"
#include "engine.h"
#include "fft.cuh"
#include "phase.cuh"

namespace cg = cooperative_groups;

namespace sfft {

static constexpr double kPi = 3.14159265358979323846;

__device__ __forceinline__ double2 ld_x(const void *base, int in_type, long i) {
  if (in_type == IN_C128) return __ldg((const double2 *)base + i);
  const float2 v = __ldg((const float2 *)base + i);
  return make_double2((double)v.x, (double)v.y);
}

// True if a component's magnitude is at least 2^e: a bucket none of whose
// components is, is known to be empty without any FP64 instruction.
__device__ __forceinline__ bool reaches(double2 v, int e) {
  const int a = __double2hiint(v.x) & 0x7fffffff, b = __double2hiint(v.y) & 0x7fffffff;
  return max(a, b) >= ((1023 + e) << 20);
}

__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {  // a b + c
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}

// --------------------------------------------------------------- filters --

int v3_max_smem_fft() { return 8192; }

// The filters of one signal of n = 2^24, k = 1000: 103 us with a CTA per role
// (96 k cycles for the contiguous Gaussian's alone), 22 us spread like this.
//
// Work of k_v3_first per signal, in CTAs of V3_T threads: Mansour tiles of
// both shifts, groups of buckets of the two Gaussian folds (both shifts, each
// bucket's taps over several lanes), and blocks of the result table to clear.
constexpr int V3_T = 128;
constexpr int V3_S1 = 4, V3_S2 = 8;            // lanes per bucket and shift of the two folds
constexpr int V3_G1 = V3_T / (2 * V3_S1);      // buckets per CTA
constexpr int V3_G2 = V3_T / (2 * V3_S2);
constexpr int V3_CLEAR = 16 * 4 * V3_T;        // table entries cleared per CTA

struct V3Shape {
  int elems[2];    // Mansour tile entries of the two launches
  int man[2];      // Mansour CTAs per shift of the two launches
  int n1, n2, nc;  // Gaussian fold CTAs, table-clearing CTAs
  int chunks2;
};

// Buckets [b0, b0 + G) of one Gaussian filter, both shifts: thread = ((bucket
// - b0) * 2 + shift) * S + part; part p takes taps p, p + S, ... of its bucket.
template <int G, int S, typename Val>
__device__ __forceinline__ void v3_fold(int b0, int B, int chunks, const double2 *taps, double2 *dst, Val val) {
  const int part = threadIdx.x % S, o = threadIdx.x / S, l = o & 1, b = b0 + (o >> 1);
  double2 acc = make_double2(0.0, 0.0);
  if (b < B) {
#pragma unroll 4
    for (int c = part; c < chunks; c += S) acc = cfma(val(b - b0, c, l), __ldg(taps + (long)c * B + b), acc);
  }
#pragma unroll
  for (int s = S / 2; s > 0; s >>= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, s);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, s);
  }
  if (b < B && part == 0) dst[2 * b + l] = acc;
}

__global__ void __launch_bounds__(V3_T) k_v3_first(V3Dev d, V3Shape sh) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int slot = blockIdx.y;
  int x = blockIdx.x;
  const int *rp = d.rparams + (long)slot * d.rp_stride;
  const unsigned mask = (unsigned)d.n - 1u;
  const void *in = d.inputs[slot];
  const int in_type = d.in_type;
  if (x == 0 && threadIdx.x < CNT_STRIDE) d.counters[slot * CNT_STRIDE + threadIdx.x] = 0;
  if (x < 2 * sh.man[0]) {  // Mansour: x[(init_offset + l + i * n/W) mod n]
    const int l = x / sh.man[0], tile = x - l * sh.man[0], W = d.W;
    const int M = W / fft_m2(W), lc = fft_lc(sh.elems[0], M, W);
    const unsigned sigma = (unsigned)(d.n / W), o = (unsigned)(rp[3] + l);
    double2 *dst = (double2 *)d.man_tmp + ((long)slot * 2 + l) * W;
    fft_tile<double>((double2 *)smem_raw, M, lc, 1, W, tile << lc, floor_log2(W) & 1, (const double2 *)d.tw_man,
                     [=](int i) { return ld_x(in, in_type, (long)((o + (unsigned)i * sigma) & mask)); },
                     [=](int i, double2 v) { dst[i] = v; });
    return;
  }
  x -= 2 * sh.man[0];
  if (x < sh.n1) {  // Gaussian 1: taps over x[init_G_offset + l + t]
    const int b0 = x * V3_G1, B = d.B1;
    const unsigned base = (unsigned)rp[4];
    v3_fold<V3_G1, V3_S1>(b0, B, d.w1 / B, (const double2 *)d.taps1, (double2 *)d.g1 + (long)slot * 2 * B,
                          [=](int b, int c, int l) {
                            return ld_x(in, in_type, (long)((base + (unsigned)(c * B + b0 + b + l)) & mask));
                          });
    return;
  }
  x -= sh.n1;
  if (x < sh.n2) {
    // Gaussian 2 on permuted, phase-shifted samples.  permute_fourier
    // (computefourier-3.0.cc:66-87): sample i is x[(ig + i*ai) mod n] *
    // shift_i with shift_0 = e^{2 pi i ig b / n} and shift_{i+1} = shift_i *
    // e^{2 pi i ai b / n}, a running product.  The two angles are formed as
    // there (the same FP64 products); shift_i = e^{i (a0 + i a1)} directly,
    // one sample per thread -- replaying the product serially costs about 64
    // cycles per operation (2945 steps at n = 2^24, k = 1000: 0.58 ms).  Its
    // error, about 3e-16, is below the serial chain's accumulated rounding
    // (about i * 2^-53) and far inside the 1e-10 value tolerance.
    const int b0 = x * V3_G2, B = d.B2, chunks = sh.chunks2, G = min(V3_G2, B - b0);
    const unsigned ig = (unsigned)rp[4], ai = (unsigned)rp[1];
    const int bb = rp[2];
    const double a0 = 2 * kPi * rp[4] * bb / d.n, a1 = 2 * kPi * rp[1] * bb / d.n;
    const double2 *trig = (const double2 *)d.trig;
    double2 *P = (double2 *)smem_raw;  // [chunk][G + 1]: the shifts use samples b and b + 1
    for (int t = threadIdx.x; t < chunks * (V3_G2 + 1); t += V3_T) {
      const int c = t / (V3_G2 + 1), k = t - c * (V3_G2 + 1);
      if (k > G) continue;
      const int i = c * B + b0 + k;
      P[t] = cfma(ld_x(in, in_type, (long)((ig + (unsigned)i * ai) & mask)), cis_step(trig, a0, i, a1),
                  make_double2(0.0, 0.0));
    }
    __syncthreads();
    v3_fold<V3_G2, V3_S2>(b0, B, chunks, (const double2 *)d.taps2, (double2 *)d.g2 + (long)slot * 2 * B,
                          [=](int b, int c, int l) { return P[c * (V3_G2 + 1) + b + l]; });
    return;
  }
  x -= sh.n2;
  int4 *keys = (int4 *)(d.map_keys + (long)slot * d.table_cap) + (long)x * (V3_CLEAR / 4);
  for (int t = threadIdx.x; t < V3_CLEAR / 4 && (long)x * V3_CLEAR + 4 * t < d.table_cap; t += V3_T)
    keys[t] = make_int4(-1, -1, -1, -1);
}

// blockDim.x >= V3_T: a quarter of the longest Gaussian bucket FFT (at most
// 1024, PER butterflies per thread).
template <int PER>
__global__ void __launch_bounds__(1024) k_v3_second(V3Dev d, V3Shape sh) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int slot = blockIdx.y;
  int x = blockIdx.x;
  if (x < 2 * sh.man[1]) {
    const int l = x / sh.man[1], tile = x - l * sh.man[1], W = d.W, M = fft_m2(W), lc = fft_lc(sh.elems[1], M, W);
    const double2 *src = (const double2 *)d.man_tmp + ((long)slot * 2 + l) * W;
    double2 *dst = (double2 *)d.man + (long)slot * 2 * W;
    fft_tile<double>((double2 *)smem_raw, M, lc, W / M, W, tile << lc, false, (const double2 *)d.tw_man,
                     [=](int i) { return src[i]; }, [=](int i, double2 v) { dst[2 * i + l] = v; });
    return;
  }
  x -= 2 * sh.man[1];
  const int l = x & 1, B = x < 2 ? d.B1 : d.B2;
  double2 *buf = (double2 *)smem_raw, *g = (x < 2 ? (double2 *)d.g1 : (double2 *)d.g2) + (long)slot * 2 * B;
  for (int i = threadIdx.x; i < B; i += blockDim.x) buf[i] = g[2 * i + l];
  __syncthreads();
  block_fft<double, PER>(buf, B, floor_log2(B), (const double2 *)(x < 2 ? d.tw_g1 : d.tw_g2));
  for (int i = threadIdx.x; i < B; i += blockDim.x) g[2 * i + l] = buf[i];
}

// ------------------------------------------------------------------ peel --
//
// A request's rounds run each piece of this kernel a few times, so its time
// is latency: chains of FP64 instructions (about 100 from a bucket's values
// to the subtraction of its tone), L2 round trips and cluster barriers.  What
// was taken out of the chains, with the kernel's time for one signal of n =
// 2^24, k = 1000 (6 or 9 rounds, by the signal) and for 16 of n = 2^18, k = 100: library atan2 /
// sincos and 8 CTAs 202 / 208 us; table phases and 16 CTAs 148 / 168; no
// divisions for constants in every warp (8 warps a sub-partition, 64 cycles
// an instruction) and lists by exponent 104 / 114; tones peeled by the CTA
// that found them, from shared memory, and the barrier after reading the
// buckets split around the estimates' arithmetic 83 / 101.

// State of a signal's rounds, the same for every thread of a CTA (shared
// memory).
struct PeelCtx {
  V3Dev d;
  int n1, lw, a, ai, b, io, ig, aG, shift, tmask, rank, nb;
  double2 *man, *g1, *g2;
  int *tkey;
  double2 *tval;
  int *list;
  int *est_f;
  double2 *est_v;
  int *counters;
  double slope[2], off[2];  // 2 pi ig / n and 2 pi a ig / n; the comb offsets io and io + 1
  // counters of the cluster (the first CTA's shared memory)
  int *count, *err;
  double2 trig[1 << TRIG_BITS];  // V3Dev::trig: a cluster barrier drops what L1 holds
};

__device__ __forceinline__ double2 win_at(const double2 *win, int half, int n, int dist, int *err) {
  int ds = dist >= (n >> 1) ? dist - n : dist;
  if (ds < -half || ds > half) {
    atomicOr(err, ERR_V3_CAP);
    ds = ds < -half ? -half : half;
  }
  return __ldg(win + ds + half);
}

__device__ __forceinline__ int wrapmul(int x, int y) { return (int)((unsigned)x * (unsigned)y); }

// Subtraction of a recovered tone from one filter's buckets of one shift:
// part = 2 * filter + shift, filter 0 the permuted Gaussian, 1 the
// contiguous Gaussian (the three nearest buckets, computefourier-3.0.cc:
// 354-463), 2 the Mansour comb (:300-351).  The six parts of a tone are
// independent (atomic subtractions), so they are separate work items: their
// FP64 chains run on different sub-partitions.
__device__ __forceinline__ void update_part(const PeelCtx &c, int key, double2 v, int part) {
  const V3Dev &d = c.d;
  const int l = part & 1;
  const double2 zero = make_double2(0.0, 0.0);
  if (part < 4) {
    const bool perm = part < 2;
    const int B = perm ? d.B2 : d.B1, half = perm ? d.win2_half : d.win1_half;
    const double2 *win = (const double2 *)(perm ? d.win2 : d.win1);
    double2 *samp = perm ? c.g2 : c.g1;
    const unsigned f = perm ? ((unsigned)key * (unsigned)c.ai + (unsigned)c.shift) & (unsigned)c.n1 : (unsigned)key;
    const int lq = d.logn - floor_log2(B);
    const unsigned q = 1u << lq;
    const int h = (int)(((f + (q >> 1)) >> lq) & (unsigned)(B - 1));  // (int)(f / q + 0.5)
    const unsigned dist = (unsigned)h * q - f;
    // shift l: time offset `offset` + l; the phase 2 pi ko / n is the integer
    // ko mod n of n-ths of a turn
    const unsigned ko = (f * ((unsigned)(perm ? c.aG : c.ig) + (unsigned)l)) & (unsigned)c.n1;
    const double2 vl = cfma(v, cis_turn(c.trig, (unsigned long long)ko << (64 - d.logn)), zero);
#pragma unroll 1
    for (int qd = -1; qd < 2; qd++) {
      const double2 r = cfma(vl, win_at(win, half, d.n, (int)((dist + (unsigned)qd * q) & (unsigned)c.n1), c.err), zero);
      double *p = (double *)&samp[2 * ((h + qd) & (B - 1)) + l];
      atomicAdd(p, -r.x);
      atomicAdd(p + 1, -r.y);
    }
  } else {
    const double2 r = cfma(v, cis(c.trig, d.pi2_over_n * key * c.off[l]), zero);
    double *p = (double *)&c.man[2 * (key & (d.W - 1)) + l];
    atomicAdd(p, -(d.w_dbl * r.x));
    atomicAdd(p + 1, -(d.w_dbl * r.y));
  }
}

// Result map: key -> accumulated value; returns nothing, keys of one round
// are distinct so the value update has a single writer.
__device__ __forceinline__ void map_add(const PeelCtx &c, int key, double2 v, bool assign) {
  unsigned h = ((unsigned)key * 2654435761u) & (unsigned)c.tmask;
  for (int probe = 0; probe <= c.tmask; probe++) {
    const int cur = atomicCAS(&c.tkey[h], -1, key);
    if (cur == -1) {
      const int idx = atomicAdd(c.count, 1);
      if (idx < c.d.map_cap)
        c.list[idx] = (int)h;
      else
        atomicOr(c.err, ERR_V3_CAP);
      c.tval[h] = v;
      return;
    }
    if (cur == key) {
      if (assign) {
        c.tval[h] = v;
      } else {
        double2 o = c.tval[h];
        c.tval[h] = make_double2(o.x + v.x, o.y + v.y);
      }
      return;
    }
    h = (h + 1) & (unsigned)c.tmask;
  }
  atomicOr(c.err, ERR_V3_CAP);
}

// The estimation loops below visit every bucket, but FP64 work is done only
// on listed ones: a warp's FP64 instruction occupies its SM sub-partition's
// FP64 pipe for 64 cycles and more whether one lane or 32 are active.  So each
// CTA lists the buckets that are not empty by their exponents alone, deals
// the list out one per lane over warps of all four sub-partitions, keeps the
// entries that pass the reference's tests in a second list, and deals those
// out again: an item per angle and one per magnitude, then one per value.
constexpr int V3_LIST = 1024;  // list entries per CTA and pass (= threads per CTA)

// Position in the list of thread `tid` of a 1024-thread CTA: consecutive
// entries go to consecutive sub-partitions (warp mod 4), then lanes.
__device__ __forceinline__ int v3_spread(int tid) {
  return ((tid >> 7) << 7) | ((tid & 31) << 2) | ((tid >> 5) & 3);
}

// Per-CTA shared scratch of the estimation loops, and the tones that the CTA
// found in the current phase (beyond V3_LIST in est_f / est_v).
struct EstScratch {
  int raw[V3_LIST], list[V3_LIST], key[V3_LIST];
  int nraw, cnt, tones;
  double c0[V3_LIST], ang[2 * V3_LIST], mag[V3_LIST];
  double2 s[2 * V3_LIST], val[V3_LIST];
};

__device__ __forceinline__ void tone_put(const PeelCtx &c, EstScratch &x, int key, double2 v) {
  const int i = atomicAdd(&x.tones, 1);
  if (i < V3_LIST) {
    x.key[i] = key;
    x.val[i] = v;
  } else {
    c.est_f[i - V3_LIST] = key;
    c.est_v[i - V3_LIST] = v;
  }
}
__device__ __forceinline__ int tone_key(const PeelCtx &c, const EstScratch &x, int i) {
  return i < V3_LIST ? x.key[i] : c.est_f[i - V3_LIST];
}
__device__ __forceinline__ double2 tone_val(const PeelCtx &c, const EstScratch &x, int i) {
  return i < V3_LIST ? x.val[i] : c.est_v[i - V3_LIST];
}

// Finds this CTA's tones of one filter.  stage 0: estimate_freq_mansour_loops2
// (computefourier-3.0.cc:642-776) on the comb; 1, 2:
// estimate_freq_gauss_loops2 (:484-640) on the contiguous and the permuted
// Gaussian buckets.  Every thread of the CTA calls it.  The cluster barrier's
// first half (arrive) comes once the CTA has read its last bucket; the caller
// waits for the second half before it changes any bucket.
__device__ __noinline__ void estimate(const PeelCtx &c, int stage, EstScratch &x) {
  const V3Dev &d = c.d;
  const int gt = v3_spread(threadIdx.x) * c.nb + c.rank, T = V3_LIST * c.nb, t = v3_spread(threadIdx.x);
  const bool comb = stage == 0, perm = stage == 2;
  const double2 *s = comb ? c.man : perm ? c.g2 : c.g1;
  const int B = comb ? d.W : perm ? d.B2 : d.B1, lw = comb ? c.lw : 0;
  const double norm2 = comb ? d.inv_w2 : 1.0, tol = comb ? d.tol_man : d.tol_gauss;
  const unsigned n1 = (unsigned)c.n1;
  if (threadIdx.x == 0) x.tones = 0;
#pragma unroll 1
  for (int base = 0; base < B; base += T) {
    // not empty: c0 + c1 > 1e-8 needs a component of at least 5e-5
    if (threadIdx.x == 0) x.nraw = x.cnt = 0;
    __syncthreads();
    const int bk0 = base + gt;
    if (bk0 < B && (reaches(s[2 * bk0], lw - 15) || reaches(s[2 * bk0 + 1], lw - 15)))
      x.raw[atomicAdd(&x.nraw, 1)] = bk0;
    __syncthreads();
    // c0 + c1 > 1e-8, c0 > 0.01 and |c1 / c0 - 1| < tol (without the square,
    // which overflows where c0 does not)
    if (t < x.nraw) {
      const int bk = x.raw[t];
      const double2 s0 = s[2 * bk], s1 = s[2 * bk + 1];
      const double c0 = fma(s0.x, s0.x, s0.y * s0.y) * norm2, c1 = fma(s1.x, s1.x, s1.y * s1.y) * norm2;
      if (c0 + c1 > 1e-8 && c0 > 0.01 && fabs(c1 - c0) < tol * c0) {
        const int i = atomicAdd(&x.cnt, 1);
        x.list[i] = bk;
        x.c0[i] = c0;
        x.s[2 * i] = s0;
        x.s[2 * i + 1] = s1;
      }
    }
    __syncthreads();
    if (base + T >= B) cg::this_cluster().barrier_arrive();
    const int cnt = x.cnt, m0 = (2 * cnt + 127) & ~127;  // magnitudes in warps of their own
#pragma unroll 1
    for (int w = t; w < m0 + cnt; w += V3_LIST) {
      if (w < 2 * cnt)
        x.ang[w] = angle_of(c.trig, x.s[w].y, x.s[w].x);  // the scale does not change the angle
      else if (w >= m0)
        x.mag[w - m0] = sqrt_of(x.c0[w - m0]);
    }
    __syncthreads();
#pragma unroll 1
    for (int e = t; e < cnt; e += V3_LIST) {
      const double d0 = x.ang[2 * e], ab = x.mag[e];
      const int fr = (int)__double2ll_rn((x.ang[2 * e + 1] - d0) * d.n_over_pi2);
      const int bk = x.list[e];
      unsigned freq, dist = 0;
      double ph;
      if (comb) {
        freq = ((unsigned)fr & n1 & ~((unsigned)B - 1u)) | (unsigned)bk;
        ph = d0 - d.pi2_over_n * wrapmul((int)freq, c.io);
      } else {
        freq = (unsigned)(fr + d.n) & n1;
        const int lq = d.logn - floor_log2(B);
        const unsigned q = 1u << lq, down = freq >> lq, rest = 2u * (freq & (q - 1u));
        // freq / q rounded to nearest, ties to even
        const unsigned hashed = (down + (rest > q || (rest == q && (down & 1u)))) & ((unsigned)B - 1u);
        if (hashed != (unsigned)bk) continue;
        dist = (hashed * q - freq) & n1;
        ph = d0 - c.slope[perm] * (int)freq;
      }
      // the window's value is asked for before the phase is worked out
      const double2 f = comb ? make_double2(1.0, 0.0)
                             : win_at((const double2 *)(perm ? d.win2 : d.win1), perm ? d.win2_half : d.win1_half, d.n,
                                      (int)dist, c.err);
      const double2 w = cis(c.trig, ph);
      double2 v = make_double2(ab * w.x, ab * w.y);
      if (!comb) {  // divided by the window
        const double den = fma(f.x, f.x, f.y * f.y), inv = recip_of(den);
        const double2 num = make_double2(fma(v.x, f.x, v.y * f.y), fma(v.y, f.x, -(v.x * f.y)));
        const double2 q0 = make_double2(num.x * inv, num.y * inv);  // corrected by the remainders
        v = make_double2(fma(fma(-q0.x, den, num.x), inv, q0.x), fma(fma(-q0.y, den, num.y), inv, q0.y));
        if (perm) freq = (freq * (unsigned)c.a - (unsigned)c.b) & n1;
      }
      tone_put(c, x, (int)freq, v);
    }
    __syncthreads();  // the tones are complete, and the lists free for the next pass
  }
}

__device__ __forceinline__ void trace_rec(const PeelCtx &c, int round, int stage, int key, double2 v) {
  if (!c.d.trace) return;
  const int i = atomicAdd(&c.counters[CNT_TRACE], 1);
  if (i < c.d.trace_cap) {
    double *t = c.d.trace + 5 * (long)i;
    t[0] = round;
    t[1] = stage;
    t[2] = key;
    t[3] = v.x;
    t[4] = v.y;
  }
}

// Peels parts p0 .. p0 + np of `mine` tones: the CTA's estimates, or (known)
// the entries rank, rank + nb, ... of the result map.  A warp takes one part
// of 32 tones, so the two forms of update_part do not meet in a warp; new
// estimates go to the map (add: to what it holds, else in its place) as a
// part of their own.
__device__ __noinline__ void subtract(const PeelCtx &c, const EstScratch &x, int mine, int p0, int np, bool known,
                                      bool to_map, bool assign, int round, int stage) {
  const int parts = np + (to_map ? 1 : 0), warps = parts * ((mine + 31) >> 5);
#pragma unroll 1
  for (int u = threadIdx.x >> 5; u < warps; u += V3_LIST / 32) {
    const int part = u % parts, i = (u / parts) * 32 + (threadIdx.x & 31);
    if (i >= mine) continue;
    const int h = known ? c.list[i * c.nb + c.rank] : 0;
    const int key = known ? c.tkey[h] : tone_key(c, x, i);
    const double2 v = known ? c.tval[h] : tone_val(c, x, i);
    if (part < np) {
      update_part(c, key, v, p0 + part);
    } else {
      trace_rec(c, round, stage, key, v);
      map_add(c, key, v, assign);
    }
  }
}

// One thread-block cluster (8 or 16 CTAs) per signal runs the estimate /
// peel rounds: every loop over buckets, estimates and map entries is spread
// over the cluster's threads, and each block-wide barrier of the round
// structure is a cluster barrier (release / acquire at cluster scope, so the
// global-memory bucket arrays and the map written before it are visible
// after it).  The round's counters live in the shared memory of the
// cluster's first CTA and are updated through distributed shared memory; a
// counter that a check adds to was cleared by the one before, so clearing
// needs no barrier of its own.  A CTA peels the tones it found itself, from its
// own shared memory: no estimate crosses L2, and the barrier between reading
// the buckets and changing them runs beside the estimates' arithmetic.
// Control flow is uniform across the cluster: every branch is taken on values
// read after a barrier.
struct PeelShared {
  int found, count, err, cnt[2][3];
};

struct PeelMem {
  PeelCtx c;
  PeelShared sh;
  EstScratch x;
};

__global__ void __launch_bounds__(V3_LIST) k_v3_peel(V3Dev dev) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PeelMem &mem = *(PeelMem *)smem_raw;
  PeelCtx &c = mem.c;
  PeelShared &sh_local = mem.sh;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), nb = (int)cl.num_blocks();
  PeelShared *S = cl.map_shared_rank(&sh_local, 0);
  const int slot = blockIdx.x / nb;
  const int *rp = dev.rparams + (long)slot * dev.rp_stride;
  if (rank == 0 && threadIdx.x < sizeof(PeelShared) / sizeof(int)) ((int *)&sh_local)[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    c.d = dev;
    if (slot) c.d.trace = nullptr;
    c.n1 = dev.n - 1;
    c.lw = floor_log2(dev.W);
    c.man = (double2 *)dev.man + (long)slot * 2 * dev.W;
    c.g1 = (double2 *)dev.g1 + (long)slot * 2 * dev.B1;
    c.g2 = (double2 *)dev.g2 + (long)slot * 2 * dev.B2;
    c.tkey = dev.map_keys + (long)slot * dev.table_cap;
    c.tval = (double2 *)dev.map_vals + (long)slot * dev.table_cap;
    c.list = dev.map_table + (long)slot * dev.map_cap;
    c.tmask = dev.table_cap - 1;
    // this CTA's share of the spill arrays.  Bucket counts and nb are powers of
    // two: of B buckets it visits at most V3_LIST, all in shared memory, or
    // B / nb, the first V3_LIST of whose tones are
    const long share = dev.est_cap / nb;
    c.est_f = dev.est_f + (long)slot * dev.est_cap + rank * share;
    c.est_v = (double2 *)dev.est_v + (long)slot * dev.est_cap + rank * share;
    c.counters = dev.counters + slot * CNT_STRIDE;
    c.a = rp[0];
    c.ai = rp[1];
    c.b = rp[2];
    c.io = rp[3];
    c.ig = rp[4];
    c.aG = wrapmul(c.a, c.ig);
    c.shift = ((wrapmul(c.ai, c.b) % dev.n) + dev.n) % dev.n;
    c.rank = rank;
    c.nb = nb;
    c.count = &S->count;
    c.err = &S->err;
  }
  if (threadIdx.x >= 32 && threadIdx.x < 34) {
    // the reference's products; n is a power of two: times 1 / n equals the quotient
    const int i = threadIdx.x - 32;
    c.slope[i] = 2 * kPi * (i ? rp[0] : 1) * rp[4] * dev.inv_n;
    c.off[i] = (double)(rp[3] + i);
  }
  for (int i = threadIdx.x; i < (1 << TRIG_BITS); i += V3_LIST) c.trig[i] = __ldg((const double2 *)dev.trig + i);
  const int T = V3_LIST * nb, gt = v3_spread(threadIdx.x) * nb + rank;
  const bool lead = rank == 0 && threadIdx.x == 0;
  cl.sync();

  // ---- Mansour estimate; first tones are assigned, their buckets cleared
  estimate(c, 0, mem.x);
  const int first = mem.x.tones;  // the CTA's
  if (threadIdx.x == 0 && first) atomicAdd(&S->found, first);
  cl.barrier_wait();
  for (int i = threadIdx.x; i < first; i += V3_LIST) {
    const int bk = tone_key(c, mem.x, i) & (dev.W - 1);
    c.man[2 * bk] = make_double2(0.0, 0.0);
    c.man[2 * bk + 1] = make_double2(0.0, 0.0);
  }
  // ---- first Gaussian filter: peel the known tones, estimate, peel
  subtract(c, mem.x, first, 2, 2, false, true, true, -2, 0);
  cl.sync();
  if (S->found == dev.k) {  // the reference returns before writing its output (:859-860)
    if (lead) {
      c.counters[CNT_OUT] = 0;
      if (dev.out_count) dev.out_count[slot] = 0;
      c.counters[CNT_V3] = -1;
    }
    cl.sync();     // the first CTA's shared memory outlives every reader
    return;
  }
  estimate(c, 1, mem.x);
  cl.barrier_wait();
  subtract(c, mem.x, mem.x.tones, 2, 4, false, true, false, -1, 1);
  cl.sync();

  // ---- second (permuted) Gaussian filter: peel every known tone
  subtract(c, mem.x, (min(S->count, dev.map_cap) - rank + nb - 1) / nb, 0, 2, true, false, false, 0, 0);
  cl.sync();

  // ---- round robin: G2, then Mansour, G1, G2, ... until the counts of
  //      non-empty buckets repeat after a G2 round (:959-1076)
  int stage = 2, rounds = 0, checks = 0, prev[3] = {0, 0, 0};
  for (;;) {
    estimate(c, stage, mem.x);
    cl.barrier_wait();
    subtract(c, mem.x, mem.x.tones, 0, 6, false, true, false, rounds, stage);
    cl.sync();
    if (stage == 2 && rounds >= 1) {
      int *cn = S->cnt[checks & 1];
      if (lead) {
        int *other = S->cnt[~checks & 1];
        other[0] = other[1] = other[2] = 0;
      }
      checks++;
#pragma unroll 1
      for (int i = 0; i < 3; i++) {  // comb, contiguous, permuted
        const double2 *s = i == 0 ? c.man : i == 1 ? c.g1 : c.g2;
        const int B = i == 0 ? dev.W : i == 1 ? dev.B1 : dev.B2, st = i == 0 ? 2 : 1;
        const double norm2 = i == 0 ? dev.inv_w2 : 1.0;  // W is a power of two: exact scaling
        int k = 0;
        for (int j = gt; j < B; j += T) {
          const double2 v = s[st * j];
          // |v|^2 > 1e-6 needs a component of at least 7e-4
          if (reaches(v, (i == 0 ? c.lw : 0) - 11)) k += ((v.x * v.x + v.y * v.y) * norm2 > 1e-6);
        }
        if (k) atomicAdd(&cn[i], k);
      }
      cl.sync();
      bool same = true;
      for (int i = 0; i < 3; i++) {
        const int v = cn[i];
        same = same && v == prev[i];
        prev[i] = v;
      }
      if (same) break;
    }
    rounds++;
    if (rounds > dev.max_passes) {
      if (lead) atomicOr(&S->err, ERR_V3_NOCONVERGE);
      break;
    }
    stage = (stage + 1) % 3;
  }
  cl.sync();

  // ---- output: every key of the map with its accumulated value
  const int M = min(S->count, dev.map_cap), outn = min(M, dev.out_cap);
  for (int i = gt; i < outn; i += T) {
    const int h = c.list[i];
    dev.out_idx[(long)slot * dev.out_stride + i] = c.tkey[h];
    ((double2 *)dev.out_val)[(long)slot * dev.out_stride + i] = c.tval[h];
  }
  if (lead) {
    c.counters[CNT_OUT] = outn;
    if (dev.out_count) dev.out_count[slot] = outn;
    c.counters[CNT_V3] = rounds;
    c.counters[CNT_ERR] |= S->err | (M > dev.out_cap ? ERR_OUT_OVERFLOW : 0);
  }
  cl.sync();       // the first CTA's shared memory outlives every reader
}

// ---------------------------------------------------------------- launch --

// CTAs per cluster of the peel kernel: 16 (beyond the portable 8, so only
// where the device says that it can hold such clusters) for few signals,
// whose rounds then have twice the FP64 pipes; 8 once 16 would leave signals
// waiting for one another.
static cudaError_t v3_cluster(int nslots, int &nb) {
  static std::mutex mu;
  static std::map<int, int> held;  // device -> clusters of 16 at once
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e) return e;
  std::lock_guard<std::mutex> g(mu);
  auto it = held.find(dev);
  if (it == held.end()) {
    int n = 0;
    if ((e = set_smem(k_v3_peel, sizeof(PeelMem)))) return e;
    if (cudaFuncSetAttribute(k_v3_peel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 16;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(16);
      cfg.blockDim = dim3(V3_LIST);
      cfg.dynamicSmemBytes = sizeof(PeelMem);
      cfg.attrs = at;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&n, k_v3_peel, &cfg) != cudaSuccess) n = 0;
    }
    cudaGetLastError();
    it = held.emplace(dev, n).first;
  }
  nb = nslots <= it->second / 2 ? 16 : 8;
  return cudaSuccess;
}

static cudaError_t v3_peel(const V3Dev &d, int nslots, cudaStream_t s) {
  int nb = 8;
  cudaError_t e = v3_cluster(nslots, nb);
  if (e) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = nb;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(nslots * nb);
  cfg.blockDim = dim3(V3_LIST);
  cfg.dynamicSmemBytes = sizeof(PeelMem);
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_v3_peel, d);
}

cudaError_t v3_run(const V3Dev &d, int nslots, cudaStream_t s, StageEvents *se, cudaEvent_t input_read) {
  cudaError_t e;
  mark(se, s);
  const int Bmax = std::max(d.B1, d.B2), m2 = fft_m2(d.W);
  V3Shape sh;
  sh.elems[0] = sh.elems[1] = 4 * V3_T;  // W is at most 2^17: tiles of up to 512 rows
  if (d.W / m2 > sh.elems[0] || m2 > sh.elems[1]) return cudaErrorInvalidValue;
  sh.man[0] = fft_ctas(sh.elems[0], d.W / m2, d.W);
  sh.man[1] = fft_ctas(sh.elems[1], m2, d.W);
  sh.n1 = (d.B1 + V3_G1 - 1) / V3_G1;
  sh.n2 = (d.B2 + V3_G2 - 1) / V3_G2;
  sh.nc = (d.table_cap + V3_CLEAR - 1) / V3_CLEAR;
  sh.chunks2 = d.w2 / d.B2;
  const size_t tile = sizeof(double2) * (size_t)sh.elems[0];
  const size_t sa = std::max(tile, sizeof(double2) * (size_t)sh.chunks2 * (V3_G2 + 1));
  const size_t sb = std::max(tile, sizeof(double2) * (size_t)Bmax);
  if ((e = set_smem(k_v3_first, sa))) return e;
  k_v3_first<<<dim3(2 * sh.man[0] + sh.n1 + sh.n2 + sh.nc, nslots), V3_T, sa, s>>>(d, sh);
  if ((e = cudaGetLastError())) return e;
  const dim3 grid(2 * sh.man[1] + 4, nslots);
  const int T = std::min(1024, std::max(V3_T, Bmax / 4));
  if (Bmax / 4 <= 1024) {
    if ((e = set_smem(k_v3_second<1>, sb))) return e;
    k_v3_second<1><<<grid, T, sb, s>>>(d, sh);
  } else if (Bmax / 4 <= 2048) {
    if ((e = set_smem(k_v3_second<2>, sb))) return e;
    k_v3_second<2><<<grid, T, sb, s>>>(d, sh);
  } else {
    return cudaErrorInvalidValue;
  }
  if ((e = cudaGetLastError())) return e;
  mark(se, s);
  if (input_read && (e = cudaEventRecord(input_read, s))) return e;
  if ((e = v3_peel(d, nslots, s))) return e;
  mark(se, s);
  note_launches(3);
  return cudaGetLastError();
}

}  // namespace sfft
