// fft.cuh — the project's Stockham FFT (common.cuh) in the two shapes the
// v1/v2 kernels use, and the selection that follows it.
//
// Both keep the operations and their order of common.cuh's radix-2 / radix-4
// stages; they differ in where the intermediate values live:
//
//   block_fft16  one CTA, N / 16 threads, two radix-4 stages per pass in
//                registers, so N points cross shared memory log16 N times
//                instead of log4 N (FP32: the exchange and its barriers are
//                what a one-CTA FFT spends its time on).
//   fft_tile     M points of an N-point transform on a tile of columns:
//                stages Ns = A .. A M.  Two launches of it (M1, then M2 =
//                N / M1) make a whole transform with every SM at work, which
//                pays for FP64 -- on GB300 one FP64 warp instruction holds a
//                sub-partition's FP64 pipe for 64 to 76 cycles, so a
//                4096-point transform costs one CTA's four sub-partitions
//                about 55 us however many threads it has -- and is the only
//                shape for transforms beyond a CTA's shared memory.
#pragma once

#include "common.cuh"

namespace sfft {

// ------------------------------------------------------------ butterflies --

// Radix-4 butterfly of common.cuh: outputs in order r = 0..3.
template <typename R>
__device__ __forceinline__ void bfly4(c2_t<R> &a, c2_t<R> &b, c2_t<R> &c, c2_t<R> &d) {
  using V = c2_t<R>;
  const V t0 = cadd<R>(a, c), t1 = csub<R>(a, c), t2 = cadd<R>(b, d), t3 = csub<R>(b, d);
  V u3;  // t3 * (-i)
  u3.x = t3.y;
  u3.y = -t3.x;
  a = cadd<R>(t0, t2);
  b = cadd<R>(t1, u3);
  c = csub<R>(t0, t2);
  d = csub<R>(t1, u3);
}

// Twiddle product.  FP32: the two fused operations spelled out, so that every
// FFT shape rounds alike (left to the compiler, the product that is fused
// varied from kernel to kernel).
template <typename R>
__device__ __forceinline__ c2_t<R> twmul(c2_t<R> x, c2_t<R> w) {
  if constexpr (sizeof(R) == 4) {
    c2_t<R> r;
    r.x = __fmaf_rn(x.x, w.x, -__fmul_rn(x.y, w.y));
    r.y = __fmaf_rn(x.y, w.x, __fmul_rn(x.x, w.y));
    return r;
  } else {
    return cmul<R>(x, w);
  }
}

// The same behind its twiddles: butterfly k of stage Ns (none when k is 0).
// tw is the stage-by-stage table (block_fft): its entries r Ns + k lie side
// by side for neighbouring k.  (A natural-order table read at r k N / (4 Ns)
// spreads a warp's 32 loads over up to 32 lines; the 8192- and 16384-point
// comb FFTs took 30 k and 79 k cycles with it.)
template <typename R>
__device__ __forceinline__ void bfly4_tw(c2_t<R> &a, c2_t<R> &b, c2_t<R> &c, c2_t<R> &d, int k, int Ns,
                                         const c2_t<R> *__restrict__ tw) {
  if (k) {
    b = twmul<R>(b, __ldg(tw + Ns + k));
    c = twmul<R>(c, __ldg(tw + 2 * Ns + k));
    d = twmul<R>(d, __ldg(tw + 3 * Ns + k));
  }
  bfly4<R>(a, b, c, d);
}

// ------------------------------------------------------- one-CTA radix 16 --

// Place of element i in the padded shared-memory array: one spare entry per
// 16, so that the stride-16 stores of a pass meet no bank twice.
__host__ __device__ __forceinline__ int fft16_at(int i) { return i + (i >> 4); }
__host__ __device__ __forceinline__ int fft16_size(int N) { return N + (N >> 4) + 1; }

// Two radix-4 stages, Ns = A and 4 A, of the 16 elements i = g + m N / 16 (m
// = 0 .. 15) in v; element o of the result (place (g - k0) 16 + k0 + o A,
// k0 = g mod A) ends in v[fft16_out(o)].
template <typename R>
__device__ __forceinline__ void pass16(c2_t<R> (&v)[16], int k0, int A, const c2_t<R> *__restrict__ tw) {
#pragma unroll
  for (int i = 0; i < 4; i++) bfly4_tw<R>(v[i], v[i + 4], v[i + 8], v[i + 12], k0, A, tw);
#pragma unroll
  for (int i = 0; i < 4; i++) bfly4_tw<R>(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3], i * A + k0, 4 * A, tw);
}
__host__ __device__ constexpr int fft16_out(int o) { return 4 * (o & 3) + (o >> 2); }

// Forward FFT of N = 2^logN >= 16 points; threads t < N / 16 work, every
// thread of the block calls.  ld(i): input i.  The result is
// buf[fft16_at(i)], visible to the whole block on return.
template <typename R, typename Ld>
__device__ __forceinline__ void block_fft16(c2_t<R> *buf, int N, int logN, const c2_t<R> *__restrict__ tw, Ld ld) {
  using V = c2_t<R>;
  const int T = N >> 4, t = threadIdx.x, q4 = N >> 2;
  const bool act = t < T;
  V v[16];
  int Ns;
  if (logN & 1) {  // radix 2 and radix 4: two transforms of 8 points per thread
    if (act) {
#pragma unroll
      for (int s = 0; s < 2; s++) {
        V *u = v + 8 * s;
#pragma unroll
        for (int m = 0; m < 8; m++) u[m] = ld(t + s * T + m * (N >> 3));
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const V a = u[i], b = u[i + 4];
          u[i] = cadd<R>(a, b);      // element 2 i
          u[i + 4] = csub<R>(a, b);  // element 2 i + 1
        }
        // butterfly i of Ns = 2 takes the elements i, i + 2, i + 4, i + 6
        bfly4<R>(u[0], u[1], u[2], u[3]);
        bfly4_tw<R>(u[4], u[5], u[6], u[7], 1, 2, tw);
#pragma unroll
        for (int r = 0; r < 4; r++) {
          buf[fft16_at(8 * (t + s * T) + 2 * r)] = u[r];
          buf[fft16_at(8 * (t + s * T) + 2 * r + 1)] = u[4 + r];
        }
      }
    }
    Ns = 8;
  } else if ((logN >> 1) & 1) {  // an odd number of radix-4 stages: the first one, without twiddles, alone
    if (act) {
#pragma unroll
      for (int s = 0; s < 4; s++) {
#pragma unroll
        for (int r = 0; r < 4; r++) v[4 * s + r] = ld(t + s * T + r * q4);
        bfly4<R>(v[4 * s], v[4 * s + 1], v[4 * s + 2], v[4 * s + 3]);
#pragma unroll
        for (int r = 0; r < 4; r++) buf[fft16_at(4 * (t + s * T) + r)] = v[4 * s + r];
      }
    }
    Ns = 4;
  } else {
    if (act) {
#pragma unroll
      for (int m = 0; m < 16; m++) v[m] = ld(t + m * T);
      pass16<R>(v, 0, 1, tw);
#pragma unroll
      for (int o = 0; o < 16; o++) buf[fft16_at(16 * t + o)] = v[fft16_out(o)];
    }
    Ns = 16;
  }
  __syncthreads();
  while (Ns < N) {
    if (16 * Ns <= N) {
      const int k0 = t & (Ns - 1), base = (t - k0) * 16 + k0;
      if (act) {
#pragma unroll
        for (int m = 0; m < 16; m++) v[m] = buf[fft16_at(t + m * T)];
        pass16<R>(v, k0, Ns, tw);
      }
      __syncthreads();
      if (act) {
#pragma unroll
        for (int o = 0; o < 16; o++) buf[fft16_at(base + o * Ns)] = v[fft16_out(o)];
      }
      __syncthreads();
      Ns *= 16;
    } else {  // one stage left: Ns = N / 4
      if (act) {
#pragma unroll
        for (int s = 0; s < 4; s++) {
          const int j = t + s * T;
#pragma unroll
          for (int r = 0; r < 4; r++) v[4 * s + r] = buf[fft16_at(j + r * q4)];
          bfly4_tw<R>(v[4 * s], v[4 * s + 1], v[4 * s + 2], v[4 * s + 3], j, Ns, tw);
        }
#pragma unroll
        for (int s = 0; s < 4; s++)  // the stage is in place: butterfly j reads and writes j + r N / 4
#pragma unroll
          for (int r = 0; r < 4; r++) buf[fft16_at(t + s * T + r * q4)] = v[4 * s + r];
      }
      __syncthreads();
      Ns = N;
    }
  }
}

// ------------------------------------------------- tiles of a long FFT --

// Split of an N-point transform into two launches of M1 and M2 = N / M1
// points; M2 is a power of four, M1 takes the radix-2 stage if there is one.
__host__ __device__ __forceinline__ int floor_log2(unsigned v) {
#ifdef __CUDA_ARCH__
  return 31 - __clz(v);
#else
  return 31 - __builtin_clz(v);
#endif
}
__host__ __device__ __forceinline__ int fft_m2(int N) { return 1 << (2 * ((floor_log2(N) >> 1) >> 1)); }

// Stages Ns = A .. A M of an N-point transform on the columns g0 .. g0 + C
// (C = 2^lc) of a CTA's tile: column g has the elements g + m N / M (m <
// M).  One butterfly per thread and stage, M C / 4 threads work; sm: M C
// entries.  RADIX2: the first stage is the radix-2 one (A = 1 only).  ld(i)
// reads element i, st(i, v) takes element i of the result.
template <typename R, typename Ld, typename St>
__device__ __forceinline__ void fft_tile(c2_t<R> *sm, int M, int lc, int A, int N, int g0, bool radix2,
                                         const c2_t<R> *__restrict__ tw, Ld ld, St st) {
  using V = c2_t<R>;
  const int C = 1 << lc, c = threadIdx.x & (C - 1), i = threadIdx.x >> lc;
  const int g = g0 + c, k0 = g & (A - 1), q4 = M >> 2, row = N / M;
  const bool act = i < q4;
  const long base = (long)(g - k0) * M + k0;
  if (M == 1) {  // nothing left to do: the tile's columns are passed on
    if (i < 1) st(g, ld(g));
    return;
  }
  V v[4];
  if (act) {
#pragma unroll
    for (int r = 0; r < 4; r++) v[r] = ld(g + (i + r * q4) * row);
  }
  int ns = 1;
  if (radix2) {
    if (act) {
      const V a = v[0], b = v[1];
      sm[(2 * i) * C + c] = cadd<R>(a, v[2]);
      sm[(2 * i + 1) * C + c] = csub<R>(a, v[2]);
      sm[(2 * (i + q4)) * C + c] = cadd<R>(b, v[3]);
      sm[(2 * (i + q4) + 1) * C + c] = csub<R>(b, v[3]);
    }
    ns = 2;
    __syncthreads();
    if (act) {
#pragma unroll
      for (int r = 0; r < 4; r++) v[r] = sm[(i + r * q4) * C + c];
    }
  }
  for (;;) {
    const int kl = i & (ns - 1), o0 = (i - kl) * 4 + kl;
    if (act) bfly4_tw<R>(v[0], v[1], v[2], v[3], kl * A + k0, A * ns, tw);
    if (4 * ns == M) {
      if (act) {
#pragma unroll
        for (int r = 0; r < 4; r++) st((int)(base + (long)(o0 + r * ns) * A), v[r]);
      }
      return;
    }
    __syncthreads();  // the previous stage's values are in registers
    if (act) {
#pragma unroll
      for (int r = 0; r < 4; r++) sm[(o0 + r * ns) * C + c] = v[r];
    }
    __syncthreads();
    ns *= 4;
    if (act) {
#pragma unroll
      for (int r = 0; r < 4; r++) v[r] = sm[(i + r * q4) * C + c];
    }
  }
}

// Shape of the two launches over arrays of Na and Nb points (Nb may equal
// Na): every CTA holds `elems` entries, so a launch's tile of an array with
// M rows has elems / M columns.  At least 512 entries (128 threads, one warp
// for each sub-partition); more where a tile would be narrower than a
// 32-byte sector.
struct FftShape {
  int elems[2];  // entries per CTA of the first and the second launch
};
inline FftShape fft_shape2(int Na, int Nb, int vbytes) {
  FftShape f;
  for (int p = 0; p < 2; p++) {
    int e = 512;
    for (int N : {Na, Nb}) {
      const int m2 = fft_m2(N), M = p ? m2 : N / m2;
      e = e > M * (32 / vbytes) ? e : M * (32 / vbytes);
    }
    f.elems[p] = e < 4096 ? e : 4096;  // 1024 threads; M is at most 4096 (N at most 2^22)
  }
  return f;
}
// log2 of the columns per CTA, and the CTAs of one array.
__host__ __device__ __forceinline__ int fft_lc(int elems, int M, int N) {
  const int cols = N / M, c = elems / M < cols ? elems / M : cols;
  return floor_log2(c);
}
__host__ __device__ __forceinline__ int fft_ctas(int elems, int M, int N) { return (N / M) >> fft_lc(elems, M, N); }

// -------------------------------------------------------------- selection --

// Indices of the `num` largest of N keys with the tie rule of the
// reference's find_largest_indices (src/utils.cc:130-158): the cutoff is the
// (N-num-1)-th smallest value, every index above it is taken, then indices
// equal to it in increasing order until num; the output is ascending.
//
// A histogram over the range the keys span (not over fixed digits: powers of
// one signal share their leading bits) leaves few keys in the cutoff's bin,
// which are listed and ranked against each other; a fuller bin is split
// again.  Each thread keeps the leading 32 bits of its keys in registers (S of
// them; S = 0: too many keys, read again from where they are) and goes back
// for a whole 64-bit key only where those decide nothing.  Against one
// histogram per 8 bits over keys in shared memory (and together with the FFT
// shapes above): the bucket and vote stage of 32 FP32 signals (640 FFTs of 4096
// points) 120 -> 78 us, the bucket stage of one FP64 signal of 2^24 points 212
// -> 60 us.  Registers instead of shared memory: 160 lists of 4096 64-bit keys
// 12.8 -> 9.2 us, three of 16384 20.7 -> 13.9 us.
constexpr int SEL_BINS = 1024, SEL_CAP = 256;

template <typename K>
struct SelShared {
  int hist[SEL_BINS];
  K list[SEL_CAP], cut;
  unsigned lo[32], hi[32];
  int a[32], b[32], bin, rem, cnt, n;
};

// The histogram's bin that holds rank `rem` (cum <= rem < cum + count) into
// s.bin, s.rem (rank within it) and s.cnt.  Ends with a barrier.
template <typename K>
__device__ __forceinline__ void select_bin(SelShared<K> &s, int bins, int rem) {
  constexpr unsigned FULL = 0xffffffffu;
  const int T = blockDim.x, t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int per = T >= bins ? 1 : bins / T;
  int sum = 0;
  if (t * per < bins)
    for (int q = 0; q < per; q++) sum += s.hist[t * per + q];
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(FULL, inc, o);
    if (lane >= o) inc += x;
  }
  if (lane == 31) s.a[wid] = inc;
  __syncthreads();
  int cum = __reduce_add_sync(FULL, lane < wid ? s.a[lane] : 0) + inc - sum;
  if (rem >= cum && rem < cum + sum)
    for (int q = 0; q < per; q++) {
      const int c = s.hist[t * per + q];
      if (rem >= cum && rem < cum + c) {
        s.bin = t * per + q;
        s.rem = rem - cum;
        s.cnt = c;
      }
      cum += c;
    }
  __syncthreads();
}

// keyat(i): the key of entry i.  out[0..num) (optional) receives the indices;
// bits (optional) one bit per entry, ceil(N / 32) words.  Every thread calls;
// blockDim.x is a multiple of 32, at most 1024; S = 0 or ceil(N / 32) groups
// of 32 entries are at most S per warp.  Ends with a barrier.
template <typename K, int S, typename KeyAt>
__device__ __forceinline__ void block_select(KeyAt keyat, int N, int num, int *__restrict__ out,
                                             unsigned *__restrict__ bits, SelShared<K> &s) {
  constexpr bool WIDE = sizeof(K) == 8;
  constexpr unsigned FULL = 0xffffffffu;
  const int t = threadIdx.x, T = blockDim.x, lane = t & 31, wid = t >> 5, nw = T >> 5;
  // about two keys per bin, so that short lists do not pay for 1024 bins
  const int lbins = min(10, max(5, floor_log2(N) - 1)), bins = 1 << lbins;
  // each warp owns consecutive groups of 32 entries
  const int groups = (N + 31) >> 5, per = (groups + nw - 1) / nw, g0 = min(groups, wid * per);
  const int mine = min(per, groups - g0), SN = S ? S : mine;
  auto at = [&](int g) { return ((g0 + g) << 5) + lane; };
  auto top = [&](int i) -> unsigned {
    if constexpr (WIDE)
      return (unsigned)(keyat(i) >> 32);
    else
      return keyat(i);
  };
  unsigned H[S ? S : 1];
  unsigned lo = FULL, hi = 0;
#pragma unroll
  for (int g = 0; g < (S ? S : 0); g++) {
    const bool in = g < mine && at(g) < N;
    H[g] = in ? top(at(g)) : 0u;
    lo = min(lo, in ? H[g] : FULL);
    hi = max(hi, H[g]);
  }
  auto lead = [&](int g) -> unsigned {
    if constexpr (S != 0)
      return H[g];
    else
      return at(g) < N ? top(at(g)) : 0u;
  };
  if constexpr (S == 0) {
#pragma unroll 4
    for (int g = 0; g < mine; g++)
      if (at(g) < N) {
        const unsigned h = top(at(g));
        lo = min(lo, h);
        hi = max(hi, h);
      }
  }
  lo = __reduce_min_sync(FULL, lo);
  hi = __reduce_max_sync(FULL, hi);
  if (lane == 0) {
    s.lo[wid] = lo;
    s.hi[wid] = hi;
  }
  for (int i = t; i < bins; i += T) s.hist[i] = 0;
  if (t == 0) s.n = 0;
  __syncthreads();
  lo = __reduce_min_sync(FULL, lane < nw ? s.lo[lane] : FULL);
  hi = __reduce_max_sync(FULL, lane < nw ? s.hi[lane] : 0u);
  int w = 32 - __clz(hi - lo);  // the cutoff's leading bits lie in [lo, lo + 2^w)
  int rem = N - num - 1;        // its rank among the keys there
  bool listed = false;
  for (;;) {
    const int sh = max(0, w - lbins);
#pragma unroll
    for (int g = 0; g < SN; g++) {
      const unsigned d = lead(g) - lo;  // keys below lo wrap to the top
      if (g < mine && at(g) < N && (w >= 32 || (d >> (w & 31)) == 0)) atomicAdd(&s.hist[d >> sh], 1);
    }
    __syncthreads();
    select_bin(s, bins, rem);
    lo += (unsigned)s.bin << sh;
    w = sh;
    rem = s.rem;
    listed = s.cnt <= SEL_CAP && (WIDE || w > 0);
    if (listed || w == 0) break;
    for (int i = t; i < bins; i += T) s.hist[i] = 0;
    __syncthreads();
  }
  K cut = (K)lo;
  if constexpr (WIDE) {
    // more than SEL_CAP keys share the leading bits: the same on the others
    unsigned lo2 = 0;
    int w2 = 32;
    while (!listed && w2 > 0) {
      for (int i = t; i < bins; i += T) s.hist[i] = 0;
      __syncthreads();
      const int sh = max(0, w2 - lbins);
#pragma unroll
      for (int g = 0; g < SN; g++)
        if (g < mine && at(g) < N && lead(g) == lo) {
          const unsigned d = (unsigned)keyat(at(g)) - lo2;
          if (w2 >= 32 || (d >> (w2 & 31)) == 0) atomicAdd(&s.hist[d >> sh], 1);
        }
      __syncthreads();
      select_bin(s, bins, rem);
      lo2 += (unsigned)s.bin << sh;
      w2 = sh;
      rem = s.rem;
      if (s.cnt <= SEL_CAP && w2 > 0) break;
    }
    cut = ((K)lo << 32) | lo2;
    if (!listed && w2 > 0) {  // list the keys of [cut, cut + 2^w2)
#pragma unroll
      for (int g = 0; g < SN; g++)
        if (g < mine && at(g) < N && lead(g) == lo) {
          const K k = keyat(at(g));
          if (((k - cut) >> w2) == 0) s.list[atomicAdd(&s.n, 1)] = k;
        }
      listed = true;
      w = -1;
    }
  }
  if (listed) {
    if (w >= 0) {
#pragma unroll
      for (int g = 0; g < SN; g++)
        if (g < mine && at(g) < N && ((lead(g) - lo) >> w) == 0) {
          const int p = atomicAdd(&s.n, 1);
          if constexpr (WIDE)
            s.list[p] = keyat(at(g));
          else
            s.list[p] = lead(g);
        }
    }
    __syncthreads();
    const int cnt = s.cnt;
    for (int e = t; e < cnt; e += T) {
      const K k = s.list[e];
      int r = 0;
      for (int u = 0; u < cnt; u++) {
        const K x = s.list[u];
        r += x < k || (x == k && u < e);
      }
      if (r == rem) s.cut = k;
    }
    __syncthreads();
    cut = s.cut;
  }
  // ordered compaction
  auto place = [&](int g, bool &gt, bool &eq) {
    const bool in = g < mine && at(g) < N;
    const unsigned h = lead(g);
    if constexpr (WIDE) {
      const unsigned c = (unsigned)(cut >> 32);
      gt = in && h > c;
      eq = false;
      if (in && h == c) {
        const unsigned l = (unsigned)keyat(at(g));
        gt = l > (unsigned)cut;
        eq = l == (unsigned)cut;
      }
    } else {
      gt = in && h > cut;
      eq = in && h == cut;
    }
  };
  int ngt = 0, neq = 0;
#pragma unroll
  for (int g = 0; g < SN; g++) {
    bool gt, eq;
    place(g, gt, eq);
    ngt += __popc(__ballot_sync(FULL, gt));
    neq += __popc(__ballot_sync(FULL, eq));
  }
  if (lane == 0) {
    s.a[wid] = ngt;
    s.b[wid] = neq;
  }
  __syncthreads();
  const int ca = lane < nw ? s.a[lane] : 0, cb = lane < nw ? s.b[lane] : 0;
  const int need = max(0, num - __reduce_add_sync(FULL, ca));  // entries equal to the cutoff to take
  int bgt = __reduce_add_sync(FULL, lane < wid ? ca : 0), beq = __reduce_add_sync(FULL, lane < wid ? cb : 0);
  const unsigned below = (1u << lane) - 1u;
#pragma unroll
  for (int g = 0; g < SN; g++) {
    bool gt, eq;
    place(g, gt, eq);
    const unsigned mg = __ballot_sync(FULL, gt), me = __ballot_sync(FULL, eq);
    const int pe = beq + __popc(me & below);
    const int pos = bgt + __popc(mg & below) + min(pe, need);
    const bool take = (gt || (eq && pe < need)) && pos < num;
    if (out && take) out[pos] = at(g);
    if (bits) {
      const unsigned m = __ballot_sync(FULL, take);
      if (lane == 0 && g < mine) bits[g0 + g] = m;
    }
    bgt += __popc(mg);
    beq += __popc(me);
  }
  __syncthreads();
}

}  // namespace sfft
