// tild_fft.cu — the grid half of a step as five passes over the grid lines, from the fixed-point
// densities to the float4 force field:
//
//   x forward    u64 accumulator -> float densities (kept for density reads) -> x transform
//   y forward    in place                                                        (3D)
//   z            z transform, k-space multiply, and the inverse z transforms of P and -i kz P
//   y inverse    P -> -i kx P and -i ky P, and the z derivative                  (3D)
//   x inverse    three fields at once, written as float4 nodes
//
// (small planes take x and y in one kernel each way).
//
// The channels (types, then the charge grid) are transformed in pairs, channel 2p as the real and
// 2p + 1 as the imaginary part of one complex field (an odd last channel with a zero partner).
// P(k) = Phi_2p(k) + i Phi_2p+1(k) is the pair's potential, and the pair's force along d is the
// transform of -i k_d P, so the derivative along an axis is taken just before that axis is
// transformed back: 2 + 3 + 3 line transforms per line instead of 3 + 3 + 3, and the spectra never
// exist in the three directions.  With the conversion, the multiply and the interleave inside the
// passes a pair's grid costs 5 reads and writes instead of the 13 of separate kernels around
// library transforms.
//
// A line of N = R1 R2 points is transformed in two register stages: R1-point transforms over the
// residues modulo R2, twiddles, an exchange through shared memory, R2-point transforms.  The
// radices are chosen at run time (a switch around templated butterflies), so one launch covers
// systems of different grid shapes.  A factor above 16 (a prime edge, or one with a large prime
// factor) takes a direct odd-length transform as its second stage.  Inverse transforms run the
// forward code on swapped components: swap(F(swap(x))) is the unnormalised inverse.
#include "tild_internal.cuh"
#include <algorithm>
#include <cmath>
#include <type_traits>

namespace {

inline unsigned nblk(long long n, int b) { return (unsigned)((n + b - 1) / b); }

// 64 registers: radix-16 stages with next to no spills, 1,024 threads per SM
constexpr int kThreads = 128, kMinCtas = 8;
constexpr int kTilePairs = TILD_MAXT_FAST * (TILD_MAXT_FAST + 1) / 2;
constexpr int kThreadsZ = 256, kMinCtasZ = 4;
constexpr int kThreadsX = 256, kMinCtasX = 4;
constexpr int kColsFwd = 16, kColsZ = 8;  // columns per CTA: 128- and 64-byte runs
constexpr int kXBatch = 8;         // points per thread and channel that the x forward pass loads at once

// ---- compile-time unit roots -------------------------------------------------------------------
constexpr double kTwoPi = 6.283185307179586476925286766559;
// power series on [-pi, pi]
constexpr double series_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int k = 1; k < 18; k++) {
    t *= -x * x / ((2 * k - 1) * (2 * k));
    s += t;
  }
  return s;
}
constexpr double series_sin(double x) {
  double t = x, s = x;
  for (int k = 1; k < 18; k++) {
    t *= -x * x / ((2 * k) * (2 * k + 1));
    s += t;
  }
  return s;
}
constexpr double root_angle(int k, int n) {
  k %= n;
  return kTwoPi * (2 * k > n ? k - n : k) / n;
}
template <int K, int N>
struct Root {  // exp(-2 pi i K / N) = c - i s
  static constexpr float c = (float)series_cos(root_angle(K, N));
  static constexpr float s = (float)series_sin(root_angle(K, N));
};

template <int I>
using IC = std::integral_constant<int, I>;
template <int B, int E, class F>
__device__ __forceinline__ void unrolled(F&& f) {
  if constexpr (B < E) {
    f(IC<B>{});
    unrolled<B + 1, E>(f);
  }
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 w) {
  return make_float2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}
// a exp(-2 pi i K / N)
template <int K, int N>
__device__ __forceinline__ float2 cmul_root(float2 a) {
  constexpr int k = K % N;
  if constexpr (k == 0) return a;
  else if constexpr (2 * k == N) return make_float2(-a.x, -a.y);
  else if constexpr (4 * k == N) return make_float2(a.y, -a.x);
  else if constexpr (4 * k == 3 * N) return make_float2(-a.y, a.x);
  else {
    constexpr float c = Root<k, N>::c, s = Root<k, N>::s;
    return make_float2(a.x * c + a.y * s, a.y * c - a.x * s);
  }
}

// ---- butterflies: v <- its forward transform, natural order --------------------------------------
constexpr int split_radix(int R) { return R == 16 ? 4 : R == 8 ? 4 : R % 4 == 0 ? 4 : R % 2 == 0 ? 2 : R % 3 == 0 ? 3 : 0; }

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 4) {
    const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
    v[0] = cadd(a, c);
    v[2] = csub(a, c);
    v[1] = make_float2(b.x + d.y, b.y - d.x);
    v[3] = make_float2(b.x - d.y, b.y + d.x);
  } else if constexpr (R == 3 || R == 5 || R == 7 || R == 11 || R == 13) {
    // odd prime: sums and differences of the mirrored inputs, cosines on the sums, sines on the differences
    constexpr int H = (R - 1) / 2;
    const float2 x0 = v[0];
    float2 s[H], d[H];
    float2 t = x0;
#pragma unroll
    for (int j = 0; j < H; j++) {
      s[j] = cadd(v[j + 1], v[R - 1 - j]);
      d[j] = csub(v[j + 1], v[R - 1 - j]);
      t = cadd(t, s[j]);
    }
    v[0] = t;
    unrolled<1, H + 1>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      float2 a = x0, b = make_float2(0.f, 0.f);
      unrolled<1, H + 1>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        constexpr float c = Root<j * k, R>::c, sn = Root<j * k, R>::s;
        a.x += s[j - 1].x * c;
        a.y += s[j - 1].y * c;
        b.x += d[j - 1].x * sn;
        b.y += d[j - 1].y * sn;
      });
      v[k] = make_float2(a.x + b.y, a.y - b.x);
      v[R - k] = make_float2(a.x - b.y, a.y + b.x);
    });
  } else {  // R = A B
    constexpr int A = split_radix(R), B = R / A;
    static_assert(A > 1 && A * B == R, "radix");
    float2 w[R];
    unrolled<0, B>([&](auto bc) {
      constexpr int b = decltype(bc)::value;
      float2 t[A];
#pragma unroll
      for (int a = 0; a < A; a++) t[a] = v[a * B + b];
      dft<A>(t);
      unrolled<0, A>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        w[k * B + b] = cmul_root<b * k, R>(t[k]);
      });
    });
#pragma unroll
    for (int k = 0; k < A; k++) {
      float2 t[B];
#pragma unroll
      for (int b = 0; b < B; b++) t[b] = w[k * B + b];
      dft<B>(t);
#pragma unroll
      for (int b = 0; b < B; b++) v[k + A * b] = t[b];
    }
  }
}

template <class F>
__device__ __forceinline__ void with_radix(int R, F&& f) {
  switch (R) {
    case 1: f(IC<1>{}); break;
    case 2: f(IC<2>{}); break;
    case 3: f(IC<3>{}); break;
    case 4: f(IC<4>{}); break;
    case 5: f(IC<5>{}); break;
    case 6: f(IC<6>{}); break;
    case 7: f(IC<7>{}); break;
    case 8: f(IC<8>{}); break;
    case 9: f(IC<9>{}); break;
    case 10: f(IC<10>{}); break;
    case 11: f(IC<11>{}); break;
    case 12: f(IC<12>{}); break;
    case 13: f(IC<13>{}); break;
    case 14: f(IC<14>{}); break;
    case 15: f(IC<15>{}); break;
    default: f(IC<16>{}); break;
  }
}

__device__ __forceinline__ float2 swapped(float2 a) { return make_float2(a.y, a.x); }

// asynchronous 16-byte copies into shared memory
__device__ __forceinline__ void copy_async16(void* smem, const void* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(global));
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A stride as an opaque value: its multiples are computed where they are used.  Hoisted out of the
// (mostly single-trip) item loops, 15 of them per radix-16 access pattern spill (x forward at 128^3:
// 22.7 against 15.9 us).
__device__ __forceinline__ int here(int v) {
  asm volatile("" : "+r"(v));
  return v;
}

// An address that advances by a 32-bit byte step: one wide multiply-add per access.
struct Run {
  char* p;
  unsigned step;
  __device__ __forceinline__ Run(const void* at, unsigned bytes) : p((char*)at), step(here(bytes)) {}
  __device__ __forceinline__ float2& operator[](int k) const {
    return *reinterpret_cast<float2*>(p + (unsigned long long)step * (unsigned)k);
  }
};

// R-point transform of v and the twiddles exp(-2 pi i j k / N) of residue j; tw: rows of R (rounded
// up to even) twiddles per residue, read as 16-byte pairs
template <int R>
__device__ __forceinline__ void dft_twiddle(float2 (&v)[R], int j, const float2* __restrict__ tw) {
  dft<R>(v);
  const float4* t = reinterpret_cast<const float4*>(tw) + j * ((R + 1) / 2);
#pragma unroll
  for (int k = 0; k < R; k += 2) {
    const float4 w = __ldg(t + k / 2);
    if (k) v[k] = cmul(v[k], make_float2(w.x, w.y));
    if (k + 1 < R) v[k + 1] = cmul(v[k + 1], make_float2(w.z, w.w));
  }
}

// The same for lanes along j (row passes): tw holds one row of R2 twiddles per k1, so that the lanes
// of a load read consecutive twiddles (rows per residue, lanes j apart 128 bytes, cost an 8-way bank
// conflict in L1: 16 of the 48 wavefronts per 32 points of the x forward pass at 128^3).
template <int R>
__device__ __forceinline__ void dft_twiddle_rows(float2 (&v)[R], int j, int R2, const float2* __restrict__ tw) {
  dft<R>(v);
  const Run t(tw + j, R2 * sizeof(float2));
#pragma unroll
  for (int k = 1; k < R; k++) v[k] = cmul(v[k], __ldg(&t[k]));
}

// Direct transform of odd length L of e[0], e[stride], ..: outputs k0 .. k0 + K - 1 (at most
// (L - 1) / 2) and their mirrors L - k to st(k, value).  Mirrored inputs are added and subtracted
// first, so an output and its mirror cost 2 (L - 1) multiply-adds together.  roots: for each j =
// 1 .. (L - 1) / 2 a row of exp(-2 pi i j k / L) over k, padded to whole groups of 2, 4 or 6; the lanes of
// a warp share k0, so its 16-byte loads are broadcast (stepping an index j k mod L through one row of
// roots took 54 instead of 36 instructions per j).
__host__ __device__ constexpr int direct_row(int L) { return ((L + 1) / 2 + 11) / 12 * 12; }
template <int K, class St>
__device__ __forceinline__ void dft_direct(const float2* __restrict__ e, int stride, int L, int k0,
                                           const float2* __restrict__ roots, St&& st) {
  static_assert(K % 2 == 0, "pairs of roots");
  const int H = (L - 1) / 2;
  const float2 x0 = e[0];
  float2 a[K], b[K];
#pragma unroll
  for (int q = 0; q < K; q++) {
    a[q] = x0;
    b[q] = make_float2(0.f, 0.f);
  }
  const float2 *lo = e + stride, *hi = e + (L - 1) * stride;
  const float4* w = reinterpret_cast<const float4*>(roots + k0);
  const int wrow = direct_row(L) / 2;
#pragma unroll 4
  for (int j = 1; j <= H; j++, lo += stride, hi -= stride, w += wrow) {
    const float2 u = *lo, v = *hi;
    const float2 s = cadd(u, v), d = csub(u, v);
#pragma unroll
    for (int q = 0; q < K; q += 2) {
      const float4 c = __ldg(w + q / 2);  // (cos, -sin) of k0 + q and k0 + q + 1
      a[q].x += s.x * c.x;
      a[q].y += s.y * c.x;
      b[q].x -= d.x * c.y;
      b[q].y -= d.y * c.y;
      a[q + 1].x += s.x * c.z;
      a[q + 1].y += s.y * c.z;
      b[q + 1].x -= d.x * c.w;
      b[q + 1].y -= d.y * c.w;
    }
  }
#pragma unroll
  for (int q = 0; q < K; q++) {
    const int k = k0 + q;
    if (k > H) break;
    st(k, make_float2(a[q].x + b[q].y, a[q].y - b[q].x));
    if (k) st(L - k, make_float2(a[q].x - b[q].y, a[q].y + b[q].x));
  }
}

// item / d for d >= 1 and item * d < 2^32: one multiply-high
struct FastDiv {
  unsigned d, m;
  __device__ __forceinline__ explicit FastDiv(int dd) : d(dd), m(dd > 1 ? 0xFFFFFFFFu / (unsigned)dd + 1u : 0u) {}
  __device__ __forceinline__ int div(int v) const { return d == 1 ? v : (int)__umulhi((unsigned)v, m); }
};

// Second stage by threads tid of nthreads: q counts (line, k1) combinations; src(q) is the first of its
// R2 values, `stride` their distance; dst(q) is indexed by k2 for the results; put(dst, k2, value).
// DIRECT: some system of the launch has R2 > 16.  Kernels without it are separate: the direct
// transform's accumulators cost the radix stages beside it registers (128^3 z pass 36.7 against 33 us).  Only the x forward pass has one kernel
// for both: it came out slower without (22 against 16.5 us).
template <bool DIRECT, class Src, class Dst, class Put>
__device__ __forceinline__ void second_stage(int tid, int nthreads, int nq, int R1, int R2, int stride,
                                             const float2* __restrict__ tw, Src&& src, Dst&& dst, Put&& put) {
  if (!DIRECT || R2 <= 16) {
    with_radix(R2, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
#pragma unroll 1
      for (int q = tid; q < nq; q += nthreads) {
        const float2* e = src(q);
        const int pitch = here(stride);
        float2 v[R];
#pragma unroll
        for (int n = 0; n < R; n++) v[n] = e[n * pitch];
        dft<R>(v);
        const auto d = dst(q);
#pragma unroll
        for (int k = 0; k < R; k++) put(d, k, v[k]);
      }
    });
  } else {
    const float2* roots = tw + R2 * ((R1 + 1) & ~1);  // after the twiddles
    const FastDiv dq(nq);
    auto groups = [&](auto kc) {
      constexpr int K = decltype(kc)::value;
      const int ng = ((R2 + 1) / 2 + K - 1) / K;
#pragma unroll 1
      for (int i = tid; i < nq * ng; i += nthreads) {
        const int gr = dq.div(i), q = i - gr * nq;
        const auto d = dst(q);
        dft_direct<K>(src(q), stride, R2, gr * K, roots, [&](int k, float2 v) { put(d, k, v); });
      }
    };
    // More outputs per thread share the inputs' loads, fewer keep every thread at work: rounds of the
    // threads times the instructions per input (17^3: 32.7 us a step with 2 outputs, 40.6 with 6).
    auto rounds = [&](int K) { return (nq * (((R2 + 1) / 2 + K - 1) / K) + nthreads - 1) / nthreads; };
    const int c2 = rounds(2) * 17, c4 = rounds(4) * 26, c6 = rounds(6) * 35;
    if (c6 <= c4 && c6 <= c2) groups(IC<6>{});
    else if (c4 <= c2) groups(IC<4>{});
    else groups(IC<2>{});
  }
}

// Grid of a system as the passes see it: a 2D system is one with ny = 1 whose second axis is z.
struct Lines {
  int nx, ny, nz;
  long long M;
  __device__ __forceinline__ Lines(const Geom& g, int D)
      : nx(g.nx[0]), ny(D == 3 ? g.nx[1] : 1), nz(D == 3 ? g.nx[2] : g.nx[1]), M(g.M) {}
};

// active_at with its three reads under way together: their latency is on the path of every pass (40^3:
// 28.7 us a step, one after another 29.6).  past: `ahead`, or kFirstStep in place of 0.
constexpr int kFirstStep = -(1 << 30);
__device__ __forceinline__ bool moves(const SysDev* sd, int past) {
  const long long stop = sd->stop_at, step = sd->step;
  return sd->active && (stop < 0 || step + past < stop);
}

// rows of an x pass's CTA: about `points` points of each field
__host__ __device__ inline int rows_per_cta(int nx, int points) {
  return points < nx ? 1 : points / nx > 32 ? 32 : points / nx;
}

// ---- x forward ---------------------------------------------------------------------------------
// A CTA takes consecutive rows of one channel pair.  write_rho: the float densities are stored too
// (the last step before the host can read them, and every step with fieldphase styles).  Inactive
// systems are converted, not transformed.
__global__ void __launch_bounds__(kThreads, kMinCtas) k_fft_x_fwd(unsigned long long* __restrict__ fx, float* __restrict__ rho,
                                                   float2* __restrict__ zk, const float2* __restrict__ twid,
                                                   const int2* __restrict__ blocks, const SysDev* __restrict__ sysd,
                                                   int D, int points, int write_rho, int past, int blk_off) {
  extern __shared__ __align__(16) float2 ex[];
  const int2 bk = blocks[blockIdx.x + blk_off];
  const SysDev& sd = sysd[bk.x];
  const Lines g(sd.g, D);
  const int R1 = sd.fft_r1[0], R2 = sd.fft_r2[0], R2p = R2 | 1, LT = rows_per_cta(g.nx, points);
  const float2 *tw = twid + sd.fft_tw[0], *twr = tw + sd.fft_twr;
  const int rows = g.ny * g.nz, tiles = (rows + LT - 1) / LT;
  const int p = bk.y / tiles, row0 = (bk.y - p * tiles) * LT, nl = min(LT, rows - row0);
  const bool two = 2 * p + 1 < sd.T + sd.C, paired = sd.fwd_packed;
  unsigned long long* a = fx + sd.grid0 + 2 * (long long)p * g.M + (long long)row0 * g.nx;
  float* ra = rho + sd.grid0 + 2 * (long long)p * g.M;
  float2* rp = reinterpret_cast<float2*>(ra) + (long long)row0 * g.nx;
  ra += (long long)row0 * g.nx;
  grid_launch_next();
  grid_wait();
  const bool act = moves(after_wait(&sd), past);
  a = after_wait(a);
  unsigned long long* b = a + g.M;
  // the rows are one run of the grid: coalesced loads, kXBatch of each channel in flight per thread
  float2* in = ex + LT * R1 * R2p;
  const int npt = nl * g.nx;
  auto batch = [&](int i0, auto full) {
    long long va[kXBatch], vb[kXBatch];
#pragma unroll
    for (int q = 0; q < kXBatch; q++) {
      const int i = i0 + q * kThreads;
      const bool in_run = decltype(full)::value || i < npt;
      va[q] = in_run ? (long long)a[i] : 0;
      vb[q] = two && in_run ? (long long)b[i] : 0;
    }
#pragma unroll
    for (int q = 0; q < kXBatch; q++) {
      const int i = i0 + q * kThreads;
      if (!decltype(full)::value && i >= npt) break;
      a[i] = 0ull;
      if (two) b[i] = 0ull;
      const float2 v = make_float2(__ll2float_rn(va[q]) * 0x1p-32f, __ll2float_rn(vb[q]) * 0x1p-32f);
      if (write_rho) {
        if (paired) {
          rp[i] = v;
        } else {
          ra[i] = v.x;
          if (two) ra[g.M + i] = v.y;
        }
      }
      in[i] = v;
    }
  };
  for (int i0 = 0; i0 < npt; i0 += kXBatch * kThreads) {
    if (i0 + kXBatch * kThreads <= npt) batch(i0 + threadIdx.x, IC<1>{});
    else batch(i0 + threadIdx.x, IC<0>{});
  }
  if (!act) return;  // one system per CTA
  __syncthreads();
  const FastDiv dj(R2);
  with_radix(R1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
#pragma unroll 1
    for (int i = threadIdx.x; i < nl * R2; i += kThreads) {
      const int line = dj.div(i), j = i - line * R2;
      const float2* s = in + line * g.nx + j;
      const int from = here(R2), to = here(R2p);
      float2 v[R];
#pragma unroll
      for (int n = 0; n < R; n++) v[n] = s[n * from];
      dft_twiddle_rows<R>(v, j, R2, twr);
      float2* e = ex + line * R * R2p + j;
#pragma unroll
      for (int k = 0; k < R; k++) e[k * to] = v[k];
    }
  });
  __syncthreads();
  float2* z = zk + sd.zk0 + (long long)p * g.M + (long long)row0 * g.nx;
  const FastDiv dk(R1);
  const unsigned step = R1 * sizeof(float2);
  second_stage<true>(threadIdx.x, kThreads, nl * R1, R1, R2, 1, tw, [&](int q) { return ex + q * R2p; },
               [&](int q) {
                 const int line = dk.div(q);
                 return Run(z + line * g.nx + (q - line * R1), step);
               },
               [](const Run& d, int k2, float2 v) { d[k2] = v; });
}

// ---- y forward, in place -------------------------------------------------------------------------
// A CTA takes kColsFwd consecutive columns (x fastest, then z); lanes along the columns.  Past the
// last column the last one is transformed again and not stored.
template <bool DIRECT>
__global__ void __launch_bounds__(kThreads, kMinCtas) k_fft_y_fwd(float2* __restrict__ zk, const float2* __restrict__ twid,
                                                   const int2* __restrict__ blocks, const SysDev* __restrict__ sysd,
                                                   int past, int blk_off) {
  extern __shared__ __align__(16) float2 ex[];
  constexpr int LT = kColsFwd;
  const int2 bk = blocks[blockIdx.x + blk_off];
  const SysDev& sd = sysd[bk.x];
  const Lines g(sd.g, 3);
  const int R1 = sd.fft_r1[1], R2 = sd.fft_r2[1];
  const float2* tw = twid + sd.fft_tw[1];
  const int cols = g.nx * g.nz, tiles = (cols + LT - 1) / LT;
  const int p = bk.y / tiles, c0 = (bk.y - p * tiles) * LT;
  const int line = threadIdx.x % LT, c = min(c0 + line, cols - 1);
  const bool ok = c0 + line < cols;
  const int cz = c / g.nx, row = g.nx * sizeof(float2);
  char* z = reinterpret_cast<char*>(zk + sd.zk0 + (long long)p * g.M + (long long)cz * g.nx * g.ny + (c - cz * g.nx));
  grid_launch_next();
  grid_wait();
  if (!moves(after_wait(&sd), past)) return;
  z = after_wait(z);
  with_radix(R1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
#pragma unroll 1
    for (int j = threadIdx.x / LT; j < R2; j += kThreads / LT) {
      const Run s(z + j * row, R2 * row);
      float2 v[R];
#pragma unroll
      for (int n = 0; n < R; n++) v[n] = s[n];
      dft_twiddle<R>(v, j, tw);
      float2* e = ex + j * (R * LT) + line;
#pragma unroll
      for (int k = 0; k < R; k++) e[k * LT] = v[k];
    }
  });
  __syncthreads();
  second_stage<DIRECT>(threadIdx.x, kThreads, R1 * LT, R1, R2, R1 * LT, tw, [&](int q) { return ex + q; },
               [&](int q) { return Run(z + (q / LT) * row, R1 * row); },
               [&](const Run& d, int k2, float2 v) {
                 if (ok) d[k2] = v;
               });
}

// ---- z forward, k-space multiply, z inverse --------------------------------------------------------
// The z columns (kx, ky) in the order of the z pass: rows 0 < ky < ny / 2 in full, then the rows that
// are their own mirror for kx <= nx / 2.  Every other column is the mirror (-kx, -ky) of one of these.
struct ZColumn {
  int kx, ky, mx, my;  // the column and its mirror
  __device__ __forceinline__ ZColumn(int c, int nx, int ny) {
    const int full = (ny - 1) / 2 * nx, nxh = nx / 2 + 1;
    if (c < full) {
      ky = c / nx;
      kx = c - ky * nx;
      ky += 1;
    } else {
      const int r = c - full, second = r >= nxh;
      ky = second ? ny / 2 : 0;
      kx = r - second * nxh;
    }
    mx = kx ? nx - kx : 0;
    my = ky ? ny - ky : 0;
  }
};
__host__ __device__ inline int z_columns(int nx, int ny) { return (ny - 1) / 2 * nx + (1 + (ny % 2 == 0)) * (nx / 2 + 1); }

// Multipliers in the order in which the z pass reads them, [CTA][type pair, then charge][kz][column],
// so that a CTA fetches its own with 16-byte copies: U_ab / 2 summed over the styles of the types
// (a, b), a self pair twice (Phi_a takes u rho_a from both sides); the half is that of pair_unpack.
__global__ void k_fft_multipliers(float* __restrict__ ztab, const float* __restrict__ utab, const float* __restrict__ ctab,
                                  SysDev sd, int D) {
  const Lines g(sd.g, D);
  const int nu = sd.T * (sd.T + 1) / 2, nq = nu + sd.C, cols = z_columns(g.nx, g.ny);
  const long long n = (long long)((cols + kColsZ - 1) / kColsZ) * nq * g.nz * kColsZ;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int col = (int)(i % kColsZ);
  long long r = i / kColsZ;
  const int kz = (int)(r % g.nz);
  r /= g.nz;
  const int q = (int)(r % nq), blk = (int)(r / nq);
  const ZColumn zc(min(blk * kColsZ + col, cols - 1), g.nx, g.ny);
  const int nxh = g.nx / 2 + 1;
  const long long h = zc.kx > g.nx / 2
                          ? ((long long)(kz ? g.nz - kz : 0) * g.ny + zc.my) * nxh + zc.mx
                          : ((long long)kz * g.ny + zc.ky) * nxh + zc.kx;
  float w = 0.f;
  if (q == nu) w = 0.5f * ctab[sd.ctab0 + h];
  for (int k = 0; q < nu && k < sd.nfft; k++) {
    const int a = min(sd.sa[k], sd.sb[k]), b = max(sd.sa[k], sd.sb[k]);
    if (b * (b + 1) / 2 + a == q) w += (a == b ? 1.f : 0.5f) * utab[sd.utab0 + (long long)k * sd.g.Mh + h];
  }
  ztab[sd.zt0 + i] = w;
}

// Phi_a(k) = sum_b U_ab(k) rho_b(k) for up to NT types, with 2 rho from spectrum() and U / 2 from
// multiplier(pair index)
template <int NT, class U, class Spec, class Put>
__device__ __forceinline__ void multiply_tile(int T, U&& multiplier, Spec&& spectrum, Put&& put, bool types_last) {
  float2 rk[NT], phi[NT];
#pragma unroll
  for (int t = 0; t < NT; t++) {
    rk[t] = (t < T) ? spectrum(t) : make_float2(0.f, 0.f);
    phi[t] = make_float2(0.f, 0.f);
  }
#pragma unroll
  for (int b = 0; b < NT; b++)
#pragma unroll
    for (int a = 0; a <= b; a++) {
      if (b >= T) break;
      const float w = multiplier(b * (b + 1) / 2 + a);
      phi[a].x += w * rk[b].x;
      phi[a].y += w * rk[b].y;
      if (a != b) {
        phi[b].x += w * rk[a].x;
        phi[b].y += w * rk[a].y;
      }
    }
#pragma unroll
  for (int t = 0; t < NT; t++)
    if (t < T) put(t, phi[t], types_last && t == T - 1);
}

// The column (kx, ky) and its mirror (-kx, -ky) hold both k and -k of every kz, which is what taking
// a pair's spectra apart needs: X_2p(k) = (Z(k) + conj Z(-k)) / 2, X_2p+1 = (Z(k) - conj Z(-k)) / 2i.
// A CTA takes kColsZ columns and their mirrors (as many further lines) of every pair of a system.
// Its halves transform two pairs at once, and the two inverse fields of a pair.
template <bool DIRECT>
__global__ void __launch_bounds__(kThreadsZ, kMinCtasZ) k_fft_z_kmul(const float2* zk, float2* __restrict__ gk,
                                                    const float* __restrict__ ztab, const float* __restrict__ utab_all,
                                                    const float* __restrict__ ctab_all, const float* __restrict__ kd_all,
                                                    const float2* __restrict__ twid, const int2* __restrict__ blocks,
                                                    const SysDev* __restrict__ sysd, int D, int integrate, int ahead, int blk_off) {
  extern __shared__ __align__(16) float2 sm[];
  __shared__ float s_scale[kTilePairs];  // ramp factor of each type pair
  constexpr int LT = kColsZ, LL = 2 * LT;
  const int2 bk = blocks[blockIdx.x + blk_off];
  const SysDev& sd = sysd[bk.x];
  const Lines g(sd.g, D);
  const int T = sd.T, C = sd.C, np = (T + C + 1) / 2;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int R1 = sd.fft_r1[D - 1], R2 = sd.fft_r2[D - 1];
  const float2* tw = twid + sd.fft_tw[D - 1];
  const int exn = nz * LL;
  const int half = threadIdx.x / (kThreadsZ / 2), ht = threadIdx.x % (kThreadsZ / 2);
  float2* ex = sm + half * exn;               // [j][k1][line], one per half
  float2* pb = sm + 2 * exn;                  // the pairs' columns [pair][kz][line]
  // multipliers [type pair, then charge][kz][column]: with one pair they share the second half's
  // exchange buffer, which is first used after them
  const bool tile = sd.ztile, shared_ub = sd.ztile == 2;
  const int nu = T * (T + 1) / 2, nuz = (nu + C) * nz * LT;
  float* ub = reinterpret_cast<float*>(shared_ub ? sm + exn : pb + np * exn);
  // this thread's column (line % LT) and line, the same in every stage
  const int line = threadIdx.x % LL;
  const int cols = z_columns(nx, ny), c0 = bk.y * LT + line % LT;
  const bool ok = c0 < cols;
  const ZColumn zc_(ok ? c0 : cols - 1, nx, ny);
  const int kx = zc_.kx, ky = zc_.ky, mx = zc_.mx, my = zc_.my;
  if (tile) {
    const float4* u = reinterpret_cast<const float4*>(ztab + sd.zt0 + (long long)bk.y * nuz);
    for (int i = threadIdx.x; i < nuz / 4; i += kThreadsZ) copy_async16(reinterpret_cast<float4*>(ub) + i, u + i);
  }
  const bool mirror = line >= LT;
  const bool store = ok && !(mirror && mx == kx && my == ky);  // a self-mirrored column is written once
  const long long at = mirror ? (long long)my * nx + mx : (long long)ky * nx + kx;
  const unsigned pl = (unsigned)(nx * ny * (int)sizeof(float2));
  grid_wait();
  grid_launch_next();  // only now: what starts early from here on (the gather) finds the last step's kernels done
  const SysDev* now = after_wait(&sd);
  const long long est = now->step + ahead + (integrate ? 1 : 0);
  if (!moves(now, ahead ? ahead : kFirstStep)) {
    copies_wait();  // the multipliers are still on their way into this block's shared memory
    return;
  }
  zk = after_wait(zk);
  if (tile && threadIdx.x < nu) s_scale[threadIdx.x] = sd.zramp[threadIdx.x] < 0 ? 1.f : ramp_ratio(sd, sd.zramp[threadIdx.x], est);
  for (int p0 = 0; p0 < np; p0 += 2) {
    const int p = p0 + half;
    const bool on = p < np;
    if (p0) __syncthreads();
    if (on) {
      const char* z = reinterpret_cast<const char*>(zk + sd.zk0 + (long long)p * g.M + at);
      with_radix(R1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
#pragma unroll 1
        for (int j = ht / LL; j < R2; j += kThreadsZ / 2 / LL) {
          const Run s(z + (unsigned long long)pl * (unsigned)j, pl * R2);
          float2 v[R];
#pragma unroll
          for (int n = 0; n < R; n++) v[n] = s[n];
          dft_twiddle<R>(v, j, tw);
          float2* e = ex + j * (R * LL) + line;
#pragma unroll
          for (int k = 0; k < R; k++) e[k * LL] = v[k];
        }
      });
    }
    __syncthreads();
    float2* pz = pb + p * exn;
    if (on)
      second_stage<DIRECT>(ht, kThreadsZ / 2, R1 * LL, R1, R2, R1 * LL, tw, [&](int q) { return ex + q; },
                   [&](int q) { return pz + q; },
                   [&](float2* d, int k2, float2 v) { d[k2 * (R1 * LL)] = v; });
  }
  copies_wait();
  __syncthreads();
  // multiply: one thread per (column, kz), which writes k and -k
  {
    const int l = threadIdx.x % LT;
    for (int kz = threadIdx.x / LT; kz < nz; kz += kThreadsZ / LT) {
      const int mz = kz ? nz - kz : 0;
      float2* zc = pb + kz * LL + l;
      float2* zm = pb + mz * LL + LT + l;
      auto spectrum = [&](int ch) {  // twice pair_unpack
        const float2 a = zc[(ch >> 1) * exn], b = zm[(ch >> 1) * exn];
        return ch & 1 ? make_float2(a.y + b.y, b.x - a.x) : make_float2(a.x + b.x, a.y - b.y);
      };
      float2 held = make_float2(0.f, 0.f);
      auto put = [&](int ch, float2 P, bool last) {  // channels come in order
        if (!(ch & 1) && !last) {
          held = P;
          return;
        }
        const float2 A = (ch & 1) ? held : P, B = (ch & 1) ? P : make_float2(0.f, 0.f);
        zc[(ch >> 1) * exn] = make_float2(A.x - B.y, A.y + B.x);
        zm[(ch >> 1) * exn] = make_float2(A.x + B.y, B.x - A.y);
      };
      const float2 rc = C ? spectrum(T) : make_float2(0.f, 0.f);
      float cm = 0.f;
      if (tile) {
        const float* u = ub + kz * LT + l;
        const int step = nz * LT;
        auto multiplier = [&](int q) { return u[q * step] * s_scale[q]; };
        if (T == 1) multiply_tile<1>(T, multiplier, spectrum, put, !C);
        else if (T == 2) multiply_tile<2>(T, multiplier, spectrum, put, !C);
        else if (T == 3) multiply_tile<3>(T, multiplier, spectrum, put, !C);
        else multiply_tile<TILD_MAXT_FAST>(T, multiplier, spectrum, put, !C);
        if (C) cm = u[nu * step];
      } else {  // more types, or ramped and constant styles on one pair of types: style by style from the tables
        const bool fold = kx > nx / 2;  // the tables cover kx <= nx / 2: their mirrors stand for the others
        const long long h = fold ? ((long long)mz * ny + my) * (nx / 2 + 1) + mx : ((long long)kz * ny + ky) * (nx / 2 + 1) + kx;
        float2 phi[TILD_MAX_TYPES];
        for (int t = 0; t < T; t++) phi[t] = make_float2(0.f, 0.f);
        for (int k = 0; k < sd.nfft; k++) {
          const float u = 0.5f * __ldg(utab_all + sd.utab0 + k * sd.g.Mh + h) * ramp_ratio(sd, k, est);
          const int a = sd.sa[k], b = sd.sb[k];
          const float2 ra = spectrum(a), rb = spectrum(b);
          phi[a].x += u * rb.x; phi[a].y += u * rb.y;
          phi[b].x += u * ra.x; phi[b].y += u * ra.y;
        }
        for (int t = 0; t < T; t++) put(t, phi[t], !C && t == T - 1);
        if (C) cm = 0.5f * __ldg(ctab_all + sd.ctab0 + h);
      }
      if (C) put(T, make_float2(cm * rc.x, cm * rc.y), true);
    }
  }
  // inverse: P (2D: its x derivative -i kx P) and -i kz P along z
  const float* kz_tab = kd_all + sd.kd0 + nx + (D == 3 ? ny : 0);
  const float kx_f = D == 2 ? __ldg(kd_all + sd.kd0 + (mirror ? mx : kx)) : 0.f;
  const int f = half;
  for (int p = 0; p < np; p++) {
    const float2* pz = pb + p * exn + line;
    char* out = reinterpret_cast<char*>(gk + sd.gkp0 + (long long)(p * D + f * (D - 1)) * g.M + at);
    __syncthreads();
    with_radix(R1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
#pragma unroll 1
      for (int j = ht / LL; j < R2; j += kThreadsZ / 2 / LL) {
        const float2* s = pz + j * LL;
        const int step = here(R2 * LL);
        float2 v[R];
#pragma unroll
        for (int n = 0; n < R; n++) v[n] = swapped(s[n * step]);
        if (f) {
#pragma unroll
          for (int n = 0; n < R; n++) {  // swapped(-i k P) from swapped(P)
            const float k = __ldg(kz_tab + n * R2 + j);
            v[n] = make_float2(-k * v[n].y, k * v[n].x);
          }
        }
        dft_twiddle<R>(v, j, tw);
        float2* e = ex + j * (R * LL) + line;
#pragma unroll
        for (int k = 0; k < R; k++) e[k * LL] = v[k];
      }
    });
    __syncthreads();
    second_stage<DIRECT>(ht, kThreadsZ / 2, R1 * LL, R1, R2, R1 * LL, tw, [&](int q) { return ex + q; },
                 [&](int q) { return Run(out + (unsigned long long)pl * (q / LL), pl * R1); },
                 [&](const Run& d, int k2, float2 v) {
                   if (store) d[k2] = D == 2 && !f ? make_float2(kx_f * v.x, -kx_f * v.y) : swapped(v);
                 });
  }
}

struct Field {
  Run run;
  int f;
};

// ---- y inverse: (P, z derivative) -> (x, y, z derivatives) -----------------------------------------
// LT = 8: the CTA's threads transform the three fields of 8 columns at once (small grids: the most
// threads at work).  LT = 16: 128-byte runs, one field after another (large grids: 64-byte runs at
// power-of-two strides cost twice the L1 wavefronts).
template <int LT, bool DIRECT>
__global__ void __launch_bounds__(LT == 8 ? 192 : 128, LT == 8 ? 5 : 8)
    k_fft_y_inv(float2* __restrict__ gk, const float* __restrict__ kd_all, const float2* __restrict__ twid,
                const int2* __restrict__ blocks, const SysDev* __restrict__ sysd, int past, int blk_off) {
  extern __shared__ __align__(16) float2 ex[];
  constexpr int THREADS = LT == 8 ? 192 : 128, NF = LT == 8 ? 3 : 1;  // NF fields at once
  const int2 bk = blocks[blockIdx.x + blk_off];
  const SysDev& sd = sysd[bk.x];
  const Lines g(sd.g, 3);
  const int R1 = sd.fft_r1[1], R2 = sd.fft_r2[1], R1p = R1 | 1;  // odd rows of LT: no bank conflicts between residues
  const float2* tw = twid + sd.fft_tw[1];
  const int cols = g.nx * g.nz, tiles = (cols + LT - 1) / LT;
  const int p = bk.y / tiles, c0 = (bk.y - p * tiles) * LT;
  const int line = threadIdx.x % LT, c = min(c0 + line, cols - 1);
  const bool ok = c0 + line < cols;
  const int cz = c / g.nx, row = g.nx * sizeof(float2);
  char* z = reinterpret_cast<char*>(gk + sd.gkp0 + (long long)p * 3 * g.M + (long long)cz * g.nx * g.ny + (c - cz * g.nx));
  const unsigned long long field = (unsigned long long)g.M * sizeof(float2);
  const float* ky = kd_all + sd.kd0 + g.nx;
  const float kx = __ldg(kd_all + sd.kd0 + (c - cz * g.nx));
  const int exn = R2 * R1p * LT, nq = R1 * LT;
  const FastDiv dr(R2), df(nq);
  grid_launch_next();
  grid_wait();
  if (!moves(after_wait(&sd), past)) return;
  z = after_wait(z);
  // P's y derivative first: P itself is overwritten by its x derivative
  for (int f0 = 0; f0 < 3; f0 += NF) {
    if (f0) __syncthreads();
    with_radix(R1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
#pragma unroll 1
      for (int i = threadIdx.x / LT; i < NF * R2; i += THREADS / LT) {
        const int fi = NF == 1 ? 0 : dr.div(i), j = i - fi * R2, f = f0 + fi;  // 0: y, 1: x, 2: z derivative
        const Run s(z + (f == 2 ? 2 * field : 0) + j * row, R2 * row);
        float2 v[R];
#pragma unroll
        for (int n = 0; n < R; n++) v[n] = swapped(s[n]);
        if (f == 0) {
#pragma unroll
          for (int n = 0; n < R; n++) {  // v is swapped(P): swapped(-i k P) = (-k P.x, k P.y)
            const float k = __ldg(ky + n * R2 + j);
            v[n] = make_float2(-k * v[n].y, k * v[n].x);
          }
        }
        dft_twiddle<R>(v, j, tw);
        float2* e = ex + fi * exn + j * ((R | 1) * LT) + line;
#pragma unroll
        for (int k = 0; k < R; k++) e[k * LT] = v[k];
      }
    });
    __syncthreads();
    second_stage<DIRECT>(threadIdx.x, THREADS, NF * nq, R1, R2, R1p * LT, tw,
                 [&](int q) {
                   const int fi = NF == 1 ? 0 : df.div(q);
                   return ex + fi * exn + (q - fi * nq);
                 },
                 [&](int q) {
                   const int fi = NF == 1 ? 0 : df.div(q), r = q - fi * nq, f = f0 + fi;
                   return Field{Run(z + (f == 0 ? 1 : f == 1 ? 0 : 2) * field + (r / LT) * row, R1 * row), f};
                 },
                 [&](const Field& d, int k2, float2 v) {  // v is swapped(result); the x derivative is -i kx P
                   if (ok) d.run[k2] = d.f == 1 ? make_float2(kx * v.x, -kx * v.y) : swapped(v);
                 });
  }
}

// ---- x inverse and interleave ----------------------------------------------------------------------
// A CTA takes consecutive rows of one pair in all D fields; the second stage leaves its results in
// shared memory and the rows are written as float4 nodes (real parts to channel 2p, imaginary parts
// to 2p + 1), lanes along x.
template <bool DIRECT>
__global__ void __launch_bounds__(kThreadsX, kMinCtasX) k_fft_x_inv(const float2* __restrict__ gk, float4* __restrict__ g4_all,
                                                   const float2* __restrict__ twid, const int2* __restrict__ blocks,
                                                   const SysDev* __restrict__ sysd, int D, int points, int layout, int past, int blk_off) {
  extern __shared__ __align__(16) float2 ex[];
  __shared__ int s_row[32];  // node offset of each row
  const int2 bk = blocks[blockIdx.x + blk_off];
  const SysDev& sd = sysd[bk.x];
  const Lines g(sd.g, D);
  const int R1 = sd.fft_r1[0], R2 = sd.fft_r2[0], R2p = R2 | 1, LT = rows_per_cta(g.nx, points), nx = g.nx;
  const float2 *tw = twid + sd.fft_tw[0], *twr = tw + sd.fft_twr;
  const int rows = g.ny * g.nz, tiles = (rows + LT - 1) / LT;
  const int p = bk.y / tiles, row0 = (bk.y - p * tiles) * LT, nl = min(LT, rows - row0);
  const float2* src = gk + sd.gkp0 + (long long)p * D * g.M + (long long)row0 * nx;
  const int exn = LT * R1 * R2p;
  const FastDiv dj(R2), dl(nl), dk(R1);
  const bool linear = layout == TILD_FIELD_LINEAR;
  if (threadIdx.x < nl) {
    const int row = row0 + threadIdx.x, z = row / g.ny, y = row - z * g.ny;
    s_row[threadIdx.x] = linear ? row * nx : tild_field_off(layout, 1, y, sd.g) + tild_field_off(layout, 2, z, sd.g);
  }
  grid_launch_next();
  grid_wait();
  if (!moves(after_wait(&sd), past)) return;
  src = after_wait(src);
  with_radix(R1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
#pragma unroll 1
    for (int i = threadIdx.x; i < D * nl * R2; i += kThreadsX) {
      const int fl = dj.div(i), j = i - fl * R2, f = dl.div(fl), line = fl - f * nl;
      const Run s(src + f * g.M + line * nx + j, R2 * sizeof(float2));
      float2 v[R];
#pragma unroll
      for (int n = 0; n < R; n++) v[n] = swapped(s[n]);
      dft_twiddle_rows<R>(v, j, R2, twr);
      float2* e = ex + f * exn + line * R * R2p + j;
      const int to = here(R2p);
#pragma unroll
      for (int k = 0; k < R; k++) e[k * to] = v[k];
    }
  });
  __syncthreads();
  float4* ga = g4_all + sd.g4_0 + 2 * (long long)p * sd.Mb;
  const long long second = 2 * p + 1 < sd.T + sd.C ? sd.Mb : 0;
  // the values are swapped(result): the real part, channel 2p's force, is in .y
  auto node = [&](int dst, float2 vx, float2 vy, float2 vz) {
    ga[dst] = make_float4(vx.y, vy.y, vz.y, 0.f);
    if (second) ga[second + dst] = make_float4(vx.x, vy.x, vz.x, 0.f);
  };
  // a regular second stage writes each (field, row, k1)'s results over its own inputs, a direct one
  // into a second buffer
  const int nq = nl * R1;
  float2* res = ex + (R2 > 16 ? D * exn : 0);
  const FastDiv df(nq);
  auto slot = [&](int q) {
    const int f = df.div(q);
    return f * exn + (q - f * nq) * R2p;
  };
  second_stage<DIRECT>(threadIdx.x, kThreadsX, D * nq, R1, R2, 1, tw, [&](int q) { return ex + slot(q); },
               [&](int q) { return res + slot(q); }, [](float2* d, int k2, float2 v) { d[k2] = v; });
  __syncthreads();
#pragma unroll 1
  for (int i = threadIdx.x; i < nl * nx; i += kThreadsX) {
    const int k2 = df.div(i), q = i - k2 * nq, line = dk.div(q), x = q - line * R1 + R1 * k2;
    const float2* r = res + q * R2p + k2;
    node(s_row[line] + (linear ? x : ((x >> 2) << 6) | (x & 3)), r[0], r[exn], D == 3 ? r[2 * exn] : make_float2(0.f, 0.f));
  }
}

// ---- small planes: x and y passes in one kernel each -------------------------------------------------
// A plane of up to kPlanePoints points fits in shared memory twice, so a CTA converts and transforms a
// whole z plane of a pair, and takes one field of a plane back through y and x to its component of the
// float4 nodes (4-byte stores in place of 16-byte ones).  Two kernels less on the path of a step whose
// passes take 4 us each, us a step with and without: 40^3 diblock 28.4 / 29.7, 45^3 melt 51.5 / 54.0,
// 33x52x75 lamella 67.2 / 70.9, 8 slots of 24^3 to 45^3 60.9 / 64.4.  512 threads take every stage of a
// plane in one round; the inverse of more than 2 planes' fields per SM is better off with twice the CTAs
// (the 8 slots: 16.8 against 20.7 us, 48^3: 33.3 against 30.3 a step).
constexpr int kPlanePoints = 2304, kThreadsPlane = 512;
__host__ __device__ inline int plane_exchange(int nx, int ny, int r1x, int r2x) {  // complex values of the exchange
  const int rows = ny * r1x * (r2x | 1);
  return rows > nx * ny ? rows : nx * ny;
}

template <bool DIRECT>
__global__ void __launch_bounds__(kThreadsPlane, 1024 / kThreadsPlane)
    k_fft_plane_fwd(unsigned long long* __restrict__ fx, float* __restrict__ rho, float2* __restrict__ zk,
                    const float2* __restrict__ twid, const int2* __restrict__ blocks, const SysDev* __restrict__ sysd,
                    int write_rho, int past, int blk_off) {
  extern __shared__ __align__(16) float2 ex[];
  const int2 bk = blocks[blockIdx.x + blk_off];
  const SysDev& sd = sysd[bk.x];
  const Lines g(sd.g, 3);
  const int nx = g.nx, ny = g.ny, npt = nx * ny;
  const int R1 = sd.fft_r1[0], R2 = sd.fft_r2[0], R2p = R2 | 1, Y1 = sd.fft_r1[1], Y2 = sd.fft_r2[1];
  const float2 *tw = twid + sd.fft_tw[0], *twr = tw + sd.fft_twr, *twy = twid + sd.fft_tw[1];
  const int p = bk.y / g.nz, plane = bk.y - p * g.nz;
  const bool two = 2 * p + 1 < sd.T + sd.C, paired = sd.fwd_packed;
  float2* in = ex + plane_exchange(nx, ny, R1, R2);
  unsigned long long* a = fx + sd.grid0 + 2 * (long long)p * g.M + (long long)plane * npt;
  float* ra = rho + sd.grid0 + 2 * (long long)p * g.M;
  float2* rp = reinterpret_cast<float2*>(ra) + (long long)plane * npt;
  ra += (long long)plane * npt;
  grid_launch_next();
  grid_wait();
  const bool act = moves(after_wait(&sd), past);
  a = after_wait(a);
  unsigned long long* b = a + g.M;
  for (int i0 = threadIdx.x; i0 < npt; i0 += kXBatch * kThreadsPlane) {
    long long va[kXBatch], vb[kXBatch];
#pragma unroll
    for (int q = 0; q < kXBatch; q++) {
      const int i = i0 + q * kThreadsPlane;
      va[q] = i < npt ? (long long)a[i] : 0;
      vb[q] = two && i < npt ? (long long)b[i] : 0;
    }
#pragma unroll
    for (int q = 0; q < kXBatch; q++) {
      const int i = i0 + q * kThreadsPlane;
      if (i >= npt) break;
      a[i] = 0ull;
      if (two) b[i] = 0ull;
      const float2 v = make_float2(__ll2float_rn(va[q]) * 0x1p-32f, __ll2float_rn(vb[q]) * 0x1p-32f);
      if (write_rho) {
        if (paired) {
          rp[i] = v;
        } else {
          ra[i] = v.x;
          if (two) ra[g.M + i] = v.y;
        }
      }
      in[i] = v;
    }
  }
  if (!act) return;  // one system per CTA
  __syncthreads();
  const FastDiv dj(R2), dk(R1), dx(nx);
  with_radix(R1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
#pragma unroll 1
    for (int i = threadIdx.x; i < ny * R2; i += kThreadsPlane) {
      const int line = dj.div(i), j = i - line * R2, from = here(R2), to = here(R2p);
      const float2* s = in + line * nx + j;
      float2 v[R];
#pragma unroll
      for (int n = 0; n < R; n++) v[n] = s[n * from];
      dft_twiddle_rows<R>(v, j, R2, twr);
      float2* e = ex + line * R * R2p + j;
#pragma unroll
      for (int k = 0; k < R; k++) e[k * to] = v[k];
    }
  });
  __syncthreads();
  second_stage<DIRECT>(threadIdx.x, kThreadsPlane, ny * R1, R1, R2, 1, tw, [&](int q) { return ex + q * R2p; },
                      [&](int q) {
                        const int line = dk.div(q);
                        return in + line * nx + (q - line * R1);
                      },
                      [&](float2* d, int k2, float2 v) { d[k2 * R1] = v; });
  __syncthreads();
  with_radix(Y1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
#pragma unroll 1
    for (int i = threadIdx.x; i < nx * Y2; i += kThreadsPlane) {
      const int j = dx.div(i), from = here(Y2 * nx), to = here(nx);
      const float2* s = in + i;  // row j, column i - j nx
      float2 v[R];
#pragma unroll
      for (int n = 0; n < R; n++) v[n] = s[n * from];
      dft_twiddle<R>(v, j, twy);
      float2* e = ex + j * (R - 1) * nx + i;
#pragma unroll
      for (int k = 0; k < R; k++) e[k * to] = v[k];
    }
  });
  __syncthreads();
  float2* z = zk + sd.zk0 + (long long)p * g.M + (long long)plane * npt;
  const unsigned step = Y1 * nx * sizeof(float2);
  second_stage<DIRECT>(threadIdx.x, kThreadsPlane, nx * Y1, Y1, Y2, Y1 * nx, twy, [&](int q) { return ex + q; },
                      [&](int q) { return Run(z + q, step); }, [](const Run& d, int k2, float2 v) { d[k2] = v; });
}

struct PlaneValue {
  float2* p;
  float k;
};
struct NodeRun {
  float *a, *b;
  int x;
};
template <int THREADS, bool DIRECT>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
    k_fft_plane_inv(const float2* __restrict__ gk, float4* __restrict__ g4_all, const float* __restrict__ kd_all,
                    const float2* __restrict__ twid, const int2* __restrict__ blocks, const SysDev* __restrict__ sysd,
                    int layout, int past, int blk_off) {
  extern __shared__ __align__(16) float2 ex[];
  const int2 bk = blocks[blockIdx.x + blk_off];
  const SysDev& sd = sysd[bk.x];
  const Lines g(sd.g, 3);
  const int nx = g.nx, ny = g.ny, npt = nx * ny;
  const int R1 = sd.fft_r1[0], R2 = sd.fft_r2[0], R2p = R2 | 1, Y1 = sd.fft_r1[1], Y2 = sd.fft_r2[1];
  const float2 *tw = twid + sd.fft_tw[0], *twr = tw + sd.fft_twr, *twy = twid + sd.fft_tw[1];
  const int f = bk.y % 3, r = bk.y / 3, p = r / g.nz, plane = r - p * g.nz;  // f: x, y, z derivative
  float2* pl = ex + plane_exchange(nx, ny, R1, R2);
  const float2* src = gk + sd.gkp0 + (long long)p * 3 * g.M + (f == 2 ? 2 * g.M : 0) + (long long)plane * npt;
  const float *kx = kd_all + sd.kd0, *ky = kx + nx;
  const FastDiv dj(R2), dk(R1), dx(nx);
  grid_launch_next();
  grid_wait();
  if (!moves(after_wait(&sd), past)) return;
  src = after_wait(src);
  with_radix(Y1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
#pragma unroll 1
    for (int i = threadIdx.x; i < nx * Y2; i += THREADS) {
      const int j = dx.div(i), to = here(nx);
      const Run s(src + i, Y2 * nx * sizeof(float2));
      float2 v[R];
#pragma unroll
      for (int n = 0; n < R; n++) v[n] = swapped(s[n]);
      if (f == 1) {
#pragma unroll
        for (int n = 0; n < R; n++) {  // swapped(-i k P) from swapped(P)
          const float k = __ldg(ky + n * Y2 + j);
          v[n] = make_float2(-k * v[n].y, k * v[n].x);
        }
      }
      dft_twiddle<R>(v, j, twy);
      float2* e = ex + j * (R - 1) * nx + i;
#pragma unroll
      for (int k = 0; k < R; k++) e[k * to] = v[k];
    }
  });
  __syncthreads();
  second_stage<DIRECT>(threadIdx.x, THREADS, nx * Y1, Y1, Y2, Y1 * nx, twy, [&](int q) { return ex + q; },
                      [&](int q) { return PlaneValue{pl + q, f ? 0.f : __ldg(kx + (q - dx.div(q) * nx))}; },
                      [&](const PlaneValue& d, int k2, float2 v) {
                        d.p[k2 * (Y1 * nx)] = f ? v : make_float2(-d.k * v.y, d.k * v.x);
                      });
  __syncthreads();
  with_radix(R1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
#pragma unroll 1
    for (int i = threadIdx.x; i < ny * R2; i += THREADS) {
      const int line = dj.div(i), j = i - line * R2, from = here(R2), to = here(R2p);
      const float2* s = pl + line * nx + j;
      float2 v[R];
#pragma unroll
      for (int n = 0; n < R; n++) v[n] = s[n * from];
      dft_twiddle_rows<R>(v, j, R2, twr);
      float2* e = ex + line * R * R2p + j;
#pragma unroll
      for (int k = 0; k < R; k++) e[k * to] = v[k];
    }
  });
  __syncthreads();
  float* ga = reinterpret_cast<float*>(g4_all + sd.g4_0 + 2 * (long long)p * sd.Mb) + f;
  const bool two = 2 * p + 1 < sd.T + sd.C, linear = layout == TILD_FIELD_LINEAR;
  const long long second = 4 * sd.Mb;
  const int zoff = linear ? plane * npt : tild_field_off(layout, 2, plane, sd.g);
  second_stage<DIRECT>(threadIdx.x, THREADS, ny * R1, R1, R2, 1, tw, [&](int q) { return ex + q * R2p; },
                      [&](int q) {
                        const int line = dk.div(q), row = zoff + (linear ? line * nx : tild_field_off(layout, 1, line, sd.g));
                        float* at = ga + 4ll * row;
                        return NodeRun{at, at + second, q - line * R1};
                      },
                      [&](const NodeRun& d, int k2, float2 v) {  // v is swapped(result): the real part is channel 2p's
                        const int x = d.x + R1 * k2, o = 4 * (linear ? x : ((x >> 2) << 6) | (x & 3));
                        d.a[o] = v.y;
                        if (two) d.b[o] = v.x;
                      });
}

// fieldphase on the interleaved field: type a gets +rho_a f_r, type b -rho_b f_r (planar densities)
__global__ void k_fieldphase_nodes(float4* g4, long long Mb, const float* rho,
                                   const float* __restrict__ fr, int a, int b, Geom g, int D, int layout) {
  const long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (m >= g.M) return;
  long long dst = m;
  if (layout != TILD_FIELD_LINEAR) {
    const unsigned mu = (unsigned)m, r = mu / (unsigned)g.nx[0];
    const int x = (int)(mu - r * (unsigned)g.nx[0]), y = (int)(r % (unsigned)g.nx[1]), z = (int)(r / (unsigned)g.nx[1]);
    dst = tild_field_off(layout, 0, x, g) + tild_field_off(layout, 1, y, g) + tild_field_off(layout, 2, z, g);
  }
  const float f[3] = {fr[m], fr[g.M + m], D == 3 ? fr[2 * g.M + m] : 0.f};
  grid_launch_next();
  grid_wait();
  g4 = after_wait(g4);
  rho = after_wait(rho);
  const float ra = rho[(long long)a * g.M + m], rb = rho[(long long)b * g.M + m];
  float4 v = g4[(long long)a * Mb + dst];
  v.x += ra * f[0];
  v.y += ra * f[1];
  v.z += ra * f[2];
  g4[(long long)a * Mb + dst] = v;
  v = g4[(long long)b * Mb + dst];
  v.x -= rb * f[0];
  v.y -= rb * f[1];
  v.z -= rb * f[2];
  g4[(long long)b * Mb + dst] = v;
}

constexpr size_t kMaxSmem = 200 * 1024;

// N = R1 R2 with R1 <= 16 and R2 <= 16 (as square as possible, the larger first), or R2 a prime
// up to kMaxDirect for the direct second stage.
constexpr int kMaxDirect = 127;
bool split_length(int N, int* r1, int* r2) {
  if (N > 256) return false;
  int best = 0;
  for (int a = 1; a <= 16; a++)
    if (N % a == 0 && N / a <= 16 && (!best || std::max(a, N / a) < std::max(best, N / best))) best = a;
  if (best) {
    *r1 = std::max(best, N / best);
    *r2 = std::min(best, N / best);
    return true;
  }
  auto prime = [](int n) {
    for (int d = 2; d * d <= n; d++)
      if (n % d == 0) return false;
    return true;
  };
  for (int a = 16; a >= 1; a--)
    if (N % a == 0 && N / a <= kMaxDirect && prime(N / a)) {
      *r1 = a;
      *r2 = N / a;
      return true;
    }
  return false;
}

// shared memory of the z pass: exchange buffers, the pairs' columns and the multipliers
size_t z_smem(int nz, int T, int C) {
  const int np = (T + C + 1) / 2, nu = T <= TILD_MAXT_FAST ? T * (T + 1) / 2 + C : 0;
  const size_t line = (size_t)nz * kColsZ * sizeof(float);
  return (2 + np) * 4 * line + (np > 1 || nu > 4 ? nu * line : 0);
}

template <class K>
bool allow_smem(K* k) {
  const void* f = reinterpret_cast<const void*>(k);
  return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) == cudaSuccess;
}

}  // namespace

// Whether a grid shape takes these passes.  Measured against the library transforms with their separate
// conversion, multiply and interleave kernels, us a step of a small diblock system, here / library:
// 40^3 25.8 / 38.7, 64^3 36.4 / 44.6, 96^3 62.8 / 95.7, 128^3 117 / 147, 256^3 844 / 1039, 94^3 (2 x 47)
// 131 / 235.  Prime edges, which take the direct transform: 29^3 31.1 / 37.8, 61^3 75.8 / 76.7, 113^3
// 401 / 448; 8 slots of 24^3 to 45^3 59 / 111.  A second factor above 16 that is not prime (125 = 5 x 25: 213 / 164) and a
// 2D grid whose second axis is prime (101^2, 7 CTAs in the z pass: 49.6 / 36.3) stay with the library.
bool tild_fft_supports(const int* nx, int D, int T, int C) {
  int a, b;
  for (int d = 0; d < D; d++) {
    if (!split_length(nx[d], &a, &b)) return false;
    if (D == 2 && d == 1 && b > 16) return false;
  }
  return z_smem(nx[D - 1], T, C) <= kMaxSmem;
}

// Radices, unit roots and block tables of every system whose grid shape takes these passes.
int tild_fft_setup(tild_ctx* c) {
  const int D = c->D;
  std::vector<int> lens, offs;
  std::vector<float2> roots;
  for (auto& pa : c->fft_pass) pa = tild_ctx::FftPass();
  // x tiles of 256 to 1,024 points of each field, so that small grids still give every SM a few CTAs
  long long points = 0;
  for (const Bucket& b : c->buckets)
    for (int s : b.systems)
      if (b.own) points += (c->sys[s].T + c->sys[s].C + 1) / 2 * c->sys[s].g.M;
  c->fft_points = (int)std::min(1024ll, std::max(256ll, points / (4 * kSms)));
  c->fft_plane = D == 3;
  for (const Bucket& b : c->buckets)
    if (b.own) c->fft_plane = c->fft_plane && b.nx[0] * b.nx[1] <= kPlanePoints;
  c->fft_wide = points >= 16 * 32 * 4 * kSms;  // the y inverse pass still has some CTAs of 16 columns for every SM
  std::vector<int2> tab[5];
  long long ztotal = 0;
  for (Bucket& b : c->buckets) {
    for (int k = 0; k < 5; k++) b.fft_blk0[k] = (int)tab[k].size();
    if (b.own) {
      for (int s : b.systems) {
        SysDev& d = c->h_sys[s];
        const SysHost& h = c->sys[s];
        const Geom& g = h.g;
        const int np = (h.T + h.C + 1) / 2;
        for (int a = 0; a < 3; a++) d.fft_r1[a] = d.fft_r2[a] = 1, d.fft_tw[a] = 0;
        for (int a = 0; a < D; a++) {
          const int N = g.nx[a];
          int r1, r2;
          split_length(N, &r1, &r2);
          const int axis = a == D - 1 ? 2 : a;  // of the passes: x, y, z
          b.fft_direct[axis] = b.fft_direct[axis] || r2 > 16;
          c->fft_direct[axis] = c->fft_direct[axis] || r2 > 16;
          d.fft_r1[a] = (short)r1;
          d.fft_r2[a] = (short)r2;
          size_t k = 0;
          while (k < lens.size() && lens[k] != N) k++;
          if (k == lens.size()) {
            lens.push_back(N);
            offs.push_back((int)roots.size());
            // twiddles [j][k1], rows padded to even, the rows of a direct second stage, twiddles [k1][j]
            auto root = [&](int m, int n) {
              roots.push_back(make_float2((float)std::cos(kTwoPi * m / n), (float)-std::sin(kTwoPi * m / n)));
            };
            for (int j = 0; j < r2; j++)
              for (int q = 0; q < (r1 + 1) / 2 * 2; q++) root(j * q % N, N);
            if (r2 > 16)
              for (int j = 1; j <= (r2 - 1) / 2; j++)
                for (int q = 0; q < direct_row(r2); q++) root(j * q % r2, r2);
            for (int q = 0; q < r1; q++)
              for (int j = 0; j < r2; j++) root(j * q % N, N);
            if (roots.size() % 2) root(0, 1);
          }
          d.fft_tw[a] = offs[k];
          if (a == 0) d.fft_twr = r2 * ((r1 + 1) / 2 * 2) + (r2 > 16 ? (r2 - 1) / 2 * direct_row(r2) : 0);
        }
        const int nx = g.nx[0], ny = D == 3 ? g.nx[1] : 1, nz = D == 3 ? g.nx[2] : g.nx[1];
        const int zcols = z_columns(nx, ny);
        const int ltx = rows_per_cta(nx, c->fft_points);
        const long long rows = (long long)ny * nz, cols = (long long)nx * nz;
        int nblocks[5] = {np * (int)nblk(rows, ltx), np * (int)nblk(cols, kColsFwd), (int)nblk(zcols, kColsZ),
                                np * (int)nblk(cols, c->fft_wide ? 16 : 8), np * (int)nblk(rows, ltx)};
        d.zt0 = ztotal;
        if (h.T <= TILD_MAXT_FAST) ztotal += (long long)nblocks[2] * (h.T * (h.T + 1) / 2 + h.C) * nz * kColsZ;
        const int rx2 = d.fft_r2[0], row = d.fft_r1[0] * (rx2 | 1);
        size_t smem[5] = {sizeof(float2) * ltx * (row + nx), sizeof(float2) * kColsFwd * ny, z_smem(nz, h.T, h.C),
                                sizeof(float2) * (c->fft_wide ? 16 : 3 * 8) * (d.fft_r1[1] | 1) * d.fft_r2[1], (rx2 > 16 ? 2 : 1) * D * sizeof(float2) * ltx * row};
        if (c->fft_plane) {
          nblocks[0] = np * nz;
          nblocks[4] = 3 * np * nz;
          smem[0] = smem[4] = sizeof(float2) * (nx * ny + plane_exchange(nx, ny, d.fft_r1[0], d.fft_r2[0]));
        }
        for (int k = 0; k < 5; k++) {
          if ((D == 2 || c->fft_plane) && (k == 1 || k == 3)) continue;
          auto& pa = c->fft_pass[k];
          pa.smem = std::max(pa.smem, smem[k]);
          for (int q = 0; q < nblocks[k]; q++) tab[k].push_back(make_int2(s, q));
        }
      }
    }
    for (int k = 0; k < 5; k++) b.fft_nblk[k] = (int)tab[k].size() - b.fft_blk0[k];
  }
  if (tab[0].empty()) return TILD_OK;
  if (tild_check(c, cudaMalloc(&c->ztab, sizeof(float) * std::max(ztotal, 1ll)), "alloc multipliers")) return TILD_ERR_OOM;
  if (tild_check(c, cudaMalloc(&c->fft_twid, sizeof(float2) * roots.size()), "alloc unit roots")) return TILD_ERR_OOM;
  if (tild_check(c, cudaMemcpyAsync(c->fft_twid, roots.data(), sizeof(float2) * roots.size(), cudaMemcpyHostToDevice, c->stream), "unit roots"))
    return TILD_ERR_CUDA;
  for (int k = 0; k < 5; k++) {
    if (tab[k].empty()) continue;
    c->fft_pass[k].n = (int)tab[k].size();
    if (tild_check(c, cudaMalloc(&c->fft_pass[k].blocks, sizeof(int2) * tab[k].size()), "alloc transform blocks")) return TILD_ERR_OOM;
    if (tild_check(c, cudaMemcpyAsync(c->fft_pass[k].blocks, tab[k].data(), sizeof(int2) * tab[k].size(), cudaMemcpyHostToDevice, c->stream), "transform blocks"))
      return TILD_ERR_CUDA;
  }
  auto both = [](auto* regular, auto* direct) { return allow_smem(regular) && allow_smem(direct); };
  const bool okattr = both(k_fft_plane_fwd<false>, k_fft_plane_fwd<true>) &&
                      both(k_fft_plane_inv<256, false>, k_fft_plane_inv<256, true>) &&
                      both(k_fft_plane_inv<512, false>, k_fft_plane_inv<512, true>) && allow_smem(k_fft_x_fwd) && both(k_fft_y_fwd<false>, k_fft_y_fwd<true>) &&
                      both(k_fft_z_kmul<false>, k_fft_z_kmul<true>) && both(k_fft_y_inv<8, false>, k_fft_y_inv<8, true>) &&
                      both(k_fft_y_inv<16, false>, k_fft_y_inv<16, true>) && both(k_fft_x_inv<false>, k_fft_x_inv<true>);
  if (!okattr) {
    c->err = "shared memory of the transform passes";
    return TILD_ERR_CUDA;
  }
  return tild_check(c, cudaStreamSynchronize(c->stream), "transform setup") ? TILD_ERR_CUDA : TILD_OK;
}

void tild_fft_free(tild_ctx* c) {
  if (c->fft_twid) cudaFree(c->fft_twid);
  if (c->ztab) cudaFree(c->ztab);
  for (auto& pa : c->fft_pass)
    if (pa.blocks) cudaFree(pa.blocks);
}

// The z pass's multipliers of a system whose style tables have just been built, and which style's ramp
// scales each pair of types.  A pair with a ramped style beside others is multiplied style by style.
int tild_fft_tables(tild_ctx* c, int s) {
  SysDev& d = c->h_sys[s];
  if (!c->buckets[c->sys[s].bucket].own) return TILD_OK;
  d.ztile = 0;
  if (d.T > TILD_MAXT_FAST) return TILD_OK;
  int styles[kTilePairs] = {0};
  for (int q = 0; q < kTilePairs; q++) d.zramp[q] = -1;
  for (int k = 0; k < d.nfft; k++) {
    const int a = std::min(d.sa[k], d.sb[k]), b = std::max(d.sa[k], d.sb[k]), q = b * (b + 1) / 2 + a;
    styles[q]++;
    if (d.sramp[k]) d.zramp[q] = (short)k;
  }
  for (int q = 0; q < kTilePairs; q++)
    if (d.zramp[q] >= 0 && styles[q] > 1) return TILD_OK;
  const int ny = c->D == 3 ? d.g.nx[1] : 1, nz = d.g.nx[c->D - 1], nu = d.T * (d.T + 1) / 2 + d.C;
  d.ztile = (d.T + d.C + 1) / 2 > 1 || nu > 4 ? 1 : 2;
  const long long n = (long long)nblk(z_columns(d.g.nx[0], ny), kColsZ) * nu * nz * kColsZ;
  k_fft_multipliers<<<nblk(n, 256), 256, 0, c->stream>>>(c->ztab, c->utab, c->ctab, d, c->D);
  c->launches++;
  return tild_check(c, cudaGetLastError(), "multipliers") ? TILD_ERR_CUDA : TILD_OK;
}

// The passes of one grid shape (b), or of every shape that takes them (b null), on stream st.
int tild_fft_run(tild_ctx* c, const Bucket* b, bool integrate, bool active, cudaStream_t st) {
  int off[5], n[5];
  for (int k = 0; k < 5; k++) {
    off[k] = b ? b->fft_blk0[k] : 0;
    n[k] = b ? b->fft_nblk[k] : c->fft_pass[k].n;
  }
  if (n[0] == 0) return 0;
  float2* zk = reinterpret_cast<float2*>(c->rhok);
  float2* gk = reinterpret_cast<float2*>(c->gk);
  const auto* pa = c->fft_pass;
  const int wr = !integrate || c->last_of_call || !c->fields.empty(), ahead = c->ahead, past = ahead ? ahead : kFirstStep;
  const bool* dir = b ? b->fft_direct : c->fft_direct;
  const bool few = n[4] <= 2 * kSms;  // planes' fields
  if (!b) tild_mark(c, STAGE_ZERO);
  if (c->fft_plane)
    tild_launch_early(dir[0] || dir[1] ? k_fft_plane_fwd<true> : k_fft_plane_fwd<false>, n[0], kThreadsPlane, pa[0].smem, kCarveout, st, c->rho_fx, c->rho, zk, c->fft_twid, pa[0].blocks,
                      c->d_sys, wr, past, off[0]);
  else
    tild_launch_early(k_fft_x_fwd, n[0], kThreads, pa[0].smem, kCarveout, st, c->rho_fx, c->rho, zk, c->fft_twid, pa[0].blocks, c->d_sys, c->D, c->fft_points, wr, past, off[0]);
  c->launches++;
  if (!active) return tild_check(c, cudaGetLastError(), "grid passes");  // no system of the shape moves: densities only
  const bool columns = c->D == 3 && !c->fft_plane;
  if (columns) {
    if (!b) tild_mark(c, STAGE_R2C);
    tild_launch_early(dir[1] ? k_fft_y_fwd<true> : k_fft_y_fwd<false>, n[1], kThreads, pa[1].smem, kCarveout, st, zk, c->fft_twid, pa[1].blocks, c->d_sys, past, off[1]);
    c->launches++;
  }
  if (!b) tild_mark(c, STAGE_KMUL);
  tild_launch_early(dir[2] ? k_fft_z_kmul<true> : k_fft_z_kmul<false>, n[2], kThreadsZ, pa[2].smem, kCarveout, st, zk, gk, c->ztab, c->utab, c->ctab, c->kd, c->fft_twid, pa[2].blocks, c->d_sys,
              c->D, (int)integrate, ahead, off[2]);
  if (columns) {
    if (!b) tild_mark(c, STAGE_C2R);
    if (c->fft_wide)
      tild_launch_early(dir[1] ? k_fft_y_inv<16, true> : k_fft_y_inv<16, false>, n[3], 128, pa[3].smem, kCarveout, st, gk, c->kd, c->fft_twid, pa[3].blocks, c->d_sys, past, off[3]);
    else
      tild_launch_early(dir[1] ? k_fft_y_inv<8, true> : k_fft_y_inv<8, false>, n[3], 192, pa[3].smem, kCarveout, st, gk, c->kd, c->fft_twid, pa[3].blocks, c->d_sys, past, off[3]);
    c->launches++;
  }
  if (!b) tild_mark(c, STAGE_INTERLEAVE);
  if (c->fft_plane)
    tild_launch_early(dir[0] || dir[1] ? (few ? k_fft_plane_inv<512, true> : k_fft_plane_inv<256, true>)
                                       : (few ? k_fft_plane_inv<512, false> : k_fft_plane_inv<256, false>),
                      n[4], few ? 512 : 256, pa[4].smem, kCarveout, st, gk, c->g4, c->kd, c->fft_twid, pa[4].blocks,
                      c->d_sys, c->field_layout, past, off[4]);
  else
    tild_launch_early(dir[0] ? k_fft_x_inv<true> : k_fft_x_inv<false>, n[4], kThreadsX, pa[4].smem, kCarveout, st, gk, c->g4, c->fft_twid, pa[4].blocks, c->d_sys, c->D, c->fft_points, c->field_layout, past, off[4]);
  c->launches += 2;
  return tild_check(c, cudaGetLastError(), "grid passes");
}

int tild_fieldphase_nodes(tild_ctx* c, const FieldK& fk) {
  const SysHost& h = c->sys[fk.sys];
  tild_launch_early(k_fieldphase_nodes, (int)nblk(h.g.M, 256), 256, 0, kCarveout, c->stream, c->g4 + h.g4_0, h.Mb, c->rho + h.grid0,
                    c->frfield + fk.fr0, fk.a, fk.b, h.g, h.D, c->field_layout);
  c->launches++;
  return tild_check(c, cudaGetLastError(), "fieldphase");
}
