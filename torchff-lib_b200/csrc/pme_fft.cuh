// The PME solve of a K^3 grid in three launches, one x plane (ky row) in a block's shared memory:
//
//   forward : plane x of the charge grid -> z transform of its K real lines, y transform of the
//             K/2+1 half-spectrum columns -> spectrum [x][ky][kz]
//   solve   : the x lines of row ky -> x transform, influence function (and energy),
//             inverse x transform -> [x][ky][kz]
//   inverse : plane x -> inverse y and z transforms -> potential [x][y][z]
//
// A line of K = R1 R2 points is transformed in two steps (Cooley-Tukey): R2 transforms of R1
// points with stride R2, a twiddle, R1 transforms of R2 consecutive points. A step's transforms
// are unrolled in one thread's registers (radix up to kMaxRegRadix, again by Cooley-Tukey with
// constant twiddles; odd primes by sums over a[j] + a[R-j] and a[j] - a[R-j]); for a larger prime
// factor of K those sums run from shared memory. Two real lines go through the z transform as
// one complex line. Lanes take consecutive lines: on an odd row pitch they hit distinct banks, and
// the twiddles they share are broadcasts. Summation orders are fixed.
//
// cuFFT's transforms with the conversion to FP32 and the convolution are eight launches of 3 to 6 us
// each, all latency at these sizes: 37 us at K = 20 and 38 us at K = 48 (FP32) against 24 and 31 us
// here, and a chain of programmatic dependents leaves no gaps between the launches. Blocks of 256
// threads at 80 registers fit an SM beside the real-space kernel's: 512 threads measured the same
// alone and 7 % slower in an evaluation of 1,231 waters. For a batch, the direct transforms this
// replaces were eight launches of 205 us for 60 boxes of 250 to 4,000 waters; here 149 us.
#pragma once

#include <cmath>
#include <type_traits>
#include <utility>
#include <vector>

#include "tff_common.cuh"

namespace tff {

constexpr int kFftThreads = 256;
constexpr int kMaxRegRadix = 16;
constexpr size_t kFftSmemMax = 220 * 1024;

template <class T> struct __align__(2 * sizeof(T)) Cplx { T x, y; };

// Factor R1 <= R2 of K = R1 R2 closest to its square root.
__host__ __device__ inline int fft_radix1(int K) {
  int r = 1;
  for (int d = 2; d * d <= K; ++d)
    if (K % d == 0) r = d;
  return r;
}

__host__ __device__ inline int fft_pitch(int n) { return n | 1; }

// Table of a grid side: exp(-2 pi i m / K), m < K.
template <class T>
inline void fft_table(int K, std::vector<Cplx<T>> &out) {
  for (int m = 0; m < K; ++m) {
    const double a = 2.0 * M_PI * m / K;
    out.push_back(Cplx<T>{(T)std::cos(a), (T)-std::sin(a)});
  }
}

// Shared memory of a block: two planes of K lines, the table.
template <class T>
inline size_t fft_smem(int K) {
  return (2 * (size_t)K * fft_pitch(K) + K) * sizeof(Cplx<T>);
}

// Grid sides of the plane path: up to 78, both buffers of an FP64 plane fit the shared memory of a
// block. One energy with gradients of 3,000 charges, cuFFT -> planes, us, FP32: K = 16 37.5 -> 26.1,
// 34 51.3 -> 36.9, 48 40.1 -> 32.9, 78 55.1 -> 52.4, 80 46.1 -> 53.1, 100 53.7 -> 64.4; FP64: 34 53.2 -> 38.8,
// 48 40.3 -> 34.4, 78 85.4 -> 56.4, 80 52.8 -> 55.7. Sides with a factor beyond the registers only up to 36:
// the sums of a factor R grow as R^2. Prime sides tie to 53 (FP32 energies alone: 41 39.0 -> 37.0, 47 39.1 -> 41.3,
// 53 45.2 -> 45.2) and lose beyond (59 47.2 -> 54.9, 67 53.4 -> 65.7); twice or three times a prime can still win
// (46 51.3 -> 41.2, 51 61.5 -> 41.0, 58 55.6 -> 50.2), four times does not (68 43.1 -> 53.3, 76 47.4 -> 65.3).
inline bool fft_planes(int K) { return K <= 78 && (K <= 36 || K / fft_radix1(K) <= kMaxRegRadix); }

// Layout of a block's shared memory, in elements: plane p with the data, the other plane q, the table.
struct FftPlan {
  int K, R1, R2, p, q, tw;
};

__device__ __forceinline__ unsigned char *fft_base() {
  extern __shared__ __align__(16) unsigned char fft_smem_raw[];
  return fft_smem_raw;
}
template <class T>
__device__ __forceinline__ Cplx<T> *fft_at(int element) { return reinterpret_cast<Cplx<T> *>(fft_base()) + element; }

// Copies the table of side K into the block's shared memory. The caller synchronises before the
// first transform.
template <class T>
__device__ __forceinline__ FftPlan fft_plan(int K, const Cplx<T> *table) {
  FftPlan f;
  f.K = K;
  f.R1 = fft_radix1(K);
  f.R2 = K / f.R1;
  f.p = 0;
  f.q = K * fft_pitch(K);
  f.tw = 2 * f.q;
  for (int m = threadIdx.x; m < K; m += blockDim.x) *fft_at<T>(f.tw + m) = table[m];
  return f;
}

// Quotients by a fixed divisor of numbers below 2^16 without a division.
struct SmallDiv {
  unsigned d, magic;
  __device__ __forceinline__ explicit SmallDiv(int n) : d(n), magic(n > 1 ? 0xffffffffu / (unsigned)n + 1u : 0u) {}
  __device__ __forceinline__ int quot(int t) const { return d > 1 ? (int)__umulhi((unsigned)t, magic) : t; }
};

// a * w, or a * conj(w) for the inverse transform.
template <class T, bool INV>
__device__ __forceinline__ Cplx<T> cmul(Cplx<T> a, Cplx<T> w) {
  const T wy = INV ? -w.y : w.y;
  return Cplx<T>{fma(a.x, w.x, -a.y * wy), fma(a.x, wy, a.y * w.x)};
}

// cos(2 pi k / n) as a constant: the angle is folded into [0, pi / 4] in whole numbers, then the
// power series.
constexpr double cos_turn(int k, int n) {
  k %= n;
  if (k < 0) k += n;
  if (2 * k > n) return cos_turn(n - k, n);
  if (4 * k > n) return -cos_turn(n - 2 * k, 2 * n);
  const bool sine = 8 * k > n;  // cos(x) = sin(pi/2 - x)
  const double x = 2.0 * 3.14159265358979323846 * (sine ? n - 4 * k : k) / (sine ? 4.0 * n : n);
  double t = sine ? x : 1.0, s = t;
  for (int i = sine ? 3 : 2; i < 30; i += 2) {
    t *= -x * x / (i * (i - 1));
    s += t;
  }
  return s;
}
constexpr double sin_turn(int k, int n) { return cos_turn(4 * k - n, 4 * n); }

template <class F, int... I>
__device__ __forceinline__ void static_for(F f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F f) { static_for(f, std::make_integer_sequence<int, N>{}); }

// a * exp(-+2 pi i k / n), k and n constants.
template <class T, bool INV, int k, int n>
__device__ __forceinline__ Cplx<T> ctwiddle(Cplx<T> a) {
  if constexpr (k % n == 0) {
    return a;
  } else if constexpr (2 * (k % n) == n) {
    return Cplx<T>{-a.x, -a.y};
  } else if constexpr (4 * (k % n) == n) {
    return INV ? Cplx<T>{-a.y, a.x} : Cplx<T>{a.y, -a.x};
  } else if constexpr (4 * (k % n) == 3 * n) {
    return INV ? Cplx<T>{a.y, -a.x} : Cplx<T>{-a.y, a.x};
  } else {
    constexpr double c = cos_turn(k, n), s = sin_turn(k, n);
    return cmul<T, INV>(a, Cplx<T>{(T)c, (T)-s});
  }
}

constexpr int smallest_factor(int n) {
  for (int d = 2; d * d <= n; ++d)
    if (n % d == 0) return d;
  return n;
}

// In-register transform of R points, natural order in and out.
template <class T, int R, bool INV>
__device__ __forceinline__ void reg_dft(Cplx<T> (&a)[R]) {
  constexpr int P = smallest_factor(R);
  if constexpr (R == 2) {
    const Cplx<T> b = a[1];
    a[1] = Cplx<T>{a[0].x - b.x, a[0].y - b.y};
    a[0] = Cplx<T>{a[0].x + b.x, a[0].y + b.y};
  } else if constexpr (P == R) {
    constexpr int H = (R - 1) / 2;
    Cplx<T> s[H], d[H];  // a[j] +- a[R - j]
    Cplx<T> sum = a[0];
    static_for<H>([&](auto j) {
      s[j] = Cplx<T>{a[j + 1].x + a[R - 1 - j].x, a[j + 1].y + a[R - 1 - j].y};
      d[j] = Cplx<T>{a[j + 1].x - a[R - 1 - j].x, a[j + 1].y - a[R - 1 - j].y};
      sum.x += s[j].x;
      sum.y += s[j].y;
    });
    const Cplx<T> a0 = a[0];
    a[0] = sum;
    static_for<H>([&](auto k) {
      Cplx<T> u = a0, v{T(0), T(0)};
      static_for<H>([&](auto j) {
        constexpr int m = (decltype(j)::value + 1) * (decltype(k)::value + 1);
        constexpr double c = cos_turn(m, R), n = INV ? -sin_turn(m, R) : sin_turn(m, R);
        u.x = fma((T)c, s[j].x, u.x);
        u.y = fma((T)c, s[j].y, u.y);
        v.x = fma((T)n, d[j].x, v.x);
        v.y = fma((T)n, d[j].y, v.y);
      });
      // u - i v and its mirror u + i v
      a[k + 1] = Cplx<T>{u.x + v.y, u.y - v.x};
      a[R - 1 - k] = Cplx<T>{u.x - v.y, u.y + v.x};
    });
  } else {
    constexpr int Q = R / P;
    Cplx<T> b[Q][P];
    static_for<Q>([&](auto n2) {
      static_for<P>([&](auto n1) { b[n2][n1] = a[Q * n1 + n2]; });
      reg_dft<T, P, INV>(b[n2]);
    });
    static_for<P>([&](auto k1) {
      Cplx<T> c[Q];
      static_for<Q>([&](auto n2) {
        c[n2] = ctwiddle<T, INV, decltype(n2)::value * decltype(k1)::value, R>(b[n2][k1]);
      });
      reg_dft<T, Q, INV>(c);
      static_for<Q>([&](auto k2) { a[k1 + P * k2] = c[k2]; });
    });
  }
}

// One step over `lines` lines (element n of line l at l * pitch_line + n * pitch_el): transforms of R
// points, `groups` per line. Group g reads elements g * in_g + n * in_s and writes elements
// g * out_g + k * out_s; with `twiddle` output k of group g is multiplied by tw[g k].
struct FftStep {
  int R, groups, lines, pitch_line, pitch_el;
  int in_g, in_s, out_g, out_s;
  int in, out;  // plane read, plane written
  bool twiddle;
};

template <class T, int R, bool INV>
__device__ __forceinline__ void fft_step_r(const FftStep &s, int tw) {
  const SmallDiv by(s.lines);
  const int is = s.in_s * s.pitch_el, os = s.out_s * s.pitch_el;
  for (int t = threadIdx.x; t < s.lines * s.groups; t += blockDim.x) {
    const int g = by.quot(t), l = t - g * s.lines;
    const Cplx<T> *src = fft_at<T>(s.in + l * s.pitch_line + g * s.in_g * s.pitch_el);
    Cplx<T> *dst = fft_at<T>(s.out + l * s.pitch_line + g * s.out_g * s.pitch_el);
    Cplx<T> a[R];
#pragma unroll
    for (int n = 0; n < R; ++n) a[n] = src[n * is];
    reg_dft<T, R, INV>(a);
    if (s.twiddle) {
#pragma unroll
      for (int k = 0; k < R; ++k) dst[k * os] = k ? cmul<T, INV>(a[k], *fft_at<T>(tw + g * k)) : a[k];
    } else {
#pragma unroll
      for (int k = 0; k < R; ++k) dst[k * os] = a[k];
    }
  }
}

// The last step of a line whose radix does not fit the registers, an odd one: outputs k and R - k of
// kAnyPairs values of k at a time from the sums and differences of inputs j and R - j (as in
// reg_dft): half the multiply-adds of a direct sum, and the inputs read once for all of them. By count it
// is bound by shared memory, four loads for eight multiply-adds. An evaluation of a batch of 16 boxes of
// 300 to 1,050 waters, FP32, us, against four outputs of a direct sum per thread: K = 37 284 -> 251,
// 47 380 -> 296, 71 1,129 -> 693, 89 2,272 -> 1,169; a lone 3,000-charge grid at K = 31 40.6 -> 34.9. Two values
// of k leave the fewest threads without work at small K; three or four change K = 53 to 94 by -6 to +7 %.
constexpr int kAnyPairs = 2;

constexpr bool any_radix_is_odd() {
  for (int K = 6; K <= 96; ++K) {
    int r = 1;
    for (int d = 2; d * d <= K; ++d)
      if (K % d == 0) r = d;
    if (r > kMaxRegRadix || (K / r > kMaxRegRadix && K / r % 2 == 0)) return false;
  }
  return true;
}
static_assert(any_radix_is_odd(), "grid sides up to 96: a radix beyond the registers is odd and the last step's");

template <class T, bool INV>
__device__ __forceinline__ void fft_step_any(const FftStep &s, int tw, int stride) {
  const int R = s.R, H = (R - 1) / 2, blocks = (H + kAnyPairs - 1) / kAnyPairs;
  const SmallDiv by(s.lines), byb(blocks);
  const int is = s.in_s * s.pitch_el, os = s.out_s * s.pitch_el;
  for (int t = threadIdx.x; t < s.lines * s.groups * blocks; t += blockDim.x) {
    const int gb = by.quot(t), l = t - gb * s.lines, g = byb.quot(gb), k0 = 1 + kAnyPairs * (gb - g * blocks);
    const Cplx<T> *src = fft_at<T>(s.in + l * s.pitch_line + g * s.in_g * s.pitch_el);
    Cplx<T> *dst = fft_at<T>(s.out + l * s.pitch_line + g * s.out_g * s.pitch_el);
    const Cplx<T> a0 = src[0];
    Cplx<T> sum = a0, u[kAnyPairs], v[kAnyPairs];
    int m[kAnyPairs];  // j k mod R
#pragma unroll
    for (int q = 0; q < kAnyPairs; ++q) {
      u[q] = a0;
      v[q] = Cplx<T>{T(0), T(0)};
      m[q] = 0;
    }
#pragma unroll 4
    for (int j = 1; j <= H; ++j) {
      const Cplx<T> a = src[j * is], b = src[(R - j) * is];
      const Cplx<T> p{a.x + b.x, a.y + b.y}, d{a.x - b.x, a.y - b.y};
      sum.x += p.x;
      sum.y += p.y;
#pragma unroll
      for (int q = 0; q < kAnyPairs; ++q) {
        m[q] += k0 + q;
        m[q] -= m[q] >= R ? R : 0;
        const Cplx<T> w = *fft_at<T>(tw + m[q] * stride);
        const T n = INV ? w.y : -w.y;
        u[q].x = fma(w.x, p.x, u[q].x);
        u[q].y = fma(w.x, p.y, u[q].y);
        v[q].x = fma(n, d.x, v[q].x);
        v[q].y = fma(n, d.y, v[q].y);
      }
    }
    if (k0 == 1) dst[0] = sum;
#pragma unroll
    for (int q = 0; q < kAnyPairs; ++q) {
      const int k = k0 + q;
      if (k > H) continue;
      // u - i v and its mirror u + i v
      dst[k * os] = Cplx<T>{u[q].x + v[q].y, u[q].y - v[q].x};
      dst[(R - k) * os] = Cplx<T>{u[q].x - v[q].y, u[q].y + v[q].x};
    }
  }
}

template <class T, bool INV>
__device__ __noinline__ void fft_step(const FftStep s, int tw, int K) {
  switch (s.R) {
#define TFF_FFT_RADIX(r) \
  case r: return fft_step_r<T, r, INV>(s, tw);
    TFF_FFT_RADIX(2)
    TFF_FFT_RADIX(3)
    TFF_FFT_RADIX(4)
    TFF_FFT_RADIX(5)
    TFF_FFT_RADIX(6)
    TFF_FFT_RADIX(7)
    TFF_FFT_RADIX(8)
    TFF_FFT_RADIX(9)
    TFF_FFT_RADIX(10)
    TFF_FFT_RADIX(11)
    TFF_FFT_RADIX(12)
    TFF_FFT_RADIX(13)
    TFF_FFT_RADIX(14)
    TFF_FFT_RADIX(15)
    TFF_FFT_RADIX(16)
#undef TFF_FFT_RADIX
    default: return fft_step_any<T, INV>(s, tw, K / s.R);
  }
}

// Transforms `lines` lines of plane f.p. The result is in f.p again (the planes swap when K is
// prime). All threads of the block; ends with the result visible to it.
template <class T, bool INV>
__device__ __forceinline__ void fft_lines(FftPlan &f, int lines, int pitch_line, int pitch_el) {
  FftStep s;
  s.lines = lines;
  s.pitch_line = pitch_line;
  s.pitch_el = pitch_el;
  s.in = f.p;
  if (f.R1 > 1) {
    s.R = f.R1;
    s.groups = s.in_s = s.out_s = f.R2;
    s.in_g = s.out_g = 1;
    s.out = f.q;
    s.twiddle = true;
    fft_step<T, INV>(s, f.tw, f.K);
    __syncthreads();
    s.in = f.q;
  }
  s.R = s.in_g = f.R2;
  s.groups = s.out_s = f.R1;
  s.in_s = s.out_g = 1;
  s.out = f.R1 > 1 ? f.p : f.q;
  s.twiddle = false;
  fft_step<T, INV>(s, f.tw, f.K);
  __syncthreads();
  if (f.R1 == 1) {
    f.q = f.p;
    f.p = s.out;
  }
}

__device__ __forceinline__ float fft_real(unsigned long long v) { return (float)from_fix(v); }
__device__ __forceinline__ double fft_real(double v) { return v; }

// Plane x of `grid` -> rows [ky][kz] of the spectrum at `out`. `before_store` runs once the block has
// only its result left to write.
template <class T, class F>
__device__ __forceinline__ void fft_forward_plane(FftPlan &f, const typename Acc<T>::S *grid, Cplx<T> *out,
                                                  F before_store) {
  const int K = f.K, Kz = K / 2 + 1, st = fft_pitch(K), pairs = (K + 1) / 2;
  const SmallDiv byk(K), byz(Kz);
  // rows 2m and 2m + 1 are the real and imaginary parts of line m
#pragma unroll 4
  for (int t = threadIdx.x; t < pairs * K; t += blockDim.x) {
    const int m = byk.quot(t), z = t - m * K;
    *fft_at<T>(f.p + m * st + z) = Cplx<T>{fft_real(grid[2 * m * K + z]),
                                           2 * m + 1 < K ? fft_real(grid[(2 * m + 1) * K + z]) : T(0)};
  }
  __syncthreads();
  fft_lines<T, false>(f, pairs, st, 1);
  // their spectra: (Z[k] + conj Z[-k]) / 2 and (Z[k] - conj Z[-k]) / 2i
  for (int t = threadIdx.x; t < pairs * Kz; t += blockDim.x) {
    const int m = byz.quot(t), z = t - m * Kz;
    const Cplx<T> u = *fft_at<T>(f.p + m * st + z), v = *fft_at<T>(f.p + m * st + (z ? K - z : 0));
    *fft_at<T>(f.q + 2 * m * st + z) = Cplx<T>{T(0.5) * (u.x + v.x), T(0.5) * (u.y - v.y)};
    if (2 * m + 1 < K) *fft_at<T>(f.q + (2 * m + 1) * st + z) = Cplx<T>{T(0.5) * (u.y + v.y), T(0.5) * (v.x - u.x)};
  }
  const int spec = f.q;
  f.q = f.p;
  f.p = spec;
  __syncthreads();
  fft_lines<T, false>(f, Kz, 1, st);
  before_store();
  for (int t = threadIdx.x; t < K * Kz; t += blockDim.x) {
    const int y = byz.quot(t);
    out[t] = *fft_at<T>(f.p + y * st + t - y * Kz);
  }
}

// Rows [ky][kz] of plane x at `in` -> the plane's potential.
template <class T, class F>
__device__ __forceinline__ void fft_inverse_plane(FftPlan &f, const Cplx<T> *in, T *phi, F before_store) {
  const int K = f.K, Kz = K / 2 + 1, st = fft_pitch(K), pairs = (K + 1) / 2;
  const SmallDiv byk(K), byz(Kz);
#pragma unroll 4
  for (int t = threadIdx.x; t < K * Kz; t += blockDim.x) {
    const int y = byz.quot(t);
    *fft_at<T>(f.p + y * st + t - y * Kz) = in[t];
  }
  __syncthreads();
  fft_lines<T, true>(f, Kz, 1, st);
  // line m = A + i B of the half spectra A, B of rows 2m and 2m + 1: its transform has their real
  // lines as real and imaginary parts. The other half is conj A[K - k] + i conj B[K - k]. The
  // imaginary parts of k = 0 and K / 2 have no real counterpart: they are dropped, as in
  // cuFFT's C2R. They vanish but for rounding where the influence function of a frequency and of its mirror
  // image are equal, which the Nyquist frequencies of an even K in a sheared box are not.
  for (int t = threadIdx.x; t < pairs * Kz; t += blockDim.x) {
    const int m = byz.quot(t), z = t - m * Kz;
    const bool own = z == 0 || 2 * z == K;
    Cplx<T> a = *fft_at<T>(f.p + 2 * m * st + z), b{T(0), T(0)};
    if (2 * m + 1 < K) b = *fft_at<T>(f.p + (2 * m + 1) * st + z);
    if (own) a.y = b.y = T(0);
    *fft_at<T>(f.q + m * st + z) = Cplx<T>{a.x - b.y, a.y + b.x};
    if (!own) *fft_at<T>(f.q + m * st + K - z) = Cplx<T>{a.x + b.y, b.x - a.y};
  }
  const int lines = f.q;
  f.q = f.p;
  f.p = lines;
  __syncthreads();
  fft_lines<T, true>(f, pairs, st, 1);
  before_store();
  for (int t = threadIdx.x; t < pairs * K; t += blockDim.x) {
    const int m = byk.quot(t), z = t - m * K;
    const Cplx<T> v = *fft_at<T>(f.p + m * st + z);
    phi[2 * m * K + z] = v.x;
    if (2 * m + 1 < K) phi[(2 * m + 1) * K + z] = v.y;
  }
}

// x lines kz in [z0, z1) of row ky: transform, influence function, inverse transform, in place at
// `spec` ([x][ky][kz]). factor(x, kz) gives the influence function, scale(z) the weight of a point in
// the energy; returns this thread's share of sum_k w C(k) |S(k)|^2 / theta(k)^2. The influence
// function needs no transform: `before_load` (and it) run first.
template <class T, class Factor, class F, class G>
__device__ __forceinline__ double fft_solve_row(FftPlan &f, Cplx<T> *spec, int ky, int z0, int z1, Factor factor,
                                                F before_load, G before_store) {
  const int K = f.K, Kz = K / 2 + 1, nz = z1 - z0, st = fft_pitch(nz), total = K * nz;
  const SmallDiv byn(nz);
  // a thread's points are threadIdx.x, + blockDim.x, ...: the factors of the first few wait in registers
  constexpr int kHeld = 4;
  double held[kHeld];
#pragma unroll
  for (int u = 0; u < kHeld; ++u) {
    const int t = threadIdx.x + u * blockDim.x;
    if (t >= total) break;
    const int x = byn.quot(t);
    held[u] = factor(x, z0 + t - x * nz);
  }
  before_load();
#pragma unroll 4
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int x = byn.quot(t), z = t - x * nz;
    *fft_at<T>(f.p + x * st + z) = spec[((size_t)x * K + ky) * Kz + z0 + z];
  }
  __syncthreads();
  fft_lines<T, false>(f, nz, 1, st);
  double e = 0.0;
  const auto apply = [&](int t, double c) {
    const int x = byn.quot(t), z = t - x * nz;
    Cplx<T> &v = *fft_at<T>(f.p + x * st + z);
    const double re = v.x, im = v.y;
    e += (z0 + z == 0 || 2 * (z0 + z) == K ? 1.0 : 2.0) * c * (re * re + im * im);
    v.x = (T)(re * c);
    v.y = (T)(im * c);
  };
#pragma unroll
  for (int u = 0; u < kHeld; ++u) {
    const int t = threadIdx.x + u * blockDim.x;
    if (t < total) apply(t, held[u]);
  }
  for (int t = threadIdx.x + kHeld * blockDim.x; t < total; t += blockDim.x) {
    const int x = byn.quot(t);
    apply(t, factor(x, z0 + t - x * nz));
  }
  __syncthreads();
  fft_lines<T, true>(f, nz, 1, st);
  before_store();
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int x = byn.quot(t), z = t - x * nz;
    spec[((size_t)x * K + ky) * Kz + z0 + z] = *fft_at<T>(f.p + x * st + z);
  }
  return e;
}

}  // namespace tff
