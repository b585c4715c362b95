// Batched 2-D FFT operator of the viscoacoustic equation
// (seistorch/equations2d/vacoustic_habc.py:95-111):
//   K(x) = real(ifft2(|k| fft2(x))),  |k| = sqrt(fz^2 + fx^2),
// fz = fftfreq(nz, h), fx = fftfreq(nx, h) (cycles per metre).  |k| is real
// and even, so K maps real fields to real fields and two shots travel in one
// complex transform (shot 2p as the real part, 2p+1 as the imaginary part).
//
// Three launches: row transforms (with the input difference and optional
// pre-multiplier), column transforms forward, |k|, inverse (a block of
// columns stays in shared memory), and inverse row transforms with the
// 1/(nz nx) scale and the optional post-multiplier.  An inverse transform is
// the forward one between two conjugations.
//
// A transform is a sequence of Stockham autosort passes: a thread loads the R
// inputs of one radix-R butterfly, multiplies them by twiddles from a table
// (built in double precision), transforms them in registers and stores the R
// outputs.  The first pass reads and the last pass writes global memory
// directly, the passes between ping-pong in shared memory.  Radices 2, 3, 4,
// 5, 7, 8, 10, 11 and 13; a prime factor of 17 to 137 is a pass over shared
// memory (prime_pass: 228 x 356 with 8 shots 48 us where chirp-z takes 94); a
// length with a larger one is a chirp-z (Bluestein) convolution of the next product
// of the radices at or above 2n - 1, whose chirp and kernel spectrum sit in the
// table too.  Lengths whose convolution does not fit in shared memory (above about
// 7000, with a prime factor above 137) take the general kernels at the end, one
// output of a stage at a time.
//
// Rounding: on white noise the operator's error is at most that of direct sums over
// the prime factors at every length of 100 to 1300 (a transform 0.9 to 1.4e-7 of the
// norm, with chirp-z 1.9 to 2.5e-7), on smooth fields 0.55 to 1.06 of it.  What that
// takes beside the choice above is said where it stands: the sine of radix 5, the
// chains of radix 3, the twiddles of some lengths.
//
// What bounds it: latency of the first pass' global loads and of the twiddle
// loads (rows, 44 % of the warps resident), barriers between the passes of a
// column block (3 CTAs of 64 KB per SM); DRAM and L2 stay below 20 %, the
// fields of the loop fit in L2.  16 shots of 500 x 1100 take 146 us, about a third
// each (rows, columns, rows); one output of a stage per thread from its R inputs
// with two run-time divisions each took 115 / 494 / 115 us.  64 registers (four CTAs of 256 threads) where the
// compiler would take up to 128: rows 61 and 53 us with those.
#include <cmath>

#include "sgb_common.cuh"

namespace sgb {
namespace {

constexpr int FFT_MAX_N = 8192;
constexpr int FFT_MAX_RAD = 24;

struct FftFactors {
  int n, nrad;
  int rad[FFT_MAX_RAD];
  int fine;  // twiddles to twice the precision (see plan_axis)
  unsigned inv[FFT_MAX_RAD];  // register passes: ceil(2^32 / Ns) of the pass (Ns > 1)
};

// Prime factors (4s first) for the general kernels.
FftFactors factorize(int n) {
  FftFactors f;
  f.n = n;
  f.nrad = 0;
  for (int p : {4, 2, 3, 5, 7}) {
    while (n % p == 0 && f.nrad < FFT_MAX_RAD) {
      f.rad[f.nrad++] = p;
      n /= p;
    }
  }
  for (int p = 11; n > 1 && f.nrad < FFT_MAX_RAD; p += 2) {
    while (n % p == 0 && f.nrad < FFT_MAX_RAD) {
      f.rad[f.nrad++] = p;
      n /= p;
    }
  }
  if (n > 1) f.nrad = -1;  // cannot happen for n <= FFT_MAX_N
  return f;
}

// The largest radix transformed in registers, and the largest prime taken by
// prime_pass.  A chirp-z convolution is two transforms of more than twice the
// length: its error is 1.0 to 1.9 times that of direct sums over the factors up to
// about 130, and smaller above (0.75 to 0.96 from 139, 0.55 at 389).
constexpr int FFT_REG = 13, FFT_MAX_PRIME = 137;

// Radices of the passes; false if n has a prime factor above FFT_REG (or, with
// `primes`, above FFT_MAX_PRIME).  Odd radices come first: the first pass stores
// with stride R, which is free of bank conflicts for odd R.
bool pass_radices(int n, bool primes, FftFactors* f) {
  int odd[FFT_MAX_RAD], no = 0, even[FFT_MAX_RAD], ne = 0;
  f->n = n;
  f->fine = 0;
  if (primes) {
    int m = n;
    for (int p : {2, 3, 5, 7, 11, 13})
      while (m % p == 0) m /= p;
    for (int p = FFT_REG + 2; p <= FFT_MAX_PRIME; p += 2)
      while (m % p == 0) odd[no++] = p, m /= p, n /= p;
  }
  for (int p : {13, 11, 7})
    while (n % p == 0) odd[no++] = p, n /= p;
  int twos = 0, fives = 0;
  while (n % 2 == 0) ++twos, n /= 2;
  while (n % 5 == 0) ++fives, n /= 5;
  while (n % 3 == 0) odd[no++] = 3, n /= 3;
  if (n > 1) return false;
  // pair 2s with 5s as often as gives the fewest passes (8 = three 2s)
  int tens = 0, best = 1 << 30;
  for (int t = 0; t <= twos && t <= fives; ++t)
    if (fives + (twos - t + 2) / 3 < best) best = fives + (twos - t + 2) / 3, tens = t;
  for (int t = 0; t < tens; ++t) even[ne++] = 10, --twos, --fives;
  while (fives > 0) odd[no++] = 5, --fives;
  while (twos >= 3 && twos != 4) even[ne++] = 8, twos -= 3;
  while (twos >= 2) even[ne++] = 4, twos -= 2;
  if (twos > 0) even[ne++] = 2;
  f->nrad = 0;
  for (int i = 0; i < no; ++i) f->rad[f->nrad++] = odd[i];
  for (int i = 0; i < ne; ++i) f->rad[f->nrad++] = even[i];
  if (f->nrad == 0) f->rad[f->nrad++] = 1;
  long long Ns = 1;
  for (int i = 0; i < f->nrad; ++i) {
    // floor(j / Ns) = (j * inv) >> 32 while j * Ns < 2^32; j and Ns stay below 2^14
    f->inv[i] = Ns > 1 ? (unsigned)(((1LL << 32) + Ns - 1) / Ns) : 0u;
    Ns *= f->rad[i];
  }
  return true;
}

// One axis: length n, passes of length f.n (n, or the chirp-z length M), and
// where its tables start in the table buffer (in float2).
struct FftAxis {
  int n, chirp;         // chirp: 1 for chirp-z
  FftFactors f;         // passes; f.nrad = 0: general kernels
  int tw, ch, bh;       // W_{f.n}^m [f.n] (fine: and its rounding error [f.n]), chirp [n], kernel spectrum / M [M]
};

// The largest pass length whose two buffers fit in a CTA's shared memory.
constexpr int FFT_MAX_PASS = 13824;

FftAxis plan_axis(int n, int at) {
  FftAxis x;
  x.n = n;
  x.chirp = 0;
  x.tw = at;
  x.ch = x.bh = 0;
  x.f.fine = 0;
  if (pass_radices(n, true, &x.f)) {
    // Twiddling and transforming apart rounds once more than summing the products
    // with the roots of unity.  Lengths of 3s beside 5s and 4s or 8s would have 1 to 4 %
    // more error for it and get the tables' rounding errors added back; the others
    // are below without (500 x 1100 would take 9 % more time).
    bool three = false, four = false, five = false;
    for (int i = 0; i < x.f.nrad; ++i) {
      const int r = x.f.rad[i];
      three |= r == 3;
      four |= r == 4 || r == 8;
      five |= r == 5;
    }
    x.f.fine = three && four && five && x.f.rad[0] <= FFT_REG;
    return x;
  }
  // the chirp-z length of least work: points times passes
  long long best = -1;
  FftFactors f;
  for (int m = 2 * n - 1; m <= FFT_MAX_PASS && m < 3 * n; ++m)
    if (pass_radices(m, false, &f) && (best < 0 || (long long)m * (f.nrad + 1) < best)) {
      best = (long long)m * (f.nrad + 1);
      x.f = f;
    }
  if (best < 0) {
    x.f.n = n;
    x.f.nrad = 0;
    return x;
  }
  x.chirp = 1;
  x.ch = at + x.f.n;
  x.bh = x.ch + n;
  return x;
}
int axis_entries(const FftAxis& x) { return x.chirp ? 2 * x.f.n + x.n : (x.f.fine ? 2 : 1) * x.n; }

// How an axis is transformed: passes in registers (FINE: with twiddles to twice the
// precision), prime passes among them, or chirp-z.  Kernels of their own: one for
// the first three would take 160 us where the first takes 146 (500 x 1100).
enum { REGISTER, FINE, PRIME, CHIRP, MODES };
int axis_mode(const FftAxis& x) {
  if (x.chirp) return CHIRP;
  if (x.f.nrad > 0 && x.f.rad[0] > FFT_REG) return PRIME;
  return x.f.fine ? FINE : REGISTER;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {  // a * conj(b)
  return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 conj2(float2 a) { return make_float2(a.x, -a.y); }

// cos / sin of 2 pi k / R at compile time (Taylor series on [-pi, pi]).
constexpr double trig_series(double x, bool sine) {
  double term = sine ? x : 1.0, sum = term;
  for (int i = 1; i < 24; ++i) {
    const int k = sine ? 2 * i : 2 * i - 1;
    term = -term * x * x / (k * (k + 1.0));
    sum += term;
  }
  return sum;
}
constexpr double turn(int k, int R) { return 6.283185307179586476925 * (2 * k > R ? k - R : k) / R; }
template <int R>
struct Trig {
  float c[R], s[R], sl[R];  // and the rounding errors of the sines
  constexpr Trig() : c(), s(), sl() {
    for (int k = 0; k < R; ++k) {
      const double sd = trig_series(turn(k, R), true);
      c[k] = (float)trig_series(turn(k, R), false);
      s[k] = (float)sd;
      sl[k] = (float)(sd - (double)s[k]);
    }
  }
};

// In-place forward DFT of R values in registers: an odd prime from the sums
// and differences of its conjugate pairs, 4 and 8 from halves, 10 as the
// coprime product 2 x 5 (no twiddles).
template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const float2 t = v[0];
    v[0] = cadd(t, v[1]);
    v[1] = csub(t, v[1]);
  } else if constexpr (R == 4) {
    const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
    v[0] = cadd(a, c);
    v[2] = csub(a, c);
    v[1] = make_float2(b.x + d.y, b.y - d.x);
    v[3] = make_float2(b.x - d.y, b.y + d.x);
  } else if constexpr (R == 8) {
    float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft<4>(e);
    dft<4>(o);
    constexpr double hd = 0.70710678118654752440;
    constexpr float h = (float)hd, hl = (float)(hd - (double)h);
    auto half = [&](float t) -> float { return fmaf(h, t, hl * t); };
    o[1] = make_float2(half(o[1].x + o[1].y), half(o[1].y - o[1].x));
    o[2] = make_float2(o[2].y, -o[2].x);
    o[3] = make_float2(half(o[3].y - o[3].x), -half(o[3].x + o[3].y));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = cadd(e[k], o[k]);
      v[k + 4] = csub(e[k], o[k]);
    }
  } else if constexpr (R == 10) {
    float2 a[5], b[5];  // n = 5 n1 + 2 n2 mod 10
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      a[i] = cadd(v[(2 * i) % 10], v[(2 * i + 5) % 10]);
      b[i] = csub(v[(2 * i) % 10], v[(2 * i + 5) % 10]);
    }
    dft<5>(a);
    dft<5>(b);
#pragma unroll
    for (int k = 0; k < 10; ++k) v[k] = (k & 1) ? b[k % 5] : a[k % 5];
  } else {
    constexpr Trig<R> t;
    constexpr int H = (R - 1) / 2;
    float2 s[H], d[H];
    const float2 x0 = v[0];
    float2 sum = x0;
#pragma unroll
    for (int p = 1; p <= H; ++p) {
      s[p - 1] = cadd(v[p], v[R - p]);
      d[p - 1] = csub(v[p], v[R - p]);
      sum = cadd(sum, s[p - 1]);
    }
    v[0] = sum;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      float2 a = x0, b = make_float2(0.f, 0.f);
#pragma unroll
      for (int p = 1; p <= H; ++p) {
        const int e = (k * p) % R;
        const float c = t.c[e], sn = t.s[e];
        if constexpr (R == 5) {  // sin 72 degrees is rounded by 0.4 units in the last place, the others by 0.15
          if (e == 1 || e == 4) {
            b.x = fmaf(t.sl[e], d[p - 1].x, b.x);
            b.y = fmaf(t.sl[e], d[p - 1].y, b.y);
          }
        }
        a.x = fmaf(c, s[p - 1].x, a.x);
        a.y = fmaf(c, s[p - 1].y, a.y);
        b.x = fmaf(sn, d[p - 1].x, b.x);
        b.y = fmaf(sn, d[p - 1].y, b.y);
      }
      v[k] = make_float2(a.x + b.y, a.y - b.x);
      v[R - k] = make_float2(a.x - b.y, a.y + b.x);
    }
  }
}

// Layout of the G transforms of a CTA in shared memory and over its threads:
// rows one after another, a thread row each (block T x G); columns
// interleaved, a thread column each (block G x T).
template <bool ROWS>
struct Lay {
  int M, G;
  __device__ __forceinline__ int at(int i, int c) const { return ROWS ? c * M + i : i * G + c; }
  __device__ __forceinline__ int c() const { return ROWS ? threadIdx.y : threadIdx.x; }
  __device__ __forceinline__ int j0() const { return ROWS ? threadIdx.x : threadIdx.y; }
  __device__ __forceinline__ int step() const { return ROWS ? blockDim.x : blockDim.y; }
};

// v times the root of unity at w (FINE: whose rounding error is M entries further on).
template <bool FINE>
__device__ __forceinline__ float2 twiddle(float2 v, const float2* __restrict__ w, int M) {
  const float2 h = __ldg(w);
  if constexpr (!FINE) return make_float2(fmaf(v.x, h.x, -(v.y * h.y)), fmaf(v.y, h.x, v.x * h.y));
  const float2 l = __ldg(w + M);
  const float ex = fmaf(v.x, l.x, -v.y * l.y), ey = fmaf(v.x, l.y, v.y * l.x);
  return make_float2(fmaf(v.x, h.x, fmaf(-v.y, h.y, ex)), fmaf(v.x, h.y, fmaf(v.y, h.x, ey)));
}

// One pass: inputs from in(i, c), outputs to out(i, c, v).
template <int R, bool FINE, bool ROWS, class In, class Out>
__device__ __forceinline__ void fft_pass(const Lay<ROWS>& L, int Ns, unsigned inv, const float2* __restrict__ tw,
                                         const In& in, const Out& out) {
  const int nb = L.M / R, span = Ns * R, tws = L.M / span, c = L.c();
  for (int j = L.j0(); j < nb; j += L.step()) {
    const int blk = Ns > 1 ? (int)__umulhi((unsigned)j, inv) : j, m = j - blk * Ns, o = blk * span + m;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = in(j + r * nb, c);
    if constexpr (R == 3) {
      // twiddle and butterfly in one chain of fused operations per output: lengths
      // of many 3s have as many passes, and rounding twiddled inputs, their sums and
      // the outputs apart cost 5 to 11 % in error (8 shots of 216 x 972: 71 us a
      // transform of the field with the chains, 56 without)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int e = m * tws + q * nb;
        const float2 w1 = __ldg(tw + e), w2 = __ldg(tw + (2 * e < L.M ? 2 * e : 2 * e - L.M));
        out(o + q * Ns, c,
            make_float2(v[0].x + fmaf(-v[2].y, w2.y, fmaf(v[2].x, w2.x, fmaf(-v[1].y, w1.y, v[1].x * w1.x))),
                        v[0].y + fmaf(v[2].y, w2.x, fmaf(v[2].x, w2.y, fmaf(v[1].y, w1.x, v[1].x * w1.y)))));
      }
    } else {
      if (Ns > 1) {
        const float2* w = tw;
#pragma unroll
        for (int r = 1; r < R; ++r) {
          w += m * tws;
          v[r] = twiddle<FINE>(v[r], w, L.M);
        }
      }
      dft<R>(v);
#pragma unroll
      for (int q = 0; q < R; ++q) out(o + q * Ns, c, v[q]);
    }
  }
}

// A pass of prime radix R, 17 .. FFT_MAX_PRIME: sums and differences of the
// conjugate pairs (twiddled) into `mid`, then every output pair (k, R - k) from
// them, PR_K pairs per thread so that a pair's values are read once for all.
constexpr int PR_K = 4;
__host__ __device__ inline int prime_groups(int R) { return ((R + 1) / 2 + PR_K - 1) / PR_K; }
template <bool ROWS, class In, class Out>
__device__ __forceinline__ void prime_pass(const Lay<ROWS>& L, int R, int Ns, unsigned inv, const float2* __restrict__ tw,
                                           float2* mid, const In& in, const Out& out) {
  __shared__ float2 root[FFT_MAX_PRIME];  // W_R^e
  const int nb = L.M / R, span = Ns * R, tws = L.M / span, H = (R - 1) / 2, c = L.c();
  for (int i = threadIdx.y * blockDim.x + threadIdx.x; i < R; i += blockDim.x * blockDim.y) root[i] = __ldg(tw + i * nb);
  for (int u = L.j0(); u < (H + 1) * nb; u += L.step()) {  // u = j + p nb
    const int p = u / nb, j = u - p * nb;
    float2 a = in(u, c);
    if (p > 0) {
      const int t = j + (R - p) * nb;
      float2 b = in(t, c);
      if (Ns > 1) {
        const int m = (j - (int)__umulhi((unsigned)j, inv) * Ns) * tws;
        a = cmul(a, __ldg(tw + p * m));
        b = cmul(b, __ldg(tw + (R - p) * m));
      }
      mid[L.at(t, c)] = csub(a, b);
      a = cadd(a, b);
    }
    mid[L.at(u, c)] = a;
  }
  __syncthreads();
  for (int u = L.j0(); u < prime_groups(R) * nb; u += L.step()) {
    const int k0 = u / nb * PR_K, j = u - u / nb * nb;
    const int blk = Ns > 1 ? (int)__umulhi((unsigned)j, inv) : j, o = blk * span + (j - blk * Ns);
    float2 a[PR_K], b[PR_K];
    int e[PR_K];  // k p mod R
#pragma unroll
    for (int q = 0; q < PR_K; ++q) {
      a[q] = mid[L.at(j, c)];
      b[q] = make_float2(0.f, 0.f);
      e[q] = 0;
    }
    for (int p = 1; p <= H; ++p) {
      const float2 s = mid[L.at(j + p * nb, c)], d = mid[L.at(j + (R - p) * nb, c)];
#pragma unroll
      for (int q = 0; q < PR_K; ++q) {
        e[q] += k0 + q;  // below R: k0 + q <= H + 3
        e[q] -= e[q] >= R ? R : 0;
        const float2 w = root[e[q]];
        a[q].x = fmaf(w.x, s.x, a[q].x);
        a[q].y = fmaf(w.x, s.y, a[q].y);
        b[q].x = fmaf(w.y, d.x, b[q].x);
        b[q].y = fmaf(w.y, d.y, b[q].y);
      }
    }
#pragma unroll
    for (int q = 0; q < PR_K; ++q) {
      const int k = k0 + q;
      if (k > H) break;
      out(o + k * Ns, c, make_float2(a[q].x - b[q].y, a[q].y + b[q].x));
      if (k > 0) out(o + (R - k) * Ns, c, make_float2(a[q].x + b[q].y, a[q].y - b[q].x));
    }
  }
}

// All passes of G length-f.n transforms: the first reads in(i, c, cur), the
// last calls out(i, c, v, dst); between them cur / nxt ping-pong (a prime pass
// goes through nxt and back).  On return cur is the buffer that out could store
// to, visible to the CTA.
template <int MODE, bool ROWS, class In, class Out>
__device__ __forceinline__ void fft_passes(const FftFactors& f, const Lay<ROWS>& L, const float2* __restrict__ tw,
                                           float2*& cur, float2*& nxt, const In& in, const Out& out) {
  int Ns = 1;
  for (int s = 0; s < f.nrad; ++s) {
    const bool first = s == 0, last = s == f.nrad - 1;
    const bool prime = MODE == PRIME && f.rad[s] > FFT_REG;
    const float2* src = cur;
    float2* dst = prime ? cur : nxt;
    auto rd = [&](int i, int c) -> float2 { return first ? in(i, c, src) : src[L.at(i, c)]; };
    auto wr = [&](int i, int c, float2 v) {
      if (last)
        out(i, c, v, dst);
      else
        dst[L.at(i, c)] = v;
    };
    switch (f.rad[s]) {
      case 1: fft_pass<1, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      case 2: fft_pass<2, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      case 3: fft_pass<3, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      case 4: fft_pass<4, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      case 5: fft_pass<5, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      case 7: fft_pass<7, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      case 8: fft_pass<8, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      case 10: fft_pass<10, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      case 11: fft_pass<11, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      case 13: fft_pass<13, MODE == FINE>(L, Ns, f.inv[s], tw, rd, wr); break;
      default:
        if constexpr (MODE == PRIME) prime_pass(L, f.rad[s], Ns, f.inv[s], tw, nxt, rd, wr);
    }
    __syncthreads();
    Ns *= f.rad[s];
    if (!prime) {
      float2* t = cur;
      cur = nxt;
      nxt = t;
    }
  }
}

// The length-n DFT of an axis: its passes, or (CHIRP) the chirp-z convolution
// X[k] = c[k] sum_j (x[j] c[j]) conj(c)[k - j], c[j] = exp(-i pi j^2 / n), by
// two length-M transforms.
template <bool ROWS, int MODE, class In, class Out>
__device__ __forceinline__ void axis_dft(const FftAxis& x, const float2* __restrict__ tab, int G, float2*& cur,
                                         float2*& nxt, const In& in, const Out& out) {
  const Lay<ROWS> L{x.f.n, G};
  const float2* tw = tab + x.tw;
  if constexpr (MODE != CHIRP) {
    fft_passes<MODE>(x.f, L, tw, cur, nxt, in, out);
  } else {
    const float2* ch = tab + x.ch;
    const float2* bh = tab + x.bh;
    fft_passes<CHIRP>(
        x.f, L, tw, cur, nxt,
        [&](int i, int c, const float2* src) -> float2 {
          return i < x.n ? cmul(in(i, c, src), __ldg(ch + i)) : make_float2(0.f, 0.f);
        },
        [&](int i, int c, float2 v, float2* dst) { dst[L.at(i, c)] = conj2(cmul(v, __ldg(bh + i))); });
    fft_passes<CHIRP>(
        x.f, L, tw, cur, nxt, [&](int i, int c, const float2* src) -> float2 { return src[L.at(i, c)]; },
        [&](int i, int c, float2 v, float2* dst) {
          if (i < x.n) out(i, c, cmul(conj2(v), __ldg(ch + i)), dst);
        });
  }
}

struct KArgs {
  int nz, nx, pitch, nshots, npairs;
  long long sstride;
  float h;
  const float* __restrict__ pre;   // [nz][pitch] or null
  const float* __restrict__ u1;    // [nshots][nz][pitch]
  const float* __restrict__ u2;    // [nshots][nz][pitch] or null
  const float* __restrict__ post;  // [nz][pitch] or null
  float* __restrict__ out;         // [nshots][nz][pitch]
  float2* __restrict__ work;       // [npairs][nz][nx]
  const float2* __restrict__ tab;  // tables of both axes
  FftAxis az, ax;
  int G;                           // rows / columns per CTA
  FftFactors fz, fx;               // general kernels only
};

// W_M^m of an axis' passes, its rounding error (fine) and, for chirp-z, c[j] = exp(-i pi j^2 / n).
__global__ void table_kernel(float2* tab, const FftAxis x) {
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < x.f.n; m += gridDim.x * blockDim.x) {
    double s, c;
    sincospi(-2.0 * (double)m / (double)x.f.n, &s, &c);
    tab[x.tw + m] = make_float2((float)c, (float)s);
    if (x.f.fine) tab[x.tw + x.f.n + m] = make_float2((float)(c - (double)(float)c), (float)(s - (double)(float)s));
    if (x.chirp && m < x.n) {
      sincospi(-(double)((long long)m * m % (2LL * x.n)) / (double)x.n, &s, &c);
      tab[x.ch + m] = make_float2((float)c, (float)s);
    }
  }
}

// Spectrum over M of the chirp-z kernel b[j] = b[M - j] = conj(c[j]), 1 / M included.
__global__ void __launch_bounds__(256) chirp_spectrum_kernel(float2* tab, const FftAxis x) {
  extern __shared__ float2 sm[];
  const int M = x.f.n;
  float2 *cur = sm, *nxt = sm + M;
  const float inv = 1.f / (float)M;
  fft_passes<CHIRP>(
      x.f, Lay<true>{M, 1}, tab + x.tw, cur, nxt,
      [&](int i, int, const float2*) -> float2 {
        const int j = i < x.n ? i : M - i;
        return j < x.n ? conj2(tab[x.ch + j]) : make_float2(0.f, 0.f);
      },
      [&](int i, int, float2 v, float2*) { tab[x.bh + i] = make_float2(inv * v.x, inv * v.y); });
}

// Forward row transforms of the packed pair (shot 2p + i shot 2p+1).
template <int MODE>
__global__ void __launch_bounds__(256, 4) k_rows_fwd_kernel(const KArgs a) {
  extern __shared__ float2 sm[];
  pdl_wait();
  pdl_trigger();
  const int z = blockIdx.x * a.G + threadIdx.y, p = blockIdx.y;
  const bool in_z = z < a.nz, two = 2 * p + 1 < a.nshots;
  const long long ro = (long long)(in_z ? z : 0) * a.pitch, f0 = 2LL * p * a.sstride + ro;
  const float* ua = a.u1 + f0;
  const float* ub = a.u1 + (two ? f0 + a.sstride : f0);
  const float* va = a.u2 ? a.u2 + f0 : nullptr;
  const float* vb = a.u2 ? a.u2 + (two ? f0 + a.sstride : f0) : nullptr;
  const float* pre = a.pre ? a.pre + ro : nullptr;
  float2 *cur = sm, *nxt = sm + a.G * a.ax.f.n;
  float2* w = a.work + ((long long)p * a.nz + (in_z ? z : 0)) * a.nx;
  axis_dft<true, MODE>(
      a.ax, a.tab, a.G, cur, nxt,
      [&](int x, int, const float2*) -> float2 {
        float re = ldf(ua + x), im = ldf(ub + x);
        if (va) {
          re -= ldf(va + x);
          im -= ldf(vb + x);
        }
        const float s = pre ? __ldg(pre + x) : 1.f;
        return make_float2(s * re, two ? s * im : 0.f);
      },
      [&](int x, int, float2 v, float2*) {
        if (in_z) w[x] = v;
      });
}

// Column transforms of G adjacent columns: forward, times |k|, inverse.
template <int MODE>
__global__ void __launch_bounds__(256, 4) k_cols_kernel(const KArgs a) {
  extern __shared__ float2 sm[];
  pdl_wait();
  pdl_trigger();
  const int G = a.G, x0 = blockIdx.x * G;
  const int xg = x0 + threadIdx.x;
  const bool in_x = xg < a.nx;
  float2* w = a.work + (long long)blockIdx.y * a.nz * a.nx + (in_x ? xg : x0);
  float2 *cur = sm, *nxt = sm + G * a.az.f.n;
  const float inv_nzh = 1.f / (a.nz * a.h), inv_nxh = 1.f / (a.nx * a.h);
  const float fx = (xg < (a.nx + 1) / 2 ? xg : xg - a.nx) * inv_nxh;  // fftfreq
  const Lay<false> L{a.az.f.n, G};
  axis_dft<false, MODE>(
      a.az, a.tab, G, cur, nxt,
      [&](int z, int, const float2*) -> float2 {
        const float2* q = w + (long long)z * a.nx;
        float2 v;
        asm volatile("ld.global.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "l"(q));
        return v;
      },
      [&](int z, int c, float2 v, float2* dst) {
        const float fz = (z < (a.nz + 1) / 2 ? z : z - a.nz) * inv_nzh;
        const float kk = sqrtf(fz * fz + fx * fx);
        dst[L.at(z, c)] = make_float2(kk * v.x, -kk * v.y);
      });
  axis_dft<false, MODE>(
      a.az, a.tab, G, cur, nxt, [&](int z, int c, const float2* src) -> float2 { return src[L.at(z, c)]; },
      [&](int z, int, float2 v, float2*) {
        if (in_x) w[(long long)z * a.nx] = conj2(v);
      });
}

// Inverse row transforms, 1/(nz nx), optional post-multiplier, unpacking.
template <int MODE>
__global__ void __launch_bounds__(256, 4) k_rows_inv_kernel(const KArgs a) {
  extern __shared__ float2 sm[];
  pdl_wait();
  pdl_trigger();
  const int z = blockIdx.x * a.G + threadIdx.y, p = blockIdx.y;
  const bool in_z = z < a.nz, two = 2 * p + 1 < a.nshots;
  const long long ro = (long long)(in_z ? z : 0) * a.pitch, f0 = 2LL * p * a.sstride + ro;
  float* oa = a.out + f0;
  float* ob = a.out + f0 + a.sstride;
  const float* post = a.post ? a.post + ro : nullptr;
  float2 *cur = sm, *nxt = sm + a.G * a.ax.f.n;
  const float2* w = a.work + ((long long)p * a.nz + (in_z ? z : 0)) * a.nx;
  const float scale = 1.f / ((float)a.nz * (float)a.nx);
  axis_dft<true, MODE>(
      a.ax, a.tab, a.G, cur, nxt,
      [&](int x, int, const float2*) -> float2 {
        float2 v;
        asm volatile("ld.global.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "l"(w + x));
        return conj2(v);
      },
      [&](int x, int, float2 v, float2*) {
        const float s = scale * (post ? __ldg(post + x) : 1.f);
        if (in_z) oa[x] = s * v.x;
        if (in_z && two) ob[x] = -s * v.y;
      });
  if (in_z)
    for (int x = a.nx + threadIdx.x; x < a.pitch; x += blockDim.x) {  // padding columns get 0
      oa[x] = 0.f;
      if (two) ob[x] = 0.f;
    }
}

// ---------------------------------------------------- general kernels ---

// All stages of G length-n transforms laid out [n][G] in shared memory
// (a: input, b: scratch).  tw[m] = exp(-2 pi i m / n); inverse uses conj.
// Returns the buffer that holds the result.
__device__ float2* fft_stages(float2* a, float2* b, const float2* tw, const FftFactors& f, int G, bool inverse) {
  const int n = f.n;
  int Ns = 1;
  for (int s = 0; s < f.nrad; ++s) {
    const int R = f.rad[s], step = n / R, span = Ns * R, tws = n / span;
    for (int t = threadIdx.x; t < n * G; t += blockDim.x) {
      const int o = t / G, c = t - o * G;
      const int blk = o / span, rem = o - blk * span;
      const int j = blk * Ns + rem % Ns;
      float2 acc = make_float2(0.f, 0.f);
      int e = 0;  // r * rem mod span
      for (int r0 = 0; r0 < R; r0 += 64) {  // blocks of 64 terms: the rounding of a long sum stays that of its blocks
        float2 part = make_float2(0.f, 0.f);
        for (int r = r0; r < min(R, r0 + 64); ++r) {
          const float2 x = a[(j + r * step) * G + c];
          const float2 w = tw[e * tws];
          const float2 p = inverse ? cmulc(x, w) : cmul(x, w);
          part.x += p.x;
          part.y += p.y;
          e += rem;
          if (e >= span) e -= span;
        }
        acc.x += part.x;
        acc.y += part.y;
      }
      b[o * G + c] = acc;
    }
    __syncthreads();
    float2* t = a;
    a = b;
    b = t;
    Ns *= R;
  }
  return a;
}

// Forward row transforms of the packed pair (shot 2p + i shot 2p+1).
__global__ void __launch_bounds__(256) g_rows_fwd_kernel(const KArgs a) {
  extern __shared__ float2 sm[];
  const int n = a.nx;
  float2* A = sm;
  float2* B = sm + n;
  float2* T = sm + 2 * n;
  const int z = blockIdx.x, p = blockIdx.y;
  const int b0 = 2 * p, b1 = 2 * p + 1;
  const long long ro = (long long)z * a.pitch;
  for (int x = threadIdx.x; x < n; x += blockDim.x) {
    T[x] = a.tab[a.ax.tw + x];
    const float s = a.pre ? a.pre[ro + x] : 1.f;
    float re = a.u1[b0 * a.sstride + ro + x], im = 0.f;
    if (a.u2) re -= a.u2[b0 * a.sstride + ro + x];
    if (b1 < a.nshots) {
      im = a.u1[b1 * a.sstride + ro + x];
      if (a.u2) im -= a.u2[b1 * a.sstride + ro + x];
    }
    A[x] = make_float2(s * re, s * im);
  }
  __syncthreads();
  const float2* r = fft_stages(A, B, T, a.fx, 1, false);
  float2* w = a.work + ((long long)p * a.nz + z) * a.nx;
  for (int x = threadIdx.x; x < n; x += blockDim.x) w[x] = r[x];
}

// Column transforms of G adjacent columns: forward, times |k|, inverse.
__global__ void __launch_bounds__(256) g_cols_kernel(const KArgs a, int G) {
  extern __shared__ float2 sm[];
  const int n = a.nz;
  float2* A = sm;
  float2* B = sm + n * G;
  float2* T = sm + 2 * n * G;
  const int x0 = blockIdx.x * G, p = blockIdx.y;
  const int gw = min(G, a.nx - x0);
  float2* w = a.work + (long long)p * a.nz * a.nx;
  for (int i = threadIdx.x; i < n; i += blockDim.x) T[i] = a.tab[a.az.tw + i];
  for (int t = threadIdx.x; t < n * G; t += blockDim.x) {
    const int z = t / G, c = t - z * G;
    A[t] = c < gw ? w[(long long)z * a.nx + x0 + c] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  float2* r = fft_stages(A, B, T, a.fz, G, false);
  float2* o = (r == A) ? B : A;
  const float inv_nzh = 1.f / (a.nz * a.h), inv_nxh = 1.f / (a.nx * a.h);
  for (int t = threadIdx.x; t < n * G; t += blockDim.x) {
    const int z = t / G, c = t - z * G;
    const int xg = x0 + c;
    const int iz = z < (a.nz + 1) / 2 ? z : z - a.nz;    // fftfreq index
    const int ix = xg < (a.nx + 1) / 2 ? xg : xg - a.nx;
    const float fz = iz * inv_nzh, fx = ix * inv_nxh;
    const float kk = sqrtf(fz * fz + fx * fx);
    r[t] = make_float2(kk * r[t].x, kk * r[t].y);
  }
  __syncthreads();
  r = fft_stages(r, o, T, a.fz, G, true);
  for (int t = threadIdx.x; t < n * G; t += blockDim.x) {
    const int z = t / G, c = t - z * G;
    if (c < gw) w[(long long)z * a.nx + x0 + c] = r[t];
  }
}

// Inverse row transforms, 1/(nz nx), optional post-multiplier, unpacking.
__global__ void __launch_bounds__(256) g_rows_inv_kernel(const KArgs a) {
  extern __shared__ float2 sm[];
  const int n = a.nx;
  float2* A = sm;
  float2* B = sm + n;
  float2* T = sm + 2 * n;
  const int z = blockIdx.x, p = blockIdx.y;
  const float2* w = a.work + ((long long)p * a.nz + z) * a.nx;
  for (int x = threadIdx.x; x < n; x += blockDim.x) {
    T[x] = a.tab[a.ax.tw + x];
    A[x] = w[x];
  }
  __syncthreads();
  const float2* r = fft_stages(A, B, T, a.fx, 1, true);
  const float scale = 1.f / ((float)a.nz * (float)a.nx);
  const int b0 = 2 * p, b1 = 2 * p + 1;
  const long long ro = (long long)z * a.pitch;
  for (int x = threadIdx.x; x < a.pitch; x += blockDim.x) {
    float re = 0.f, im = 0.f;
    if (x < n) {
      const float s = scale * (a.post ? a.post[ro + x] : 1.f);
      re = s * r[x].x;
      im = s * r[x].y;
    }
    a.out[b0 * a.sstride + ro + x] = re;  // padding columns get 0
    if (b1 < a.nshots) a.out[b1 * a.sstride + ro + x] = im;
  }
}

}  // namespace

// The kernels of each axis mode.
static const struct {
  void (*rows_fwd[MODES])(KArgs);
  void (*cols[MODES])(KArgs);
  void (*rows_inv[MODES])(KArgs);
} KERNELS = {
    {k_rows_fwd_kernel<REGISTER>, k_rows_fwd_kernel<FINE>, k_rows_fwd_kernel<PRIME>, k_rows_fwd_kernel<CHIRP>},
    {k_cols_kernel<REGISTER>, k_cols_kernel<FINE>, k_cols_kernel<PRIME>, k_cols_kernel<CHIRP>},
    {k_rows_inv_kernel<REGISTER>, k_rows_inv_kernel<FINE>, k_rows_inv_kernel<PRIME>, k_rows_inv_kernel<CHIRP>}};

// Shared-memory bytes of the general column launch for G columns.
static size_t cols_smem(int nz, int G) { return (size_t)(2 * nz * G + nz) * sizeof(float2); }

int64_t vacoustic_table_floats(const sgb_grid& g) {
  const FftAxis z = plan_axis(g.nz, 0);
  return 2LL * (axis_entries(z) + axis_entries(plan_axis(g.nx, 0)));
}

// K(pre * (u1 - u2)) * post; `tables` false: the tables in tw are those of an
// earlier call for the same grid.
int vacoustic_kterm(const sgb_grid& g, const float* pre, const float* u1, const float* u2, const float* post,
                    float* out, float* work, float* tw, cudaStream_t s, bool tables) {
  if (g.nz > FFT_MAX_N || g.nx > FFT_MAX_N) return SGB_ERR_UNSUPPORTED;
  KArgs a;
  a.nz = g.nz;
  a.nx = g.nx;
  a.pitch = g.pitch;
  a.nshots = g.nshots;
  a.npairs = (g.nshots + 1) / 2;
  a.sstride = (long long)g.nz * g.pitch;
  a.h = g.h;
  a.pre = pre;
  a.u1 = u1;
  a.u2 = u2;
  a.post = post;
  a.out = out;
  a.work = reinterpret_cast<float2*>(work);
  float2* tab = reinterpret_cast<float2*>(tw);
  a.tab = tab;
  a.az = plan_axis(g.nz, 0);
  a.ax = plan_axis(g.nx, axis_entries(a.az));
  const bool general_z = a.az.f.nrad == 0, general_x = a.ax.f.nrad == 0;
  if (general_z) a.fz = factorize(g.nz);
  if (general_x) a.fx = factorize(g.nx);
  if ((general_z && a.fz.nrad < 0) || (general_x && a.fx.nrad < 0)) return SGB_ERR_UNSUPPORTED;
  constexpr int MAX_SMEM = 224 * 1024;
  static bool attr_set = false;
  if (!attr_set) {
    const void* kernels[] = {(const void*)KERNELS.rows_fwd[0], (const void*)KERNELS.rows_fwd[1],
                             (const void*)KERNELS.rows_fwd[2], (const void*)KERNELS.rows_fwd[3],
                             (const void*)KERNELS.cols[0],     (const void*)KERNELS.cols[1],
                             (const void*)KERNELS.cols[2],     (const void*)KERNELS.cols[3],
                             (const void*)KERNELS.rows_inv[0], (const void*)KERNELS.rows_inv[1],
                             (const void*)KERNELS.rows_inv[2], (const void*)KERNELS.rows_inv[3],
                             (const void*)g_rows_fwd_kernel,   (const void*)g_cols_kernel,
                             (const void*)g_rows_inv_kernel,   (const void*)chirp_spectrum_kernel};
    for (const void* k : kernels)
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM) != cudaSuccess ||
          cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100) != cudaSuccess)
        return set_cuda_error(cudaGetLastError());
    attr_set = true;
  }
  if (tables) {
    for (const FftAxis* x : {&a.az, &a.ax}) {
      table_kernel<<<(x->f.n + 255) / 256, 256, 0, s>>>(tab, *x);
      if (x->chirp) chirp_spectrum_kernel<<<1, 256, (size_t)2 * x->f.n * sizeof(float2), s>>>(tab, *x);
    }
    SGB_CUDA_CHECK(cudaGetLastError());
  }
  // rows: as many threads as the widest pass has work for (up to 256), and
  // rows per CTA to make 128 threads of it where 24 KB hold them; columns: 8
  // per CTA (64-byte segments of a row of the work array), fewer above 112 KB
  const size_t row = (size_t)2 * a.ax.f.n * sizeof(float2), col = (size_t)2 * a.az.f.n * sizeof(float2);
  auto units = [](const FftFactors& f) {  // threads that the widest pass has work for
    int u = 0;
    for (int i = 0; i < f.nrad; ++i) {
      const int n = f.n / f.rad[i] * (f.rad[i] > FFT_REG ? prime_groups(f.rad[i]) : 1);
      u = n > u ? n : u;
    }
    return u > 0 ? u : f.n;
  };
  KArgs r = a, c = a;
  int tr = (units(a.ax.f) + 31) / 32 * 32;
  tr = tr > 256 ? 256 : tr;
  r.G = 1;
  while (r.G * 2 * tr <= 128 && (size_t)r.G * 2 * row <= 24 * 1024) r.G *= 2;
  c.G = 8;
  while (c.G > 1 && c.G * col > 112 * 1024) c.G /= 2;
  const dim3 rg((unsigned)((g.nz + r.G - 1) / r.G), (unsigned)a.npairs);
  const dim3 cg((unsigned)((g.nx + c.G - 1) / c.G), (unsigned)a.npairs);
  const size_t row_general = (size_t)3 * g.nx * sizeof(float2);
  int G = 16;
  while (G > 1 && cols_smem(g.nz, G) > 160 * 1024) G /= 2;
  const int mode_x = axis_mode(a.ax), mode_z = axis_mode(a.az);
  if (general_x)
    g_rows_fwd_kernel<<<dim3((unsigned)g.nz, (unsigned)a.npairs), 256, row_general, s>>>(a);
  else
    SGB_CUDA_CHECK(launch_pdl(KERNELS.rows_fwd[mode_x], rg, dim3(tr, r.G), r.G * row, s, r));
  if (general_z)
    g_cols_kernel<<<dim3((unsigned)((g.nx + G - 1) / G), (unsigned)a.npairs), 256, cols_smem(g.nz, G), s>>>(a, G);
  else
    SGB_CUDA_CHECK(launch_pdl(KERNELS.cols[mode_z], cg, dim3(c.G, 256 / c.G), c.G * col, s, c));
  if (general_x)
    g_rows_inv_kernel<<<dim3((unsigned)g.nz, (unsigned)a.npairs), 256, row_general, s>>>(a);
  else
    SGB_CUDA_CHECK(launch_pdl(KERNELS.rows_inv[mode_x], rg, dim3(tr, r.G), r.G * row, s, r));
  SGB_CUDA_CHECK(cudaGetLastError());
  return SGB_OK;
}

}  // namespace sgb
