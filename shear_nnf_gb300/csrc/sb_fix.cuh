// sb_fix.cuh -- 64-bit block-fixed-point arithmetic for the transforms.
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM sub-partition
// (add 76), but a 32 x 32 + 64 bit integer multiply-add every 2 cycles and a
// 64-bit integer add in 2 (measured).  A discrete Fourier transform needs only
// additions and multiplications by constants of modulus <= 1 on data that share
// one scale, so it runs here on 64-bit integers: the sequence is scaled by a
// power of two taken from its largest component, every sum is exact, and a
// twiddle product keeps the upper 64 bits of the 126-bit product (error about
// one unit).  With 57-60 bits of the largest input at the start the results
// carry an error of about 2^-55 of the rms value of the output, below the
// 2^-53-class error of the FP64 transform it stands in for (measured against
// extended precision in tests/test_fix.py).
//
// Scales.  A twiddle is stored at 2^62 in two signed 32-bit halves; a product
// with one divides by 4 (w z / 4).  A plan (Plan<N>) factors N = R1 R2: with
// n = n2 + R2 n1 and k = k1 + R1 k2,
//   y[n2][k1] = W_N^(n2 k1)/4 * DFT_R1 over n1,   X[k1 + R1 k2] = DFT_R2 over n2
// (the inverse runs DFT_R2 over k2 first and DFT_R1 over k1 last).  The
// 16-point kernel divides by 4 once more inside.  Input components must stay
// below 2^bits(N): then every intermediate is below 2^62.5 in modulus, which
// the 64-bit sums and the cross products of a twiddle product can hold.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define SB_HD __host__ __device__ __forceinline__
#else
#define SB_HD inline
#endif

namespace sb {

typedef long long ll;
typedef unsigned long long ull;

struct alignas(16) q2 {
  ll x, y;
};
// a constant w = (hr + i hi) 2^-30 + (lr + i li) 2^-62
struct alignas(16) qw {
  int hr, lr, hi, li;
};

SB_HD q2 mkq(ll x, ll y) {
  q2 r;
  r.x = x;
  r.y = y;
  return r;
}
SB_HD q2 operator+(q2 a, q2 b) { return mkq(a.x + b.x, a.y + b.y); }
SB_HD q2 operator-(q2 a, q2 b) { return mkq(a.x - b.x, a.y - b.y); }
SB_HD q2 qshr(q2 a, int n) { return mkq(a.x >> n, a.y >> n); }
SB_HD q2 qdbl(q2 a) { return mkq(a.x + a.x, a.y + a.y); }
// S i a
template <int S>
SB_HD q2 qrot(q2 a) {
  return S < 0 ? mkq(a.y, -a.x) : mkq(-a.y, a.x);
}

// halves of a 64-bit integer, both signed: v = h 2^32 + l
SB_HD int qlo(ll v) { return (int)v; }
SB_HD int qhi(ll v) { return (int)(v >> 32) + (int)((unsigned)(int)v >> 31); }

// x (h 2^32 + l) / 2^64, to nearest up to the dropped product of the low halves
SB_HD ll qmulr(ll x, int h, int l) {
  const int xl = qlo(x), xh = qhi(x);
  const ll c = (ll)xl * h + (ll)xh * l + (1ll << 31);
  return (ll)xh * h + (c >> 32);
}

// z w / 4 (CJ false) or z conj(w) / 4
template <bool CJ>
SB_HD q2 qmul(q2 z, int hr, int lr, int hi, int li) {
  const int xl = qlo(z.x), xh = qhi(z.x), yl = qlo(z.y), yh = qhi(z.y);
  const int nh = -hi, nl = -li;
  const int ah = CJ ? hi : nh, al = CJ ? li : nl;  // multiplies y in the real part
  const int bh = CJ ? nh : hi, bl = CJ ? nl : li;  // multiplies x in the imaginary part
  const ll r = 1ll << 31;
  const ll cx = (ll)xl * hr + (ll)xh * lr + (ll)yl * ah + (ll)yh * al + r;
  const ll cy = (ll)yl * hr + (ll)yh * lr + (ll)xl * bh + (ll)xh * bl + r;
  q2 o;
  o.x = (ll)xh * hr + (ll)yh * ah + (cx >> 32);
  o.y = (ll)yh * hr + (ll)xh * bh + (cy >> 32);
  return o;
}
template <bool CJ>
SB_HD q2 qmul(q2 z, const qw &w) {
  return qmul<CJ>(z, w.hr, w.lr, w.hi, w.li);
}

// ---------------------------------------------------------------------------
// small transforms in registers, X_k = sum_n v_n exp(S 2 pi i n k / R), natural
// order in and out
// ---------------------------------------------------------------------------
template <int S>
SB_HD void qd2(q2 &a, q2 &b) {
  const q2 t = a - b;
  a = a + b;
  b = t;
}
// 16 64-bit adds
template <int S>
SB_HD void qd4(q2 &v0, q2 &v1, q2 &v2, q2 &v3) {
  const q2 a0 = v0 + v2, a1 = v0 - v2, b0 = v1 + v3, b1 = qrot<S>(v1 - v3);
  v0 = a0 + b0;
  v2 = a0 - b0;
  v1 = a1 + b1;
  v3 = a1 - b1;
}
// sqrt(3)/2 at 2^63: the product is halved, doubled again by an add
template <int S>
SB_HD void qd3(q2 &v0, q2 &v1, q2 &v2) {
  const q2 t = v1 + v2, d = v1 - v2;
  const q2 m = v0 - qshr(t, 1);
  const q2 e = qdbl(mkq(qmulr(d.x, 1859775393, 1630710223), qmulr(d.y, 1859775393, 1630710223)));
  const q2 j = qrot<S>(e);
  v0 = v0 + t;
  v1 = m + j;
  v2 = m - j;
}
// cos and sin of 2 pi/5 and 4 pi/5 at 2^63
template <int S>
SB_HD void qd5(q2 &v0, q2 &v1, q2 &v2, q2 &v3, q2 &v4) {
  const q2 t1 = v1 + v4, t2 = v2 + v3, t3 = v1 - v4, t4 = v2 - v3;
  auto c1 = [](ll x) { return qmulr(x, 663608942, 1607638789); };
  auto c2 = [](ll x) { return qmulr(x, -1737350766, -1607638789); };
  auto s1 = [](ll x) { return qmulr(x, 2042378317, 290717050); };
  auto s2 = [](ll x) { return qmulr(x, 1262259218, -714508361); };
  const q2 a1 = v0 + qdbl(mkq(c1(t1.x) + c2(t2.x), c1(t1.y) + c2(t2.y)));
  const q2 a2 = v0 + qdbl(mkq(c2(t1.x) + c1(t2.x), c2(t1.y) + c1(t2.y)));
  const q2 b1 = qrot<S>(qdbl(mkq(s1(t3.x) + s2(t4.x), s1(t3.y) + s2(t4.y))));
  const q2 b2 = qrot<S>(qdbl(mkq(s2(t3.x) - s1(t4.x), s2(t3.y) - s1(t4.y))));
  v0 = v0 + t1 + t2;
  v1 = a1 + b1;
  v4 = a1 - b1;
  v2 = a2 + b2;
  v3 = a2 - b2;
}
// z exp(S i pi/4): sqrt(1/2) at 2^63, doubled
template <int S>
SB_HD q2 qw8(q2 z) {
  const ll a = S < 0 ? z.x + z.y : z.x - z.y, b = S < 0 ? z.y - z.x : z.x + z.y;
  return qdbl(mkq(qmulr(a, 1518500250, -51432894), qmulr(b, 1518500250, -51432894)));
}
template <int S>
SB_HD void qd8(q2 *v) {
  qd4<S>(v[0], v[2], v[4], v[6]);
  qd4<S>(v[1], v[3], v[5], v[7]);
  // v[0,2,4,6] = E_0..E_3, v[1,3,5,7] = O_0..O_3
  const q2 o1 = qw8<S>(v[3]), o2 = qrot<S>(v[5]), o3 = qrot<S>(qw8<S>(v[7]));
  const q2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
  v[0] = e0 + o0;
  v[4] = e0 - o0;
  v[1] = e1 + o1;
  v[5] = e1 - o1;
  v[2] = e2 + o2;
  v[6] = e2 - o2;
  v[3] = e3 + o3;
  v[7] = e3 - o3;
}

// R-point transform; R = Ra Rb coprime runs without twiddles (Good, Thomas);
// 16 = 4 x 4 with its twiddles divides by 4 (kShift)
template <int R, int S>
struct Dft;
template <int S>
struct Dft<4, S> {
  static constexpr int kShift = 0;
  static SB_HD void run(q2 *v) { qd4<S>(v[0], v[1], v[2], v[3]); }
};
template <int S>
struct Dft<8, S> {
  static constexpr int kShift = 0;
  static SB_HD void run(q2 *v) { qd8<S>(v); }
};
template <int S>
struct Dft<16, S> {
  static constexpr int kShift = 2;
  static SB_HD void run(q2 *v) {
#pragma unroll
    for (int q = 0; q < 4; q++) qd4<S>(v[q], v[q + 4], v[q + 8], v[q + 12]);
    // v[n2 + 4 k1] times W_16^(n2 k1) / 4
    constexpr bool C = S > 0;
    auto w1 = [](q2 z) { return qmul<C>(z, 992008094, 1696238673, -410903207, 1364630830); };
    auto w3 = [](q2 z) { return qmul<C>(z, 410903207, -1364630830, -992008094, -1696238673); };
    // sqrt(1/2) at 2^62
    auto w2 = [](q2 z) {
      const ll a = S < 0 ? z.x + z.y : z.x - z.y, b = S < 0 ? z.y - z.x : z.x + z.y;
      return mkq(qmulr(a, 759250125, -25716447), qmulr(b, 759250125, -25716447));
    };
    v[0] = qshr(v[0], 2);
    v[1] = qshr(v[1], 2);
    v[2] = qshr(v[2], 2);
    v[3] = qshr(v[3], 2);
    v[4] = qshr(v[4], 2);
    v[8] = qshr(v[8], 2);
    v[12] = qshr(v[12], 2);
    v[5] = w1(v[5]);
    v[6] = w2(v[6]);
    v[7] = w3(v[7]);
    v[9] = w2(v[9]);
    v[10] = qrot<S>(qshr(v[10], 2));
    v[11] = qrot<S>(w2(v[11]));
    v[13] = w3(v[13]);
    v[14] = qrot<S>(w2(v[14]));
    {
      const q2 t = w1(v[15]);
      v[15] = mkq(-t.x, -t.y);  // W_16^9 = -W_16
    }
#pragma unroll
    for (int k = 0; k < 4; k++) qd4<S>(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    // X[k1 + 4 k2] sits at v[4 k1 + k2]
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = a + 1; b < 4; b++) {
        const q2 t = v[4 * a + b];
        v[4 * a + b] = v[4 * b + a];
        v[4 * b + a] = t;
      }
  }
};
template <int R, int S>
SB_HD void qdsmall(q2 *v) {
  if constexpr (R == 3)
    qd3<S>(v[0], v[1], v[2]);
  else if constexpr (R == 5)
    qd5<S>(v[0], v[1], v[2], v[3], v[4]);
  else if constexpr (R == 2)
    qd2<S>(v[0], v[1]);
  else
    Dft<R, S>::run(v);
}
SB_HD constexpr int qinv(int a, int m) {  // a^-1 mod m
  for (int i = 1; i < m; i++)
    if ((a * i) % m == 1) return i;
  return 1;
}
template <int Ra, int Rb, int S>
struct Pfa {
  static constexpr int kShift = 0;
  static SB_HD void run(q2 *v) {
    constexpr int R = Ra * Rb;
    constexpr int ea = Rb * qinv(Rb % Ra, Ra), eb = Ra * qinv(Ra % Rb, Rb);
    q2 t[R];
#pragma unroll
    for (int b = 0; b < Rb; b++) {
      q2 u[Ra];
#pragma unroll
      for (int a = 0; a < Ra; a++) u[a] = v[(Rb * a + Ra * b) % R];
      qdsmall<Ra, S>(u);
#pragma unroll
      for (int a = 0; a < Ra; a++) t[a * Rb + b] = u[a];
    }
#pragma unroll
    for (int a = 0; a < Ra; a++) {
      qdsmall<Rb, S>(t + a * Rb);
#pragma unroll
      for (int b = 0; b < Rb; b++) v[(ea * a + eb * b) % R] = t[a * Rb + b];
    }
  }
};
template <int S> struct Dft<10, S> : Pfa<5, 2, S> {};
template <int S> struct Dft<12, S> : Pfa<3, 4, S> {};
template <int S> struct Dft<20, S> : Pfa<5, 4, S> {};
template <int S> struct Dft<24, S> : Pfa<3, 8, S> {};

// ---------------------------------------------------------------------------
// plans: N = R1 R2, the bits of the largest input component
// ---------------------------------------------------------------------------
template <int N> struct Plan;
#define SB_PLAN(N, A, B, BITS)                      \
  template <> struct Plan<N> {                      \
    static constexpr int R1 = A, R2 = B, bits = BITS; \
    /* log2 of the division by the twiddles and the 16-point kernels */ \
    static constexpr int shift = 2 + (A == 16 ? 2 : 0) + (B == 16 ? 2 : 0); \
  };
// input modulus b = 2^(bits+1/2); largest intermediate: 32: 8b, 48: 12b,
// 64: 16b, 80: 20b, 96: 24b, 128: 8b, 160: 10b, 192: 12b, 256: 4b, 320: 20b,
// 384: 24b, each below 2^62.5
SB_PLAN(32, 8, 4, 58)
SB_PLAN(48, 12, 4, 58)
SB_PLAN(64, 8, 8, 57)
SB_PLAN(80, 10, 8, 57)
SB_PLAN(96, 12, 8, 57)
SB_PLAN(128, 16, 8, 58)
SB_PLAN(160, 10, 16, 58)
SB_PLAN(192, 12, 16, 58)
SB_PLAN(256, 16, 16, 59)
SB_PLAN(320, 20, 16, 57)
SB_PLAN(384, 24, 16, 57)
#undef SB_PLAN

SB_HD constexpr bool fix_length(int n) {
  return n == 32 || n == 48 || n == 64 || n == 80 || n == 96 || n == 128 || n == 160 ||
         n == 192 || n == 256 || n == 320 || n == 384;
}

// ---------------------------------------------------------------------------
// conversions.  A block's scale is the largest exponent of its components:
// `top` is the maximum of their upper words without the sign (hiword()), and
// its exponent field E = top >> 20 gives |x| < 2^(E-1022).
// ---------------------------------------------------------------------------
SB_HD ull dbits64(double d) {
#ifdef __CUDA_ARCH__
  return (ull)__double_as_longlong(d);
#else
  ull u;
  __builtin_memcpy(&u, &d, 8);
  return u;
#endif
}
SB_HD double bits64d(ull u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((ll)u);
#else
  double d;
  __builtin_memcpy(&d, &u, 8);
  return d;
#endif
}
SB_HD unsigned fbits32(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  unsigned u;
  __builtin_memcpy(&u, &f, 4);
  return u;
#endif
}
SB_HD float bits32f(unsigned u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  __builtin_memcpy(&f, &u, 4);
  return f;
#endif
}
SB_HD unsigned hiword(double d) { return (unsigned)(dbits64(d) >> 32) & 0x7fffffffu; }
// a float's bits moved to where the double of the same value has them (for a
// subnormal number those of one just below the normal range)
SB_HD unsigned hiword(float f) {
  const unsigned u = fbits32(f) & 0x7fffffffu;
  if (u >= 0x7f800000u) return 0x7ff00000u;
  return u == 0u ? 0u : (u >> 3) + (896u << 20);
}
// scale of a block: the integers are x 2^p.  Zero blocks and blocks below
// 2^-958 count as zero (a scale at which every shift empties the integer); a
// block with an infinity or a NaN is flagged
constexpr int kZeroScale = -4000;
struct QScale {
  int p;
  bool bad;
  // the scale as an exponent: the integers of a zero block weigh nothing
  SB_HD int weight() const { return p == kZeroScale ? -kZeroScale : p; }
};
// from the largest component alone: |x| 2^p < 2^bits
SB_HD QScale qscale(unsigned top, int bits) {
  QScale s;
  const int E = (int)(top >> 20);
  s.p = E < 64 ? kZeroScale : bits - (E - 1022);
  s.bad = E == 0x7ff;
  return s;
}
// x 2^p to nearest; |x| 2^p < 2^62
SB_HD ll tofix(double d, const QScale &s) {
  const ull u = dbits64(d);
  const int e = (int)((u >> 52) & 0x7ff);
  const ull m = ((u & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
  int sh = 1084 - s.p - e;  // 10 - (p + e - 1075) less the rounding bit
  if (sh > 63) sh = 63;
  const ll r = (ll)(((m >> sh) + 1) >> 1), g = (ll)u >> 63;
  return (r ^ g) - g;
}
SB_HD ll tofix(float f, const QScale &s) {
  const unsigned u = fbits32(f);
  int e = (int)((u >> 23) & 0xff);
  const ull m = (ull)((u & 0x7fffffu) | (e ? 0x800000u : 0u)) << 39;
  e = e ? e : 1;            // subnormal
  int sh = 188 - s.p - e;  // 39 - (p + e - 150) less the rounding bit
  if (sh > 63) sh = 63;
  const ll r = (ll)(((m >> sh) + 1) >> 1), g = -(ll)(u >> 31);
  return (r ^ g) - g;
}
SB_HD int qclz(ull a) {
#ifdef __CUDA_ARCH__
  return __clzll((ll)a);
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}
// v 2^t, rounded to nearest (|v| < 2^63).  The exponent t comes from a block's
// scale: blocks whose results could pass the range of R are flagged by
// qrange() first; results below the smallest normal number are zero (a
// float's down to its smallest subnormal are kept)
SB_HD bool qrange(int t) { return t > 900; }
SB_HD double fromfix(ll v, int t) {
  const ll g = v >> 63;
  ull a = (ull)((v ^ g) - g);
  const int lz = qclz(a);
  a = ((a << ((lz - 1) & 63)) + 0x200) >> 10;  // the leading bit at 52
  const int E = t + 1085 - lz;  // biased exponent less the implicit one
  const ull r = a + ((ull)(unsigned)E << 52);
  return v == 0 || E < 0 ? 0.0 : bits64d(r | ((ull)g & 0x8000000000000000ull));
}
SB_HD float fromfixf(ll v, int t) {
  const ll g = v >> 63;
  ull a = (ull)((v ^ g) - g);
  const int lz = qclz(a);
  const int E = t + 63 - lz + 126;
  unsigned r = (unsigned)(((a << ((lz - 1) & 63)) + (1ull << 38)) >> 39);  // the leading bit at 23
  if (v == 0 || E < -24) return 0.0f;
  if (E >= 254) r = 0x7f800000u;
  else r = E < 0 ? r >> -E : r + ((unsigned)E << 23);
  return bits32f(r | ((unsigned)g & 0x80000000u));
}
template <typename R> SB_HD R qout(ll v, int t);
template <> SB_HD double qout<double>(ll v, int t) { return fromfix(v, t); }
template <> SB_HD float qout<float>(ll v, int t) { return fromfixf(v, t); }

// ---------------------------------------------------------------------------
// integers times factors of any size.  A wave of a line is multiplied by a
// factor c (a derivative's symbol, a Helmholtz inverse) that spans orders of
// magnitude over the waves, so the products get a new common scale: with
// L = max over the waves of qlen(x) + qexp(c), |x c| < 2^(L+1).
// ---------------------------------------------------------------------------
SB_HD int qlen(q2 z) {  // |z.x|, |z.y| < 2^qlen; at least 32
  const unsigned h = (unsigned)((z.x ^ (z.x >> 63)) >> 32) | (unsigned)((z.y ^ (z.y >> 63)) >> 32);
#ifdef __CUDA_ARCH__
  return 64 - (h ? __clz((int)h) : 32);
#else
  return 64 - (h ? __builtin_clz(h) : 32);
#endif
}
SB_HD int qexp(double c) { return (int)((dbits64(c) >> 52) & 0x7ff) - 1023; }
// x c 2^s0, where the result is known to stay below 2^60
SB_HD q2 qscaled(q2 x, double c, int s0) {
  const ull u = dbits64(c);
  const int s = s0 + (int)((u >> 52) & 0x7ff) - 1020;
  const ull m = ((u & 0xfffffffffffffull) | 0x10000000000000ull) << 9;
  int r = s < 0 ? -s : 0, l = s > 0 ? s : 0;
  if (r > 63) r = 63;
  if (l > 63) l = 63;
  const ll g = (ll)u >> 63, w = ((ll)(m >> r) ^ g) - g;
  const int h = qhi(w), lo = qlo(w);
  return mkq(qmulr((ll)((ull)x.x << l), h, lo), qmulr((ll)((ull)x.y << l), h, lo));
}

SB_HD ll qmulhi(ll a, ll b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return (ll)(((__int128)a * b) >> 64);
#endif
}
// exp(-2 pi i X j / (N 2^64)) to about 2^-61: the leading 10 bits of the angle
// from the table turn[t] = exp(-2 pi i t/1024) (fix_twiddles), the rest
// (|r| < 2^-8) by the Taylor series of cos and sin
SB_HD qw qturn(ll X, int j, int N, const qw *turn) {
  const ll q = X / N;
  const int rem = (int)(X - q * N);
  const ull A = (ull)q * (ull)(ll)j + (ull)(ll)(rem * j / N);
  const unsigned t = (unsigned)((A + (1ull << 53)) >> 54) & 1023u;
  const ll d = (ll)(A - ((ull)t << 54));
  const ll r = qmulhi(d << 9, 7244019458077122842ll);  // 2 pi at 2^60: r at 2^69
  const ll r2 = qmulhi(r, r);                           // 2^74
  const ll r4 = qmulhi(r2, r2) >> 10, r6 = qmulhi(r4, r2) >> 10;  // 2^74
  const ll cm = -(r2 >> 1) + r4 / 24 - r6 / 720;                  // cos - 1
  const ll r3 = qmulhi(r, r2) >> 10, r5 = qmulhi(r3, r2) >> 10, r7 = qmulhi(r5, r2) >> 10;  // 2^69
  const ll sn = r - r3 / 6 + r5 / 120 - r7 / 5040;
  const qw w = turn[t];
  const ll tr = (ll)((ull)(ll)w.hr << 32) + w.lr, ti = (ll)((ull)(ll)w.hi << 32) + w.li;
  const ll re = tr + ((qmulhi(tr, cm) + 512) >> 10) + ((qmulhi(ti, sn) + 16) >> 5);
  const ll im = ti + ((qmulhi(ti, cm) + 512) >> 10) - ((qmulhi(tr, sn) + 16) >> 5);
  qw o;
  o.lr = qlo(re) == (int)0x80000000 ? qlo(re) + 1 : qlo(re);
  o.hr = (int)((re - (ll)o.lr) >> 32);
  o.li = qlo(im) == (int)0x80000000 ? qlo(im) + 1 : qlo(im);
  o.hi = (int)((im - (ll)o.li) >> 32);
  return o;
}

}  // namespace sb
