// sb_planeq.cu -- the plane stages of the FP64 step in 64-bit fixed point.
//
// The FP64 plane stages (k_p1, k_p2, k_p3 of sb_kernels.cu) are bound by the
// FP64 pipe: at 192x96x96 some 190 FP64 instructions per point of a substep at
// 64 cycles each.  Here the z and x transforms and the products u x omega run on
// 64-bit integers (sb_fix.cuh) and the planes between the stages stay integers,
// so that FP64 is left for the reconstruction of the velocity (20 instructions a
// mode) and the right-hand sides (12):
//   k_z1  per (plane, 8 kx columns, pair of fields): u, w, omega_x, omega_z
//         from v and omega_y (cross.f90:1226-1276), backward z-transform
//         (fill00, fou3D_thread.f:73-126); one power of two per column in bf.ze
//   k_x2  per (plane, two pairs of z rows): backward x-transforms of two rows at
//         once, |u| maxima (cross.f90:1438-1441), u x (omega + 2 chi z)
//         (cross.f90:1453-1462), forward x-transforms; one power of two per
//         row pair and product in bf.xe
//   k_z3  per (plane, 8 kx columns): forward z-transforms, truncation (pack00),
//         right-hand sides (cross.f90:1536-1546)
// Every sequence takes its own scale, from its largest component (physical
// rows) or from the sum of the moduli where that allows a larger one (spectra,
// which are steep: the sum bounds every intermediate of the transform).
// Bound by latency: 11-21 warps per SM (registers), issue slots 27-43% in use, no
// pipe above half of its peak (ALU 32-44%; FP64 47% in k_z1 and k_z3).
// Transforms run in place in shared memory as N = R1 R2 (Plan); a column
// transform keeps 8 columns in the 128 bytes of a row (no bank conflicts,
// full lines of global memory), a row transform pads each R2 entries by one.
#include <cuda_runtime.h>

#include "sb_common.cuh"
#include "sb_fix.cuh"
#include "sb_kernels.h"

namespace sb {

namespace {

constexpr int kCols = 8;
constexpr int kBad = 1 << 24;  // exponent of a sequence with a component that is not finite
constexpr int kNoLen = -(1 << 28);

__device__ __forceinline__ int kgrid(int k, int nz, int NZ, int mz) { return k <= nz ? k : k + (NZ - mz); }
__device__ __forceinline__ q2 qzero() { return mkq(0, 0); }
// x 2^s
__device__ __forceinline__ q2 qshift(q2 x, int s) {
  const int l = s > 0 ? (s > 63 ? 63 : s) : 0, r = s < 0 ? (s < -63 ? 63 : -s) : 0;
  return mkq((ll)((ull)x.x << l) >> r, (ll)((ull)x.y << l) >> r);
}
// v 2^-r to nearest, r >= 0 (a shift alone makes -1 of every small negative number)
__device__ __forceinline__ ll qround(ll v, int r) {
  const int c = r > 0;
  return ((v >> min(63, r - c)) + c) >> c;
}
// the same to nearest, for entries that are aligned with larger ones: beside a
// strong mean flow weak modes must vanish, not leave a unit's noise (a
// 192x96x96 step 837 -> 855 us)
__device__ __forceinline__ q2 qalign(q2 x, int s) {
  const int l = s > 0 ? (s > 63 ? 63 : s) : 0, r = s < 0 ? -s : 0;
  return mkq(qround((ll)((ull)x.x << l), r), qround((ll)((ull)x.y << l), r));
}
__device__ __forceinline__ int bitlen(unsigned v) { return 32 - __clz((int)v); }
// v 2^t, past the range as an infinity
__device__ __forceinline__ double fromfix_big(ll v, int t) {
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  const bool big = v != 0 && t + 64 - qclz((ull)(v < 0 ? -v : v)) > 1024;
  return big ? (v < 0 ? -inf : inf) : fromfix(v, t);
}
// a b / 2^64; |a|, |b| <= 2^62
__device__ __forceinline__ ll qprod(ll a, ll b) { return qmulr(a, qhi(b), qlo(b)); }

// entry j of a sequence of N modes under the 2/3 rule is zero for every j of
// the kernel's middle third (R1 a multiple of 3), or by comparison
template <int N, int R1>
__device__ __forceinline__ bool gap(int n1, int j, int keep) {
  if (R1 % 3 == 0 && n1 >= R1 / 3 && n1 < 2 * R1 / 3) return true;
  return j > keep && j < N - keep;
}

}  // namespace

// ---------------------------------------------------------------------------
// plane stage 1
// ---------------------------------------------------------------------------
template <int NZ>
struct Z1 {
  static constexpr int R1 = Plan<NZ>::R1, R2 = Plan<NZ>::R2;
  // threads as the row kernels' items (64 boxes of 64x32x32: 112 us with 64
  // against 172 with 128; 192 points: 370 us with 128 against 519 and, with 256,
  // 452), and more warps where the registers allow (96 points: 50.9 us at 85
  // registers against 55.5 at 128; 192 points 394 against 370)
  static constexpr int T = NZ < 64 ? 64 : 128;
  static constexpr int kMinB = NZ <= 96 ? 768 / T : NZ <= 192 ? 4 : 2;
  static constexpr size_t smem = 2 * sizeof(q2) * NZ * kCols;
};

template <int NZ, bool TEMP>
__global__ void __launch_bounds__(Z1<NZ>::T, Z1<NZ>::kMinB) k_z1(Grid g, Bufs bf) {
  constexpr int R1 = Z1<NZ>::R1, R2 = Z1<NZ>::R2, T = Z1<NZ>::T;
  const int ncb = (g.nkx + kCols - 1) / kCols;
  const int round = blockIdx.x / ncb, cb = blockIdx.x - round * ncb;
  const int j = blockIdx.y, b = blockIdx.z;
  const Member &M = bf.mem[b];
  if (M.halted) return;
  extern __shared__ __align__(16) unsigned char smz_raw[];
  q2 *ex = (q2 *)smz_raw;
  __shared__ unsigned s_top[2][kCols], s_sum[2][kCols];
  const int nkx = g.nkx, mz = g.mz, nz = g.nz;
  const int ci = threadIdx.x & (kCols - 1), i = cb * kCols + ci;
  const bool act = i < nkx;
  const long pb = ((long)b * g.field + (long)j * g.plane) / 2;
  if (threadIdx.x < 2 * kCols) (&s_top[0][0])[threadIdx.x] = (&s_sum[0][0])[threadIdx.x] = 0u;
  __syncthreads();
  const int nfl = TEMP && round == g.tround ? 1 : 2;
  unsigned topa = 0, topb = 0;
  {
    const double2 *vor = (const double2 *)bf.vor + pb, *phi = (const double2 *)bf.phi + pb;
    const double2 *p0 = round == 0 ? (const double2 *)bf.V + pb : round == 1 ? (const double2 *)bf.D + pb
                                                                             : (const double2 *)bf.G + pb;
    const double2 *p1 = round == 1 ? phi : vor;
#pragma unroll 2
    for (int k = threadIdx.x / kCols; k < mz; k += T / kCols) {
      double2 fa = make_double2(0.0, 0.0), fb = fa;
      if (act) {
        const long q = (long)k * nkx + i;
        const bool z00 = i == 0 && k == 0;
        if (TEMP && round == g.tround) {
          // the temperature as stored, its (0,0) mode tb00 (crosst.f90:556-559,1459-1462)
          fa = ((const double2 *)bf.tb + pb)[q];
          if (z00) fa = make_double2(((const double2 *)bf.mt)[(long)b * g.my + j].x, 0.0);
        } else {
          // omega_y and phi with the kx = 0 conjugate symmetry (cross.f90:493-502)
          const bool sym = i == 0 && k > nz;
          const double2 x = p0[q];
          double2 y = p1[sym ? (long)(mz - k) * nkx : q];
          if (sym) y.y = -y.y;
          if (round < 2) {
            // i (a x -+ gz y)/k2, i (gz x +- a y)/k2
            // (the factors from a table: half of this kernel's time is FP64 issue;
            // 192x96x96: 50 -> 44 us, and k_z3 39 -> 35 with its own)
            const double2 f2 = bf.kfac[q];
            const double an = f2.x, gn = round == 0 ? -f2.y : f2.y;
            fa = make_double2(-fma(an, x.y, gn * y.y), fma(an, x.x, gn * y.x));
            const double gp = f2.y, ap = round == 0 ? an : -an;
            fb = make_double2(-fma(gp, x.y, ap * y.y), fma(gp, x.x, ap * y.x));
            if (z00) {
              const double2 m = ((const double2 *)(round == 0 ? bf.mu : bf.mdu))[(long)b * g.my + j];
              fa = make_double2(round == 0 ? m.x : m.y, 0.0);
              fb = make_double2(round == 0 ? m.y : -m.x, 0.0);
            }
          } else {
            fa = z00 ? make_double2(M.vbulk, 0.0) : x;
            fb = y;
          }
        }
      }
      const int s = kgrid(k, nz, NZ, mz) * kCols + ci;
      ((double2 *)ex)[s] = fa;
      topa = max(topa, max(hiword(fa.x), hiword(fa.y)));
      if (nfl > 1) {
        ((double2 *)ex)[NZ * kCols + s] = fb;
        topb = max(topb, max(hiword(fb.x), hiword(fb.y)));
      }
    }
  }
  atomicMax(&s_top[0][ci], topa);
  if (nfl > 1) atomicMax(&s_top[1][ci], topb);
  __syncthreads();
  // sums of |x| + |y| in units of 2^-20 of the largest power of two
#pragma unroll 1
  for (int f = 0; f < nfl; f++) {
    const int E = (int)(s_top[f][ci] >> 20);
    unsigned sum = 0;
#pragma unroll 2
    for (int k = threadIdx.x / kCols; k < mz; k += T / kCols) {
      const double2 v = ((const double2 *)ex)[(f * NZ + kgrid(k, nz, NZ, mz)) * kCols + ci];
      const unsigned hx = hiword(v.x), hy = hiword(v.y);
      sum += (((hx & 0xfffffu) | 0x100000u) >> min(31, E - (int)(hx >> 20))) +
             (((hy & 0xfffffu) | 0x100000u) >> min(31, E - (int)(hy >> 20))) + 2u;
    }
    atomicAdd(&s_sum[f][ci], sum);
  }
  __syncthreads();
  int p[2];
#pragma unroll
  for (int f = 0; f < 2; f++) {
    const QScale s = qscale(s_top[f][ci], Plan<NZ>::bits);
    // sum < s_sum 2^(E - 1043), E the exponent field
    p[f] = s.p == kZeroScale ? s.p : max(s.p, 1105 - (int)(s_top[f][ci] >> 20) - bitlen(s_sum[f][ci]));
    if (threadIdx.x < kCols && f < nfl && act) {
      const int fz = TEMP && round == g.tround ? g.tzf : 2 * round + f;
      bf.ze[(((long)b * g.my + j) * g.nzf + fz) * nkx + i] =
          s.bad ? kBad : p[f] == kZeroScale ? kZeroScale : Plan<NZ>::shift - p[f];
    }
  }
#pragma unroll 1
  for (int it = threadIdx.x / kCols; it < nfl * R2; it += T / kCols) {
    const int f = it / R2, n2 = it - f * R2;
    q2 *e = ex + f * NZ * kCols + ci;
    QScale s;
    s.p = p[f];
    const double2 *rows = (const double2 *)e;
    q2 v[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; n1++) {
      const int q = n2 + R2 * n1;
      v[n1] = qzero();
      if (!gap<NZ, R1>(n1, q, nz)) {
        const double2 w = rows[q * kCols];
        v[n1] = mkq(tofix(w.x, s), tofix(w.y, s));
      }
    }
    Dft<R1, 1>::run(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) e[(k1 * R2 + n2) * kCols] = qmul<true>(v[k1], bf.fz[n2 * k1]);
  }
  __syncthreads();
  q2 *zb = (q2 *)bf.zbuf + ((long)b * g.my + j) * (long)NZ * g.nzf * nkx;
#pragma unroll 1
  for (int it = threadIdx.x / kCols; it < nfl * R1; it += T / kCols) {
    const int f = it / R1, k1 = it - f * R1;
    const q2 *e = ex + (f * NZ + k1 * R2) * kCols + ci;
    q2 v[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) v[n2] = e[n2 * kCols];
    Dft<R2, 1>::run(v);
    const int fz = TEMP && round == g.tround ? g.tzf : 2 * round + f;
    if (act)
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) zb[((long)(k1 + R1 * k2) * g.nzf + fz) * nkx + i] = v[k2];
  }
}

// ---------------------------------------------------------------------------
// plane stage 2
// ---------------------------------------------------------------------------
// NP row pairs of a block: two where the blocks fill the GPU and fit in shared
// memory, else one (64x32x32 alone: 10.4 us against 14.1; 384x192x192: 802 us
// against 1065, where two pairs leave two blocks an SM; with the shifts
// rounding 10.7 and 833, and 103.6 at 192x96x96 for the 99.7 below)
template <int NX, bool TEMP, int NP>
struct X2 {
  static constexpr int R1 = Plan<NX>::R1, R2 = Plan<NX>::R2;
  static constexpr int NF = TEMP ? 7 : 6, NO = TEMP ? 6 : 3;
  static constexpr int T = R2 == 16 ? 96 : R2 == 8 ? 64 : 32;
  // registers per thread: the 16-point kernels want 168 (192x96x96: 99.7 us
  // against 102 at 128 and 105 at 104), the smaller ones more warps (64 boxes
  // of 64x32x32: 233 us at 104 against 244 and 274)
  static constexpr int kRegs = R2 == 16 ? 168 : 104;
  static constexpr int BS = R1 * (R2 + 1);
  static constexpr size_t smem = sizeof(q2) * NP * NF * BS;
};

template <int NX, bool TEMP, int NP>
__global__ void __launch_bounds__(X2<NX, TEMP, NP>::T, 65536 / (X2<NX, TEMP, NP>::T * X2<NX, TEMP, NP>::kRegs))
    k_x2(Grid g, Bufs bf, int rk) {
  typedef X2<NX, TEMP, NP> C;
  constexpr int R1 = C::R1, R2 = C::R2, NF = C::NF, NO = C::NO, T = C::T, BS = C::BS;
  constexpr int IT = (NX / 3 + 31) / 32, kSh = Plan<NX>::shift, kBits = Plan<NX>::bits;
  const int j = blockIdx.y, b = blockIdx.z;
  Member &M = bf.mem[b];
  if (M.halted) return;
  extern __shared__ __align__(16) unsigned char smx_raw[];
  q2 *ex = (q2 *)smx_raw;
  __shared__ int s_e[NP * NF], s_len[NP * NF], s_ho[NP * NO], s_hl[NP * NO];
  // sums of the third moments: in units of 2^16 and what is left
  __shared__ ll s_third[NP][3], s_rest[NP][3];
  const int nkx = g.nkx, NZ = g.mgalz, z0 = 2 * NP * blockIdx.x;
  const int lane = threadIdx.x & 31;
  auto P = [](int x) { return x + x / R2; };
  if (threadIdx.x < NP * NF) s_len[threadIdx.x] = kNoLen;
  if (threadIdx.x < NP * NO) s_hl[threadIdx.x] = kNoLen;
  if (threadIdx.x < 3 * NP) (&s_third[0][0])[threadIdx.x] = (&s_rest[0][0])[threadIdx.x] = 0;
  // ---- rows in: one warp per sequence.  Two rows in one complex sequence
  // (Hermitian extension; FFTW's c2r ignores the imaginary part of kx = 0)
  {
    const long pj = (long)b * g.my + j;
    const q2 *zb = (const q2 *)bf.zbuf + pj * NZ * g.nzf * nkx;
    const int *ze = bf.ze + pj * g.nzf * nkx;
#pragma unroll 1
    for (int s = threadIdx.x >> 5; s < NP * NF; s += T / 32) {
      const int p = s / NF, f = s - p * NF, zf = f < 6 ? f : g.tzf, z = z0 + 2 * p;
      q2 X1[IT], X2[IT];
      int e[IT], len = kNoLen, emax = kNoLen;
#pragma unroll
      for (int q = 0; q < IT; q++) {
        const int i = lane + 32 * q;
        X1[q] = X2[q] = qzero();
        e[q] = kNoLen;
        if (i < nkx) {
          X1[q] = zb[((long)z * g.nzf + zf) * nkx + i];
          X2[q] = zb[((long)(z + 1) * g.nzf + zf) * nkx + i];
          e[q] = ze[zf * nkx + i];
          if (i == 0) X1[q].y = X2[q].y = 0;
          len = max(len, max(qlen(X1[q]), qlen(X2[q])) + e[q]);
          emax = max(emax, e[q]);
        }
      }
      len = __reduce_max_sync(0xffffffffu, len);
      emax = __reduce_max_sync(0xffffffffu, emax);
      // sum of the moduli's components in units of 2^(len - 20); every entry
      // appears twice in the sequence
      unsigned sum = 0;
#pragma unroll
      for (int q = 0; q < IT; q++) {
        const int sh = min(63, len - e[q] - 20);
        if (lane + 32 * q < nkx)
          sum += (unsigned)((X1[q].x < 0 ? -X1[q].x : X1[q].x) >> sh) +
                 (unsigned)((X1[q].y < 0 ? -X1[q].y : X1[q].y) >> sh) +
                 (unsigned)((X2[q].x < 0 ? -X2[q].x : X2[q].x) >> sh) +
                 (unsigned)((X2[q].y < 0 ? -X2[q].y : X2[q].y) >> sh) + 4u;
      }
      sum = __reduce_add_sync(0xffffffffu, sum);
      const int pt = max(kBits - 1 - len, 81 - len - bitlen(sum));
      q2 *x = ex + s * BS;
#pragma unroll
      for (int q = 0; q < IT; q++) {
        const int i = lane + 32 * q;
        if (i < nkx) {
          const q2 a = qalign(X1[q], pt + e[q]), c = qalign(X2[q], pt + e[q]);
          x[P(i)] = mkq(a.x - c.y, a.y + c.x);
          if (i > 0) x[P(NX - i)] = mkq(a.x + c.y, c.x - a.y);
        }
      }
      if (lane == 0) s_e[s] = emax >= kBad ? kBad : kSh - pt;
    }
  }
  __syncthreads();
  // ---- backward transforms, to the order x = k1 + R1 k2 at slot (k1, k2)
#pragma unroll 1
  for (int it = threadIdx.x; it < NP * NF * R2; it += T) {
    const int s = it / R2, n2 = it - s * R2;
    q2 *x = ex + s * BS + n2;
    q2 v[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; n1++)
      v[n1] = gap<NX, R1>(n1, n2 + R2 * n1, nkx - 1) ? qzero() : x[n1 * (R2 + 1)];
    Dft<R1, 1>::run(v);
    const qw *tw = bf.fxa + n2;  // W^(n2 k1) at k1 R2 + n2
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) x[k1 * (R2 + 1)] = qmul<true>(v[k1], tw[k1 * R2]);
  }
  __syncthreads();
#pragma unroll 1
  for (int it = threadIdx.x; it < NP * NF * R1; it += T) {
    const int s = it / R1, k1 = it - s * R1;
    q2 *x = ex + s * BS + k1 * (R2 + 1);
    q2 v[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) v[n2] = x[n2];
    Dft<R2, 1>::run(v);
    int len = kNoLen;
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) {
      x[k2] = v[k2];
      len = max(len, qlen(v[k2]));
    }
    atomicMax(&s_len[s], len);
  }
  __syncthreads();
  // ---- products.  Fields: 0 u, 1 w, 2 omega_x, 3 omega_z, 4 v, 5 omega_y
  // (, 6 tb), each shifted to |x| < 2^61; a product of two keeps 2^-64 of them
  const bool hist = rk == 1 && M.ihist;
  const double chi2 = 2.0 * g.chi;
  const double sy = g.s * ((double)j * g.dy - 0.5 * g.Ly);
  double m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0, mt = 0.0;
#pragma unroll 1
  for (int p = 0; p < NP; p++) {
    int sh[NF], e[NF];
    unsigned bad = 0;  // the fields with a number that is not finite
#pragma unroll
    for (int f = 0; f < NF; f++) {
      sh[f] = 61 - s_len[p * NF + f];
      e[f] = s_e[p * NF + f];
      bad |= e[f] >= kBad ? 1u << f : 0u;
      e[f] -= sh[f];
    }
    const int a1 = e[4] + e[3], a2 = e[1] + e[5], a3 = e[1] + e[2], a4 = e[0] + e[3], a5 = e[0] + e[5],
              a6 = e[4] + e[2];
    int o1 = max(a1, a2), o2 = max(a3, a4);
    const int o3 = max(a5, a6);
    // the rotation's term chi2 v, -chi2 u: chi2 = ch 2^(ec - 61), |ch| < 2^62
    ll ch = 0;
    int c1 = kNoLen, c2 = kNoLen;
    if (chi2 != 0.0) {
      const int ec = qexp(chi2);
      ch = (ll)scalbn(chi2, 61 - ec);
      c1 = e[4] + ec - 61;
      c2 = e[0] + ec - 61;
      o1 = max(o1, c1);
      o2 = max(o2, c2);
    }
    auto al = [](ll v, int d) { return qround(v, d); };
    int l1 = kNoLen, l2 = kNoLen, l3 = kNoLen, l4 = kNoLen, l5 = kNoLen, l6 = kNoLen;
    ll umx = INT64_MIN, umn = INT64_MAX, vm = 0, wm = 0, tm = 0, t1 = 0, t2 = 0, t3 = 0;
#pragma unroll 1
    for (int x = threadIdx.x; x < NX; x += T) {
      q2 *q = ex + p * NF * BS + P(x);
      q2 F[NF];
#pragma unroll
      for (int f = 0; f < NF; f++) F[f] = qshift(q[f * BS], sh[f]);
      const q2 u1 = F[0], u3 = F[1], w1 = F[2], w3 = F[3], u2 = F[4], w2 = F[5];
      if (rk == 1) {
        umx = max(umx, max(u1.x, u1.y));
        umn = min(umn, min(u1.x, u1.y));
        vm = max(vm, max(max(u2.x, -u2.x), max(u2.y, -u2.y)));
        wm = max(wm, max(max(u3.x, -u3.x), max(u3.y, -u3.y)));
        if (TEMP) tm = max(tm, max(max(F[NF - 1].x, -F[NF - 1].x), max(F[NF - 1].y, -F[NF - 1].y)));
      }
      if (hist) {
        // v u^2, v w^2, v^3 (cross.f90:2038-2042) of the doubled fields, < 2^58
        // each, a thread's (at most 8) and a row pair's summed exactly: the
        // roundings are below 2^-55 of the sum of |products| (with 55 bits and
        // the last six of each dropped 7e-14 of it)
        const q2 d1 = qdbl(u1), d2 = qdbl(u2), d3 = qdbl(u3);
        t1 += qprod(d2.x, qprod(d1.x, d1.x)) + qprod(d2.y, qprod(d1.y, d1.y));
        t2 += qprod(d2.x, qprod(d3.x, d3.x)) + qprod(d2.y, qprod(d3.y, d3.y));
        t3 += qprod(d2.x, qprod(d2.x, d2.x)) + qprod(d2.y, qprod(d2.y, d2.y));
      }
      q2 h1, h2, h3;
      h1.x = al(qprod(u2.x, w3.x), o1 - a1) - al(qprod(u3.x, w2.x), o1 - a2);
      h1.y = al(qprod(u2.y, w3.y), o1 - a1) - al(qprod(u3.y, w2.y), o1 - a2);
      h2.x = al(qprod(u3.x, w1.x), o2 - a3) - al(qprod(u1.x, w3.x), o2 - a4);
      h2.y = al(qprod(u3.y, w1.y), o2 - a3) - al(qprod(u1.y, w3.y), o2 - a4);
      h3.x = al(qprod(u1.x, w2.x), o3 - a5) - al(qprod(u2.x, w1.x), o3 - a6);
      h3.y = al(qprod(u1.y, w2.y), o3 - a5) - al(qprod(u2.y, w1.y), o3 - a6);
      if (chi2 != 0.0) {
        h1.x += al(qprod(u2.x, ch), o1 - c1);
        h1.y += al(qprod(u2.y, ch), o1 - c1);
        h2.x -= al(qprod(u1.x, ch), o2 - c2);
        h2.y -= al(qprod(u1.y, ch), o2 - c2);
      }
      q[0] = h1;
      q[BS] = h2;
      q[2 * BS] = h3;
      l1 = max(l1, qlen(h1));
      l2 = max(l2, qlen(h2));
      l3 = max(l3, qlen(h3));
      if (TEMP) {
        const q2 tb = F[NF - 1];
        const q2 g1 = mkq(qprod(u1.x, tb.x), qprod(u1.y, tb.y)),
                 g2 = mkq(qprod(u3.x, tb.x), qprod(u3.y, tb.y)),
                 g3 = mkq(qprod(u2.x, tb.x), qprod(u2.y, tb.y));
        q[3 * BS] = g1;
        q[4 * BS] = g2;
        q[5 * BS] = g3;
        l4 = max(l4, qlen(g1));
        l5 = max(l5, qlen(g2));
        l6 = max(l6, qlen(g3));
      }
    }
    l1 = __reduce_max_sync(0xffffffffu, l1);
    l2 = __reduce_max_sync(0xffffffffu, l2);
    l3 = __reduce_max_sync(0xffffffffu, l3);
    if (TEMP) {
      l4 = __reduce_max_sync(0xffffffffu, l4);
      l5 = __reduce_max_sync(0xffffffffu, l5);
      l6 = __reduce_max_sync(0xffffffffu, l6);
    }
    if (lane == 0) {
      atomicMax(&s_hl[p * NO], l1);
      atomicMax(&s_hl[p * NO + 1], l2);
      atomicMax(&s_hl[p * NO + 2], l3);
      if (TEMP) {
        atomicMax(&s_hl[p * NO + 3], l4);
        atomicMax(&s_hl[p * NO + 4], l5);
        atomicMax(&s_hl[p * NO + 5], l6);
      }
    }
    if (threadIdx.x == 0) {
      s_ho[p * NO] = bad ? kBad : o1 + 64;
      s_ho[p * NO + 1] = bad ? kBad : o2 + 64;
      s_ho[p * NO + 2] = bad ? kBad : o3 + 64;
      if (TEMP) {
        s_ho[p * NO + 3] = bad ? kBad : e[0] + e[NF - 1] + 64;
        s_ho[p * NO + 4] = bad ? kBad : e[1] + e[NF - 1] + 64;
        s_ho[p * NO + 5] = bad ? kBad : e[4] + e[NF - 1] + 64;
      }
    }
    if (rk == 1 && umx >= umn) {
      // a maximum passes over the numbers that are not finite
      if (!(bad & 1u)) {
        const double hi = fromfix_big(umx, e[0]), lo = fromfix_big(umn, e[0]);
        m0 = fmax(m0, fmax(fabs(hi), fabs(lo)));
        m1 = fmax(m1, fmax(fabs(hi + sy), fabs(lo + sy)));
      }
      if (!(bad & 16u)) m2 = fmax(m2, fromfix_big(vm, e[4]));
      if (!(bad & 2u)) m3 = fmax(m3, fromfix_big(wm, e[1]));
      if (TEMP && !(bad >> (NF - 1))) mt = fmax(mt, fromfix_big(tm, e[NF - 1]));
    }
    if (hist) {
      // the warp's sums by 32-bit reductions of 24-bit pieces, then one lane's
      // atomics (a 192x96x96 step 829 us; with every lane's six 933, with three
      // 885)
      static_assert(2 * ((NX + T - 1) / T) <= 8, "a thread's sum below 2^62");
      const ll t[3] = {t1, t2, t3};
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)t[q] & 0xffffffu);
        const unsigned mid = __reduce_add_sync(0xffffffffu, (unsigned)(t[q] >> 24) & 0xffffffu);
        const int hi = __reduce_add_sync(0xffffffffu, (int)(t[q] >> 48));
        if (lane == 0) {
          const ll r = ((ll)mid << 24) + lo;
          atomicAdd((ull *)&s_third[p][q], (ull)(((ll)hi << 32) + (r >> 16)));
          atomicAdd((ull *)&s_rest[p][q], (ull)(r & 0xffff));
        }
      }
    }
  }
  if (rk == 1) {
    ull bits[5] = {dbits64(m0), dbits64(m1), dbits64(m2), dbits64(m3), dbits64(mt)};
#pragma unroll
    for (int q = 0; q < (TEMP ? 5 : 4); q++) {
      for (int o = 16; o > 0; o >>= 1) bits[q] = max(bits[q], __shfl_xor_sync(0xffffffffu, bits[q], o));
      if (lane == 0) atomicMax(q < 4 ? &M.umax_bits[q] : &M.tbmax_bits, bits[q]);
    }
  }
  __syncthreads();
  if (hist && threadIdx.x < 3 * NP) {
    // one triple per (plane, row pair); k_hsum adds the pairs
    const int p = threadIdx.x / 3, q = threadIdx.x - 3 * p;
    auto ef = [&](int f) { return s_e[p * NF + f] - (61 - s_len[p * NF + f]); };
    // a sum over numbers that are not finite
    const bool bad = s_e[p * NF + 4] >= kBad || s_e[p * NF + (q == 0 ? 0 : q == 1 ? 1 : 4)] >= kBad;
    const int e2 = q == 0 ? ef(0) : q == 1 ? ef(1) : ef(4);
    const int et = ef(4) + 2 * e2 + 128 - 3;
    const double hi = fromfix_big(s_third[p][q], et + 16);
    bf.ppart[(((long)b * g.my + j) * (NZ / 2) + z0 / 2 + p) * 3 + q] =
        bad ? nan("") : isinf(hi) ? hi : hi + fromfix_big(s_rest[p][q], et);
  }
  // ---- forward transforms, to natural order
#pragma unroll 1
  for (int it = threadIdx.x; it < NP * NO * R1; it += T) {
    const int s = it / R1, k1 = it - s * R1, p = s / NO, o = s - p * NO;
    q2 *x = ex + (p * NF + o) * BS + k1 * (R2 + 1);
    const int sh = kBits - s_hl[s];
    q2 v[R2];
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) v[k2] = qshift(x[k2], sh);
    Dft<R2, -1>::run(v);
    const qw *tw = bf.fxb + k1;  // W^(k1 m) at m R1 + k1
#pragma unroll
    for (int m = 0; m < R2; m++) x[m] = qmul<false>(v[m], tw[m * R1]);
  }
  __syncthreads();
#pragma unroll 1
  for (int it = threadIdx.x; it < NP * NO * R2; it += T) {
    const int s = it / R2, m = it - s * R2, p = s / NO, o = s - p * NO;
    q2 *x = ex + (p * NF + o) * BS + m;
    q2 v[R1];
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) v[k1] = x[k1 * (R2 + 1)];
    Dft<R1, -1>::run(v);
#pragma unroll
    for (int l = 0; l < R1; l++) x[l * (R2 + 1)] = v[l];
  }
  __syncthreads();
  // ---- the two rows' spectra, (Z_k + conj Z_-k)/2 and -i (Z_k - conj Z_-k)/2
  const long pj = (long)b * g.my + j;
  q2 *xb = (q2 *)bf.xbuf + pj * NZ * NO * nkx;
  if (threadIdx.x < NP * NO) {
    const int p = threadIdx.x / NO, o = threadIdx.x - p * NO;
    bf.xe[(pj * (NZ / 2) + z0 / 2 + p) * NO + o] =
        s_ho[threadIdx.x] >= kBad ? kBad : s_ho[threadIdx.x] - (kBits - s_hl[threadIdx.x]) + kSh;
  }
#pragma unroll 1
  for (int s = threadIdx.x >> 5; s < NP * NO; s += T / 32) {
    const int p = s / NO, o = s - p * NO, z = z0 + 2 * p;
    const q2 *x = ex + (p * NF + o) * BS;
    for (int i = lane; i < nkx; i += 32) {
      const q2 zk = qshr(x[P(i)], 1), zm = qshr(x[P(i == 0 ? 0 : NX - i)], 1);
      xb[((long)z * NO + o) * nkx + i] = mkq(zk.x + zm.x, zk.y - zm.y);
      xb[((long)(z + 1) * NO + o) * nkx + i] = mkq(zk.y + zm.y, zm.x - zk.x);
    }
  }
}

// ---------------------------------------------------------------------------
// plane stage 3
// ---------------------------------------------------------------------------
template <int NZ, bool TEMP>
struct Z3 {
  static constexpr int R1 = Plan<NZ>::R1, R2 = Plan<NZ>::R2;
  static constexpr int NO = TEMP ? 6 : 3;
  static constexpr int T = NZ < 64 ? 64 : 128;
  static constexpr int kMinB = NZ < 64 ? 12 : NZ <= 96 ? 5 : NZ <= 256 ? 4 : 2;  // as Z1
  static constexpr size_t smem = sizeof(q2) * NO * NZ * kCols;
};

template <int NZ, bool TEMP>
__global__ void __launch_bounds__(Z3<NZ, TEMP>::T, Z3<NZ, TEMP>::kMinB) k_z3(Grid g, Bufs bf) {
  typedef Z3<NZ, TEMP> C;
  constexpr int R1 = C::R1, R2 = C::R2, NO = C::NO, T = C::T;
  const int j = blockIdx.y, b = blockIdx.z;
  const Member &M = bf.mem[b];
  if (M.halted) return;
  extern __shared__ __align__(16) unsigned char smz_raw[];
  q2 *ex = (q2 *)smz_raw;
  __shared__ int s_len[NO][kCols], s_e[NO * NZ / 2], s_bad;
  const int nkx = g.nkx, mz = g.mz, nz = g.nz;
  const int ci = threadIdx.x & (kCols - 1), i = blockIdx.x * kCols + ci;
  const bool act = i < nkx;
  const long pj = (long)b * g.my + j;
  const q2 *xb = (const q2 *)bf.xbuf + pj * NZ * NO * nkx + (act ? i : 0);
  const int *xe = bf.xe + pj * (NZ / 2) * NO;
  if (threadIdx.x < NO * kCols) (&s_len[0][0])[threadIdx.x] = kNoLen;
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
  for (int q = threadIdx.x; q < NO * NZ / 2; q += T) {
    const int e = xe[q];
    s_e[q] = e;
    if (e >= kBad) atomicOr(&s_bad, 1 << (q % NO));
  }
#pragma unroll 1
  for (int o = 0; o < NO; o++) {
    int len = kNoLen;
#pragma unroll 4
    for (int z = threadIdx.x / kCols; z < NZ; z += T / kCols) {
      const q2 v = xb[((long)z * NO + o) * nkx];
      ex[(o * NZ + z) * kCols + ci] = v;
      len = max(len, qlen(v) + xe[(z >> 1) * NO + o]);
    }
    atomicMax(&s_len[o][ci], len);
  }
  __syncthreads();
#pragma unroll 1
  for (int it = threadIdx.x / kCols; it < NO * R2; it += T / kCols) {
    const int o = it / R2, n2 = it - o * R2;
    q2 *e = ex + o * NZ * kCols + ci;
    const int pt = Plan<NZ>::bits - s_len[o][ci];
    q2 v[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; n1++) {
      const int z = n2 + R2 * n1;
      v[n1] = qalign(e[z * kCols], pt + s_e[(z >> 1) * NO + o]);
    }
    Dft<R1, -1>::run(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) e[(k1 * R2 + n2) * kCols] = qmul<false>(v[k1], bf.fz[n2 * k1]);
  }
  __syncthreads();
#pragma unroll 1
  for (int it = threadIdx.x / kCols; it < NO * R1; it += T / kCols) {
    const int o = it / R1, k1 = it - o * R1;
    q2 *e = ex + (o * NZ + k1 * R2) * kCols + ci;
    q2 v[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) v[n2] = e[n2 * kCols];
    Dft<R2, -1>::run(v);
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) e[k2 * kCols] = v[k2];
  }
  __syncthreads();
  if (!act) return;
  const long pb = ((long)b * g.field + (long)j * g.plane) / 2;
  double2 *Dn = (double2 *)bf.Dn + pb, *Gn = (double2 *)bf.Gn + pb, *Vv = (double2 *)bf.V + pb;
  const double2 *Gv = (const double2 *)bf.G + pb;
  // 1/(mgalx mgalz) of the forward transform, with the wavenumbers
  const double norm = 1.0 / (double)(g.mgalx * g.mgalz);
  const double a = g.alp * i, an = a * norm;
  int eo[NO];
#pragma unroll
  for (int o = 0; o < NO; o++) eo[o] = Plan<NZ>::shift - (Plan<NZ>::bits - s_len[o][ci]);
  bool bad = s_bad != 0;
#pragma unroll
  for (int o = 0; o < NO; o++) bad |= qrange(eo[o]);
  // streamwise-roll force of this plane on hv(kx=0, kz=1) (operators.f90:14-37)
  const bool force = g.force > 0;
  double fj = 0.0;
  if (force) {
    const double y = (double)j * g.dy - 0.5 * g.Ly, w = 1.0 - y * y, gm = g.gam;
    fj = (g.force == 1) ? -0.5 * g.force_roll * (-4.0 * (1.0 - 3.0 * y * y) - gm * gm * w * w)
                        : 0.5 * g.force_roll * (4.0 * y * (-3.0 + 5.0 * y * y) - y * w * w * gm * gm);
  }
#pragma unroll 1
  for (int k = threadIdx.x / kCols; k < mz; k += T / kCols) {
    const int kg = kgrid(k, nz, NZ, mz), k2 = kg / R1, k1 = kg - k2 * R1;
    const q2 *e = ex + (k1 * R2 + k2) * kCols + ci;
    auto get = [&](int o) -> double2 {
      const q2 z = e[o * NZ * kCols];
      return make_double2(fromfix(z.x, eo[o]), fromfix(z.y, eo[o]));
    };
    double2 H1 = get(0), H2 = get(1), H3 = get(2);
    const double nn = nan("");
    if (bad) H1 = H2 = H3 = make_double2(nn, nn);
    const double2 g0 = bf.gzk[2 * k], g1 = bf.gzk[2 * k + 1];  // gz, gz norm; gz s, gz^2 norm
    const double gn = g0.y;
    const long q = (long)k * nkx + i;
    const double2 v = Gv[q];
    if (TEMP) {
      // ht = -i a uT - i gz wT - bym v with the input v, and -vT
      // (crosst.f90:1148-1152,1691-1692)
      double2 uT = get(NO - 3), wT = get(NO - 2), vT = get(NO - 1);
      if (bad) uT = wT = vT = make_double2(nn, nn);
      ((double2 *)bf.Ht + pb)[q] = make_double2(fma(-g.bym, v.x, fma(an, uT.y, gn * wT.y)),
                                                fma(-g.bym, v.y, -fma(an, uT.x, gn * wT.x)));
      ((double2 *)bf.R2 + pb)[q] = make_double2(-(norm * vT.x), -(norm * vT.y));
    }
    // dvordy = i a H1 + i gz H3
    Dn[q] = make_double2(-fma(an, H1.y, gn * H3.y), fma(an, H1.x, gn * H3.x));
    // hg = -i a H3 + i gz (H1 - s v)
    const double gs = g1.x;
    Gn[q] = make_double2(-fma(-gs, v.y, fma(gn, H1.y, -(an * H3.y))),
                         fma(-gs, v.x, fma(gn, H1.x, -(an * H3.x))));
    // hv = -(kx^2 + kz^2) H2
    const double Kn = fma(a, an, g1.y);
    double2 hv = make_double2(-(Kn * H2.x), -(Kn * H2.y));
    if (force && i == 0 && k == 1) hv.x += fj;
    Vv[q] = hv;
    if (i == 0 && k == 0)
      ((double2 *)bf.mrf)[(long)b * g.my + j] = make_double2(norm * H1.x, norm * H3.x);
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// stage 0: shared-memory limits
template <int NZ, bool TEMP>
static cudaError_t launch_zt(const Grid &g, const Bufs &bf, int stage, cudaStream_t st) {
  if (stage == 0) {
    cudaError_t e = cudaFuncSetAttribute(k_z1<NZ, TEMP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)Z1<NZ>::smem);
    return e != cudaSuccess ? e
                            : cudaFuncSetAttribute(k_z3<NZ, TEMP>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)Z3<NZ, TEMP>::smem);
  }
  const unsigned ncb = (unsigned)((g.nkx + kCols - 1) / kCols);
  if (stage == 1)
    k_z1<NZ, TEMP><<<dim3((TEMP ? 4 : 3) * ncb, (unsigned)g.my, (unsigned)g.B), Z1<NZ>::T, Z1<NZ>::smem, st>>>(g, bf);
  else
    k_z3<NZ, TEMP><<<dim3(ncb, (unsigned)g.my, (unsigned)g.B), Z3<NZ, TEMP>::T, Z3<NZ, TEMP>::smem, st>>>(g, bf);
  return cudaGetLastError();
}
template <int NX, bool TEMP, int NP>
static cudaError_t launch_xn(const Grid &g, const Bufs &bf, int stage, int rk, cudaStream_t st) {
  typedef X2<NX, TEMP, NP> C;
  if (stage == 0)
    return cudaFuncSetAttribute(k_x2<NX, TEMP, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)C::smem);
  k_x2<NX, TEMP, NP><<<dim3((unsigned)(g.mgalz / (2 * NP)), (unsigned)g.my, (unsigned)g.B), C::T,
                       C::smem, st>>>(g, bf, rk);
  return cudaGetLastError();
}
template <int NX, bool TEMP>
static cudaError_t launch_xt(const Grid &g, const Bufs &bf, int stage, int rk, cudaStream_t st) {
  if constexpr (NX < 320) {
    const long blocks = (long)(g.mgalz / 4) * g.my * g.B;
    if (stage == 0) {
      const cudaError_t e = launch_xn<NX, TEMP, 2>(g, bf, 0, rk, st);
      if (e != cudaSuccess) return e;
    } else if (blocks >= 5 * 152) {
      return launch_xn<NX, TEMP, 2>(g, bf, stage, rk, st);
    }
  }
  return launch_xn<NX, TEMP, 1>(g, bf, stage, rk, st);
}
template <bool TEMP>
static cudaError_t launch_z(const Grid &g, const Bufs &bf, int stage, cudaStream_t st) {
  switch (g.mgalz) {
    case 32: return launch_zt<32, TEMP>(g, bf, stage, st);
    case 48: return launch_zt<48, TEMP>(g, bf, stage, st);
    case 64: return launch_zt<64, TEMP>(g, bf, stage, st);
    case 80: return launch_zt<80, TEMP>(g, bf, stage, st);
    case 96: return launch_zt<96, TEMP>(g, bf, stage, st);
    case 128: return launch_zt<128, TEMP>(g, bf, stage, st);
    case 160: return launch_zt<160, TEMP>(g, bf, stage, st);
    case 192: return launch_zt<192, TEMP>(g, bf, stage, st);
    case 256: return launch_zt<256, TEMP>(g, bf, stage, st);
    case 384: if constexpr (!TEMP) return launch_zt<384, TEMP>(g, bf, stage, st);
    default: return cudaErrorInvalidValue;
  }
}
template <bool TEMP>
static cudaError_t launch_x(const Grid &g, const Bufs &bf, int stage, int rk, cudaStream_t st) {
  switch (g.mgalx) {
    case 32: return launch_xt<32, TEMP>(g, bf, stage, rk, st);
    case 48: return launch_xt<48, TEMP>(g, bf, stage, rk, st);
    case 64: return launch_xt<64, TEMP>(g, bf, stage, rk, st);
    case 80: return launch_xt<80, TEMP>(g, bf, stage, rk, st);
    case 96: return launch_xt<96, TEMP>(g, bf, stage, rk, st);
    case 128: return launch_xt<128, TEMP>(g, bf, stage, rk, st);
    case 160: return launch_xt<160, TEMP>(g, bf, stage, rk, st);
    case 192: return launch_xt<192, TEMP>(g, bf, stage, rk, st);
    case 256: return launch_xt<256, TEMP>(g, bf, stage, rk, st);
    case 320: return launch_xt<320, TEMP>(g, bf, stage, rk, st);
    case 384: return launch_xt<384, TEMP>(g, bf, stage, rk, st);
    default: return cudaErrorInvalidValue;
  }
}

// Compiled four times: SB_PLANE = 0 (z stages) or 1 (x stage) times SB_TEMP
#ifndef SB_PLANE
#define SB_PLANE 0
#endif
#ifndef SB_TEMP
#define SB_TEMP 0
#endif
#if SB_PLANE == 0 && !SB_TEMP
cudaError_t planeq_z0(const Grid &g, const Bufs &bf, int stage, cudaStream_t st) {
  return launch_z<false>(g, bf, stage, st);
}
cudaError_t planeq_z1(const Grid &g, const Bufs &bf, int stage, cudaStream_t st);
cudaError_t planeq_x0(const Grid &g, const Bufs &bf, int stage, int rk, cudaStream_t st);
cudaError_t planeq_x1(const Grid &g, const Bufs &bf, int stage, int rk, cudaStream_t st);
cudaError_t launch_planeq(const Grid &g, const Bufs &bf, int stage, int rk, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  if (stage != 2) e = g.temp ? planeq_z1(g, bf, stage, st) : planeq_z0(g, bf, stage, st);
  if (e == cudaSuccess && (stage == 2 || stage == 0))
    e = g.temp ? planeq_x1(g, bf, stage, rk, st) : planeq_x0(g, bf, stage, rk, st);
  return e;
}
#elif SB_PLANE == 0
cudaError_t planeq_z1(const Grid &g, const Bufs &bf, int stage, cudaStream_t st) {
  return launch_z<true>(g, bf, stage, st);
}
#elif !SB_TEMP
cudaError_t planeq_x0(const Grid &g, const Bufs &bf, int stage, int rk, cudaStream_t st) {
  return launch_x<false>(g, bf, stage, rk, st);
}
#else
cudaError_t planeq_x1(const Grid &g, const Bufs &bf, int stage, int rk, cudaStream_t st) {
  return launch_x<true>(g, bf, stage, rk, st);
}
#endif

}  // namespace sb
