// sb_bloch.cu -- the y-line work of one explicit RK3 substep on Bloch waves.
//
// On the uniform grid with shear-periodic images u(y + Ly) = shp u(y),
// shp = exp(i psi), every compact operator of the substep (d/dy, d2/dy2, the
// Helmholtz solve) is a circulant matrix twisted by that phase, so the Bloch
// waves exp(i t_m j), t_m = (psi + 2 pi m)/my, diagonalise all of them: d/dy is
// i l1(t), d2/dy2 is l2(t), lapcdy is 1/(l2(t) - k^2), with l1 = 2 sum rh1_d
// sin(d t) / (1 + 2 sum pr1_d cos(d t)) and l2 alike (the symbols of the
// compact schemes, diffy_shear_hepta.f90:68-296).  A line goes through
//   phi      D, phi at the phase of t  -> -d(D)/dy + nu (d2/dy2 - k^2) phi,
//            RK3 update, remap (cross.f90:565-781); phi at the phase of
//            t + c_k dt -> v = lapcdy(phi) -> G, dv/dy -> V
//   omega_y  nu (d2/dy2 - k^2) omega_y, update, remap; d(omega_y)/dy -> D
//   mean     the same for u00 and w00 (nu d2/dy2, forcing, update, d/dy)
// and with the temperature, in a launch of its own after these,
//   tb       d(-vT)/dy + kappa lap(tb), update, remap (crosst.f90:633-636,
//            734-872); gbeta lap(tb) -> Lt, the buoyancy in the phi line of the
//            next substep (whose launch comes first, so Lt is complete)
//   tb00     the same for the mean profile
// with the transforms in 64-bit fixed point (sb_fix.cuh): six (phi) or four
// (omega_y) transforms of my points per line at some 80 integer instructions
// per point, where the banded solves (sb_seg.cuh) spend six solves of 46 FP64
// instructions per complex row at 64 cycles each.
//
// A block takes kCols kx columns of one kz (16 bytes x 8 columns: full lines of
// global and conflict-free rows of shared memory).  Transform of my = R1 R2
// points: thread (n2, column) owns the rows n2 + R2 n1 (R1-point kernels),
// thread (k1, column) the waves k1 + R1 k2 (R2-point kernels); one exchange
// through shared memory between them, none between a forward transform and
// the inverse ones that follow it.
//
// Bound by latency: 12 warps per SM (registers), issue slots 30% in use, the
// FP64 pipe 34%, the ALU pipe 29% (192x96x96); warps wait for the instruction
// before, for rows from global memory, for shared memory and at barriers.
//
// Errors are relative to a line: a part of it that is quiet by more than 2^-55
// of the line's rms drowns there, where a banded solve kept its own accuracy.
#include <cuda_runtime.h>

#include <type_traits>

#include "sb_common.cuh"
#include "sb_fix.cuh"
#include "sb_kernels.h"

// Compiled twelve times: SB_FLOAT_TU = 0 (FP64) or 1 (FP32-mixed) storage times
// SB_LEN = 0 (my 32..80), 1 (96..192), 2 (256..384) times SB_GEN = 0 (explicit,
// no temperature) or 1 (the rest); unit (0, 0, 0) also holds the entry points.
#ifndef SB_FLOAT_TU
#define SB_FLOAT_TU 0
#endif
#ifndef SB_LEN
#define SB_LEN 0
#endif
#ifndef SB_GEN
#define SB_GEN 0
#endif
#define SB_CAT2(a, b, c, d) a##b##_##c##_##d
#define SB_CAT(a, b, c, d) SB_CAT2(a, b, c, d)
#define SB_LINEQ_UNIT(f, l, i) SB_CAT(lineQ_unit, f, l, i)

namespace sb {

namespace {

constexpr int kCols = 8;
constexpr int kNoLen = -(1 << 28);  // scale of nothing

template <typename R> struct V2;
template <> struct V2<double> { typedef double2 t; };
template <> struct V2<float> { typedef float2 t; };
template <typename R>
__device__ __forceinline__ typename V2<R>::t mkv(R a, R b) {
  typename V2<R>::t v;
  v.x = a;
  v.y = b;
  return v;
}
template <typename V>
__device__ __forceinline__ unsigned vtop(V v) {
  const unsigned a = hiword(v.x), b = hiword(v.y);
  return a > b ? a : b;
}
template <typename V>
__device__ __forceinline__ q2 vfix(V v, const QScale &s) {
  return mkq(tofix(v.x, s), tofix(v.y, s));
}

// 1/x by two Newton steps from the 20-bit estimate
__device__ __forceinline__ double recip(double x) {
  double z;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(z) : "d"(x));
  z = fma(z, fma(-x, z, 1.0), z);
  return fma(z, fma(-x, z, 1.0), z);
}

// hides where a pointer comes from, so that the loads of a loop that runs once
// or twice are not moved ahead of it (they would not fit in the registers)
template <typename P>
__device__ __forceinline__ P *here(P *p) {
  asm volatile("" : "+l"(p));
  return p;
}

}  // namespace

template <int N>
struct LineQ {
  static constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2;
  static constexpr int RM = R1 > R2 ? R1 : R2;
  // threads of a block.  Wide: one item a thread in the widest kernel, the
  // shortest chain (one 64x32x32 box: 23 us against 37 with 32 threads,
  // 384x192x192: 755 us against 1223 with 64).  Narrow, for lines up to 96 and
  // enough blocks to fill the GPU: few idle threads between the barriers
  // (192x96x96: 90 us with 64 against 101 with 128; 64 boxes of 64x32x32: 180 us
  // with 32 against 199 with 64)
  static constexpr int kWide = N == 32 ? 64 : N == 48 ? 96 : 128;
  static constexpr int kNarrow = N < 64 ? 32 : N <= 96 ? 64 : 128;
  static constexpr int kShiftF = 2 + Plan<N>::shift;  // twist and forward transform
  static constexpr int kBits = Plan<N>::bits + 2;     // the twist divides by 4
  static constexpr size_t smem = (2 * sizeof(q2) + sizeof(double)) * N * kCols;
};
SB_HD constexpr int floor_log2(int n) { return n < 2 ? 0 : 1 + floor_log2(n / 2); }

// Forward transform, row part: the raw rows of thread (n2, ci) in its slots of
// ex, scaled and twisted, to y[k1][n2] in the same slots.  Row j and y[k1][n2]
// with j = k1 R2 + n2 share slot j, so every part works in place.
template <int N, typename V>
__device__ __forceinline__ void rows_forward(q2 *ex, const QScale &sc, const qw *__restrict__ twist,
                                             int nkx, const qw *__restrict__ tw, int n2, int ci) {
  typedef LineQ<N> L;
  q2 v[L::R1];
#pragma unroll
  for (int n1 = 0; n1 < L::R1; n1++) {
    const int j = n2 + L::R2 * n1;
    v[n1] = qmul<false>(vfix(*(const V *)(ex + j * kCols + ci), sc), twist[(long)j * nkx]);
  }
  Dft<L::R1, -1>::run(v);
#pragma unroll
  for (int k1 = 0; k1 < L::R1; k1++)
    ex[(k1 * L::R2 + n2) * kCols + ci] = qmul<false>(v[k1], tw[n2 * k1]);
}
// inverse transform, row part: y[k1][n2] of thread (n2, ci) to its rows, untwisted
template <int N>
__device__ __forceinline__ void rows_inverse(q2 *ex, const qw *__restrict__ twist, int nkx, int n2,
                                             int ci) {
  typedef LineQ<N> L;
  q2 v[L::R1];
#pragma unroll
  for (int k1 = 0; k1 < L::R1; k1++) v[k1] = ex[(k1 * L::R2 + n2) * kCols + ci];
  Dft<L::R1, 1>::run(v);
#pragma unroll
  for (int n1 = 0; n1 < L::R1; n1++) {
    const int j = n2 + L::R2 * n1;
    ex[j * kCols + ci] = qmul<true>(v[n1], twist[(long)j * nkx]);
  }
}

// registers per thread the kernel is budgeted for (192x96x96: 90 us at 128, 94 at
// 104; 384x192x192: 760 us at 168, 966 at 224)
template <int N>
struct LineQRegs {
  static constexpr int n = LineQ<N>::RM > 12 ? 168 : 128;
};
// rk1 = 1..3: the substep; 0: the start of a run (v and the first derivatives
// from the state, cross.f90:408-445).
// Two passes over the same code (unrolled twice it would not fit in the
// instruction cache, and each warp runs it only once): pass 0 takes the
// right-hand side and the update at the phase of time t, pass 1 the outputs at
// the phase of t + c_k dt.  A pass: rows in, forward, products, inverse, rows out.
// GEN: with the temperature, the semi-implicit branch or both (kept apart: their
// branches cost the plain step 3%).  The semi-implicit viscous branch (explicit = 0, cross.f90:797-989).  Pass 0
// gives the viscous term and (phi) -d(D)/dy apart, the update forms the
// right-hand side -Re ibeta_k (wk + alpha_k nu lap f + f/Dt) of the Helmholtz
// equation in the frame of t + c_k Dt, and pass 1 solves it on the waves,
// f = rhs/(l2 - k^2 - Re ibeta_k/Dt), before the outputs; the state is one
// more output.  The (0,0) line keeps its state.
template <typename R, int N, int T, bool GEN>
__global__ void __launch_bounds__(T, 65536 / (T * LineQRegs<N>::n)) k_lineQ(Grid g, Bufs bf, int rk1,
                                                                              int role0) {
  typedef LineQ<N> L;
  typedef typename V2<R>::t V;
  constexpr int R1 = L::R1, R2 = L::R2;
  constexpr int kN = floor_log2(N), kTgt = Plan<N>::bits;
  const int b = blockIdx.y;
  const Member &M = bf.mem[b];
  if (M.halted) return;  // uniform per block
  extern __shared__ __align__(16) unsigned char smq_raw[];
  q2 *const ex = (q2 *)smq_raw;              // two buffers of N x kCols
  double *const sc = (double *)(ex + 2 * N * kCols);  // factors of the waves
  __shared__ unsigned s_top[2][kCols];  // largest upper words: D, the new state
  // scales of the products: right-hand side, first, second output; semi-implicit:
  // the second of pass 0, the Helmholtz solve
  constexpr int kLens = GEN ? 5 : 3;
  __shared__ int s_len[kLens][kCols];
  const int ncb = (g.nkx + kCols - 1) / kCols, per = g.mz * ncb;
  // role0 = 0: 0 phi, 1 omega_y, 2 mean; role0 = 3: 3 tb, 4 tb00
  const int slot = blockIdx.x / per, role = GEN ? role0 + slot : slot;
  const int r = blockIdx.x - slot * per;
  const bool mean = role == 2 || (GEN && role == 4), scal = GEN && role >= 3;
  const bool im = GEN && g.impl;
  const bool din = role == 0 || scal;  // a second field in pass 0, D or -vT
  const int ci = threadIdx.x & (kCols - 1), n = threadIdx.x / kCols;
  const int k = mean ? 0 : r / ncb;
  const int i0 = mean ? ci : (r - k * ncb) * kCols + ci;
  const bool act = mean ? ci < (scal ? 1 : 2) : i0 < g.nkx;
  const int cm = ci & 1;  // mean: u00 in column 0, w00 in column 1
  const int i = mean ? 0 : (act ? i0 : g.nkx - 1);
  const bool is00 = !mean && i == 0 && k == 0;
  const int nkx = g.nkx;
  const long ps = g.plane / 2;  // complex entries per plane
  const long off = (long)b * (g.field / 2) + (long)k * nkx + i;
  const int rk = rk1 - 1;
  static_assert(T >= kLens * kCols, "one thread per slot");
  if (threadIdx.x < kLens * kCols) {
    if (threadIdx.x < 2 * kCols) (&s_top[0][0])[threadIdx.x] = 0u;
    (&s_len[0][0])[threadIdx.x] = kNoLen;
  }
  __syncthreads();
  const long tb = (long)N * nkx;
  const double a = g.alp * i, gz = g.gam * ((k <= g.nz) ? k : k - g.mz);
  const double k2 = mean ? 0.0 : a * a + gz * gz;
  const double Dt = M.Deltat;
  // of the viscous term of pass 0, and the semi-implicit right-hand side's scales
  const double mnu = scal ? g.kappa : M.nu;
  const double nu = is00 ? 0.0 : im && rk1 > 0 ? kAlpha[rk] * mnu : mnu;
  const double fb = im && rk1 > 0 ? -(scal ? 1.0 / g.kappa : M.Re) * kIbeta[rk] : 0.0, rdt = im ? 1.0 / Dt : 0.0;
  V *f = (V *)(scal ? bf.tb : role == 0 ? bf.phi : bf.vor) + off;
  R *mf = (R *)(scal ? bf.mt : bf.mu) + (long)b * 2 * N + cm;  // mean profile of this column
  // the waves of the state, kept from pass 1 for the next substep's pass 0 (the
  // same phase), and their scale
  const long wst = mean ? 2 : ps, nl = ps + 2;
  q2 *waves = mean ? bf.bwm + (long)(scal * g.B + b) * 2 * N + cm
                   : bf.bw + (scal ? 2 : role) * (g.B * (g.field / 2)) + off;
  int *wscale = bf.bwp + ((long)(scal ? 2 : role & 1) * g.B + b) * nl +
                (mean ? ps + cm : (long)k * nkx + i);
#pragma unroll 1
  for (int ph = rk1 > 0 ? 0 : 1; ph < 2; ph++) {
    // phase tables: slot 0 holds the phases of a step's start, slots 1 and 2
    // those after its first and second substep, its third refills slot 0
    const long o = ((long)((ph == 0 ? rk : rk1) % 3) * g.B + b) * tb + i;
    const qw *tw = bf.btw + o;
    const double *l1 = bf.bl1 + o, *l2 = bf.bl2 + o;
    const int nf = ph == 0 && din ? 2 : 1;  // fields in: the state, D
    const int no = (im && ph == 0 && din) || (ph == 1 && role == 0) ? 2 : 1;  // fields out
    // ---- rows in: D to buffer 1 (phi, pass 0), the state of the start of a run
    // to buffer 0 (in pass 1 the new state is there already)
    const bool rows = ph == 1 || din;
    if (ph == 0 ? din : rk1 == 0) {
      const V *src = ph == 0 ? (const V *)(scal ? bf.R2 : bf.Dn) + off : f;
      unsigned top = 0;
#pragma unroll 4
      for (int j = n; j < N; j += T / kCols) {
        const V w = mean && ph == 1 ? mkv<R>(mf[2 * j], (R)0) : src[(long)j * ps];
        *(V *)(ex + ((1 - ph) * N + j) * kCols + ci) = w;
        top = max(top, vtop(w));
      }
      atomicMax(&s_top[ph][ci], top);
    }
    if (rows) __syncthreads();
    // scales: 0 the state (pass 0: of the waves kept from the last pass 1), 1 D
    const QScale sr = qscale(s_top[ph][ci], L::kBits);
    const int kept = ph == 0 ? *wscale : 0;
    int w0 = ph == 0 ? kept : sr.weight();
    const int w1 = sr.weight();
    const bool bad = (ph == 0 && kept == kNoLen) || (rows && sr.bad);
    if (rows) {
#pragma unroll 1
      for (int it = n; it < R2; it += T / kCols)
        rows_forward<N, V>(ex + (1 - ph) * N * kCols, sr, tw, nkx, bf.bftw, it, ci);
      __syncthreads();
    }
    const int eb = L::kShiftF + Plan<N>::shift + 2 - kN - kTgt;
    const bool solve = im && ph == 1 && rk1 > 0;
    if constexpr (GEN) {
      if (solve) {
        // ---- the Helmholtz solve; the waves of the new state stay in buffer 0
        const double dtr = -fb * rdt;
#pragma unroll 1
        for (int k1 = n; k1 < R1; k1 += T / kCols) {
          const double *l = l2 + (long)k1 * nkx;
          q2 *e = ex + k1 * R2 * kCols + ci;
          q2 x[R2];
#pragma unroll
          for (int w = 0; w < R2; w++) x[w] = e[w * kCols];
          Dft<R2, -1>::run(x);
          int la = kNoLen;
#pragma unroll
          for (int w = 0; w < R2; w++) {
            const double c = recip(is00 ? 1.0 : l[(long)(R1 * w) * nkx] - k2 - dtr);
            sc[(k1 * R2 + w) * kCols + ci] = c;
            e[w * kCols] = x[w];
            la = max(la, qlen(x[w]) + qexp(c));
          }
          atomicMax(&s_len[4][ci], la);
        }
        __syncthreads();
        const int len = s_len[4][ci] + 1, sh = kTgt - len;
#pragma unroll 1
        for (int k1 = n; k1 < R1; k1 += T / kCols) {
          q2 *e = ex + k1 * R2 * kCols + ci;
          q2 x[R2];
#pragma unroll
          for (int w = 0; w < R2; w++) {
            x[w] = qscaled(e[w * kCols], sc[(k1 * R2 + w) * kCols + ci], sh);
            e[w * kCols] = x[w];
          }
          Dft<R2, 1>::run(x);
#pragma unroll
          for (int w = 0; w < R2; w++) e[(N + w) * kCols] = qmul<false>(x[w], bf.bitw[w * k1]);
        }
        __syncthreads();
#pragma unroll 1
        for (int it = n; it < R2; it += T / kCols)
          rows_inverse<N>(ex + N * kCols, here(tw), nkx, it, ci);
        __syncthreads();
        const bool none = bad || qrange(eb - w0 + len);
        const R nn = (R)nan("");
        if (act && !is00)
#pragma unroll 1
          for (int j = n; j < N; j += T / kCols) {
            const q2 z = ex[(N + j) * kCols + ci];
            const V v = none ? mkv<R>(nn, nn)
                             : mkv<R>(qout<R>(z.x, eb - w0 + len), qout<R>(z.y, eb - w0 + len));
            if (mean) mf[2 * j] = v.x;
            else f[(long)j * ps] = v;
          }
        w0 += sh;
      }
    }
    const double cn = ph == 0 ? nu : is00 ? 0.0 : g.gbeta, cnk2 = cn * k2;
    // ---- products.  Pass 0: nu (l2 - k^2) f - i l1 D; pass 1: phi f/(l2 - k^2)
    // and i l1 of it, else i l1 f.  The waves stay in the thread's own slots
    // while the scale of each product is found over the whole line.
#pragma unroll 1
    for (int k1 = n; k1 < R1; k1 += T / kCols) {
      const long p0 = (long)k1 * nkx;
      double *cw = sc + k1 * R2 * kCols + ci;
      // nu (l2 - k^2) or gbeta (l2 - k^2), 1/(l2 - k^2), l1: three arms that the
      // compiler turns into selects, so that the waves' loads and chains overlap
      // (with a fourth, or the reciprocal inlined from a function, it branched
      // for each wave: 64x32x32 29 us against 23)
#pragma unroll
      for (int q = 0; q < R2; q++) {
        const long p = p0 + (long)(R1 * q) * nkx;
        double c;
        if (ph == 0 || scal) {
          c = fma(cn, l2[p], -cnk2);
        } else if (role == 0) {
          const double den = l2[p] - k2;
          double z;
          asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(z) : "d"(den));
          z = fma(z, fma(-den, z, 1.0), z);
          z = fma(z, fma(-den, z, 1.0), z);
          c = is00 ? 0.0 : z;
        } else {
          c = l1[p];
        }
        cw[q * kCols] = c;
      }
#pragma unroll 1
      for (int q = 0; q < nf; q++) {
        q2 *e = ex + (q * N + k1 * R2) * kCols + ci;
        const double *l = here(l1) + p0;
        q2 x[R2];
        if (ph == 0 && q == 0) {
          const q2 *wv = waves + k1 * wst;
#pragma unroll
          for (int w = 0; w < R2; w++) x[w] = wv[(long)(R1 * w) * wst];
        } else {
#pragma unroll
          for (int w = 0; w < R2; w++) x[w] = e[w * kCols];
          if (!solve) Dft<R2, -1>::run(x);
        }
        if (ph == 1 && act) {
          q2 *wv = waves + k1 * wst;
#pragma unroll
          for (int w = 0; w < R2; w++) wv[(long)(R1 * w) * wst] = x[w];
        }
        int la = kNoLen, lb = kNoLen;
#pragma unroll
        for (int w = 0; w < R2; w++) {
          e[w * kCols] = x[w];
          const int len = qlen(x[w]), e1 = qexp(l[(long)(R1 * w) * nkx]), ec = qexp(cw[w * kCols]);
          la = max(la, len + (q ? e1 : ec));
          lb = max(lb, len + ec + e1 + 1);
        }
        atomicMax(&s_len[im && ph == 0 && q ? 3 : ph][ci], la - (ph == 0 ? (q ? w1 : w0) : 0));
        if (ph == 1 && no > 1) atomicMax(&s_len[2][ci], lb);
      }
      if (ph == 1 && k1 == 0 && act) *wscale = bad ? kNoLen : w0;
    }
    __syncthreads();
    // scales of the outputs; in pass 0 of the sum of two terms
    const int len1 = s_len[ph][ci] + (!im && ph == 0 ? 2 : 1);
    const int len2 = s_len[GEN && ph == 0 ? 3 : 2][ci] + 1;
#pragma unroll 1
    for (int k1 = n; k1 < R1; k1 += T / kCols) {
      const double *cw = sc + k1 * R2 * kCols + ci;
      q2 y[R2];
#pragma unroll 1
      for (int q = max(nf, no) - 1; q >= 0; q--) {
        // pass 0: q = 1 D, 0 f, added; pass 1: q = 1 the second output, 0 the first
        const q2 *e = ex + ((nf > 1 ? q : 0) * N + k1 * R2) * kCols + ci;
        const bool first = no > 1 || q == nf - 1;
        const double *l = here(l1) + (long)k1 * nkx;
        const qw *it = here(bf.bitw);
        const int sh = kTgt - (no > 1 && q ? len2 : len1) - (ph == 0 ? (q ? w1 : w0) : 0);
#pragma unroll
        for (int w = 0; w < R2; w++) {
          double d = cw[w * kCols];
          if (q) {
            const double m = l[(long)(R1 * w) * nkx];
            d = ph == 1 ? d * m : m;
          }
          q2 z = qscaled(e[w * kCols], d, sh);
          // times -i (D), i (-vT, d/dy of an output) or 1
          if (ph == 0 ? q : (role == 1 || role == 2 || q))
            z = ph == 0 && !scal ? qrot<-1>(z) : qrot<1>(z);
          y[w] = first ? z : y[w] + z;
        }
        if (no > 1 || q == 0) {
          Dft<R2, 1>::run(y);
          q2 *eo = ex + ((no > 1 ? q : 0) * N + k1 * R2) * kCols + ci;
#pragma unroll
          for (int w = 0; w < R2; w++) eo[w * kCols] = qmul<false>(y[w], it[w * k1]);
        }
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int it = n; it < no * R2; it += T / kCols) {
      const int q = it >= R2;
      rows_inverse<N>(ex + q * N * kCols, here(tw), nkx, it - q * R2, ci);
    }
    __syncthreads();
    // ---- rows out
    if (ph == 1) {
      const int e0 = eb - w0;
      const bool nan1 = bad || qrange(e0 + len1), nan2 = bad || qrange(e0 + len2);
      const R nn = (R)nan("");
      if (mean) {
        if (scal) return;
        R *dst = (R *)bf.mdu + (long)b * 2 * N + cm;
        if (act)
#pragma unroll 1
          for (int j = n; j < N; j += T / kCols)
            dst[2 * j] = nan1 ? nn : qout<R>(ex[j * kCols + ci].x, e0 + len1);
      } else if (act) {
#pragma unroll 1
        for (int q = 0; q < no; q++) {
          // the (0,0) line of v keeps the value zero it is given at the start of a run
          if (role == 0 && q == 0 && is00 && rk1 > 0) continue;
          V *dst = (V *)(scal ? bf.Lt : role != 0 ? bf.D : q ? bf.V : bf.G) + off;
          const int eo = e0 + (q ? len2 : len1);
          const bool none = q ? nan2 : nan1;
#pragma unroll 2
          for (int j = n; j < N; j += T / kCols) {
            const q2 z = ex[(q * N + j) * kCols + ci];
            dst[(long)j * ps] = none ? mkv<R>(nn, nn) : mkv<R>(qout<R>(z.x, eo), qout<R>(z.y, eo));
          }
        }
      }
      return;
    }
    // RK3 accumulation and update, zeta store, remaps (cross.f90:694-781)
    const int eo = eb + len1;
    const int ed = eb + len2;  // semi-implicit: of -d(D)/dy
    const bool nanr = bad || qrange(eo) || (im && no > 1 && qrange(ed));
    const R gk = (R)kGama[rk], zk = (R)kZeta[rk], dtr = (R)Dt;
    unsigned top = 0;
    if (mean) {
      R *mwk = (R *)(scal ? bf.mtwk : bf.mwk) + (long)b * 2 * N + cm;
      const R *mrf = (const R *)bf.mrf + (long)b * 2 * N + cm;
      const bool damp = g.damp && ci == 0 && !scal, xf = g.force == -1 && ci == 0 && !scal;
#pragma unroll 1
      for (int j = n; j < N; j += T / kCols) {
        R un = (R)0;
        if (act) {
          // forcing and damping (cross.f90:622-626; operators.f90:60-78)
          R rf0 = scal ? (R)0 : mrf[2 * j];
          if (xf) rf0 = (R)((double)rf0 + g.xforce);
          if (damp) {
            const double y = (double)j * g.dy - 0.5 * g.Ly;
            const double hw = 1.0 - (0.25 * (1.0 + tanh(6.0 * (g.damp_a - y) / g.lz + 3.0))) *
                                        (1.0 + tanh(6.0 * (g.damp_a + y) / g.lz + 3.0));
            rf0 = (R)((double)rf0 - g.damp_up * hw * (double)mf[2 * j]);
          }
          const ll z = ex[j * kCols + ci].x;
          if (im) {
            if (scal) rf0 = nanr ? (R)nan("") : qout<R>(ex[(N + j) * kCols + ci].x, ed);
            const R wk = (rk == 0) ? gk * rf0 : mwk[2 * j] + gk * rf0;
            const double vis = nanr ? nan("") : fromfix(z, eo);
            un = (R)(fb * (((double)wk + vis) + rdt * (double)mf[2 * j]));
            if (rk < 2) mwk[2 * j] = zk * rf0;
          } else {
            const R rf = rf0 + (nanr ? (R)nan("") : qout<R>(z, eo));
            R wk = (rk == 0) ? gk * rf : mwk[2 * j] + gk * rf;
            un = mf[2 * j] + dtr * wk;
            if (rk < 2) wk = rf * zk;
            mf[2 * j] = un;
            mwk[2 * j] = wk;
          }
        }
        const V w = mkv<R>(un, (R)0);
        top = max(top, vtop(w));
        *(V *)(ex + j * kCols + ci) = w;
      }
    } else {
      const V *rhs = (const V *)(scal ? bf.Ht : role == 0 ? bf.V : bf.Gn) + off;
      V *fwk = (V *)(scal ? bf.tbwk : role == 0 ? bf.phiwk : bf.vorwk) + off;
      const double2 *m1 = bf.bm1 + (long)b * tb + i, *m2 = bf.bm2 + (long)b * tb + i;
      const V none = mkv<R>((R)0, (R)0);
      const V *buoy = (const V *)bf.Lt + off;
      // one loop for each form: a branch inside waits for every row's loads
      auto update = [&](auto with, auto implicit) {
        constexpr bool IM = decltype(implicit)::value;
#pragma unroll 2
        for (int j = n; j < N; j += T / kCols) {
          const long q = (long)j * ps;
          const V fo = f[q], rh = rhs[q], w0 = rk > 0 ? fwk[q] : none;
          const q2 z = ex[j * kCols + ci];
          V h = rh;
          if constexpr (!IM) {
            h = mkv<R>(rh.x + qout<R>(z.x, eo), rh.y + qout<R>(z.y, eo));
          } else if (din) {
            const q2 d = ex[(N + j) * kCols + ci];
            h = mkv<R>(rh.x + qout<R>(d.x, ed), rh.y + qout<R>(d.y, ed));
          }
          if constexpr (decltype(with)::value) {
            const V t = buoy[q];
            h = mkv<R>(h.x + t.x, h.y + t.y);
          }
          if (nanr) h = mkv<R>((R)nan(""), (R)nan(""));
          V wk = mkv<R>(w0.x + gk * h.x, w0.y + gk * h.y);
          const double2 p2 = m2[(long)j * nkx];
          double fx, fy;
          if constexpr (IM) {
            fx = fb * (((double)wk.x + fromfix(z.x, eo)) + rdt * (double)fo.x);
            fy = fb * (((double)wk.y + fromfix(z.y, eo)) + rdt * (double)fo.y);
          } else {
            fx = (double)(fo.x + dtr * wk.x), fy = (double)(fo.y + dtr * wk.y);
          }
          V fn = mkv<R>((R)fma(fx, p2.x, -(fy * p2.y)), (R)fma(fy, p2.x, fx * p2.y));
          if (IM && is00) fn = fo;
          if (rk < 2) {
            // zeta_k h in the frame of the next substep; zeta_k is in the phase
            const double2 p1 = m1[(long)j * nkx];
            const double hx = (double)h.x, hy = (double)h.y;
            wk = mkv<R>((R)fma(hx, p1.x, -(hy * p1.y)), (R)fma(hy, p1.x, hx * p1.y));
          }
          if (act) {
            if (!IM) f[q] = fn;
            if (!IM || rk < 2) fwk[q] = wk;
          }
          top = max(top, vtop(fn));
          *(V *)(ex + j * kCols + ci) = fn;
        }
      };
      constexpr std::true_type yes;
      constexpr std::false_type no_;
      const bool with = GEN && g.temp && role == 0;
      if constexpr (GEN) {
        if (im) {
          if (with) update(yes, yes);
          else update(no_, yes);
        } else if (with) {
          update(yes, no_);
        }
      }
      if (!im && !with) update(no_, no_);
    }
    atomicMax(&s_top[1][ci], top);
  }
}

#if !SB_GEN
// The LES y-operators (iuse_LES, cross.f90:565-608,639-647) at the phase of t,
// between k_bloch and k_lineQ:
//   role 0  hg += d(rhgc2)/dy                                       (L2 -> Gn)
//   role 1  hv -= (kx^2 + kz^2 + d2/dy2) rhvc2                       (L1 -> V)
//   mean    rf0u += d(T12_00)/dy, rf0w += d(T23_00)/dy              (txy -> mrf)
// One transform and its inverse a line, where k_lineL spends a banded FP64 solve
// (384x192x192 mixed: 264 us against 909; 192x96x96 FP64: 34 against 121).  Bound
// by latency, as k_lineQ.
template <typename R, int N, int T>
__global__ void __launch_bounds__(T, 65536 / (T * LineQRegs<N>::n)) k_lineLQ(Grid g, Bufs bf, int rk) {
  typedef LineQ<N> L;
  typedef typename V2<R>::t V;
  constexpr int R1 = L::R1, R2 = L::R2;
  constexpr int kN = floor_log2(N), kTgt = Plan<N>::bits;
  const int b = blockIdx.y;
  if (bf.mem[b].halted) return;  // uniform per block
  extern __shared__ __align__(16) unsigned char smq_raw[];
  q2 *const ex = (q2 *)smq_raw;
  __shared__ unsigned s_top[kCols];
  __shared__ int s_len[kCols];
  const int ncb = (g.nkx + kCols - 1) / kCols, per = g.mz * ncb;
  const int role = blockIdx.x / per, r = blockIdx.x - role * per;
  const bool mean = role == 2;
  const int ci = threadIdx.x & (kCols - 1), n = threadIdx.x / kCols;
  const int k = mean ? 0 : r / ncb;
  const int i0 = mean ? ci : (r - k * ncb) * kCols + ci;
  const bool act = mean ? ci < 2 : i0 < g.nkx;
  const int cm = ci & 1;
  const int i = mean ? 0 : (act ? i0 : g.nkx - 1);
  const int nkx = g.nkx;
  const long ps = g.plane / 2, off = (long)b * (g.field / 2) + (long)k * nkx + i;
  if (threadIdx.x < kCols) {
    s_top[threadIdx.x] = 0u;
    s_len[threadIdx.x] = kNoLen;
  }
  __syncthreads();
  const double a = g.alp * i, gz = g.gam * ((k <= g.nz) ? k : k - g.mz);
  const double k2 = a * a + gz * gz;
  const long o = ((long)((rk - 1) % 3) * g.B + b) * N * nkx + i;
  const qw *tw = bf.btw + o;
  const V *src = (const V *)(role == 0 ? bf.L2 : bf.L1) + off;
  const R *tx = (const R *)bf.txy + (long)b * 2 * N + cm;
  unsigned top = 0;
#pragma unroll 4
  for (int j = n; j < N; j += T / kCols) {
    const V w = mean ? mkv<R>(tx[2 * j], (R)0) : src[(long)j * ps];
    *(V *)(ex + j * kCols + ci) = w;
    top = max(top, vtop(w));
  }
  atomicMax(&s_top[ci], top);
  __syncthreads();
  const QScale sr = qscale(s_top[ci], L::kBits);
#pragma unroll 1
  for (int it = n; it < R2; it += T / kCols)
    rows_forward<N, V>(ex, sr, tw, nkx, bf.bftw, it, ci);
  __syncthreads();
  // i l1 or -(l2 + k^2)
  const double *l = (role == 1 ? bf.bl2 : bf.bl1) + o;
  auto factor = [&](double v) { return role == 1 ? -(v + k2) : v; };
#pragma unroll 1
  for (int k1 = n; k1 < R1; k1 += T / kCols) {
    q2 *e = ex + k1 * R2 * kCols + ci;
    const double *lk = l + (long)k1 * nkx;
    q2 x[R2];
#pragma unroll
    for (int w = 0; w < R2; w++) x[w] = e[w * kCols];
    Dft<R2, -1>::run(x);
    int la = kNoLen;
#pragma unroll
    for (int w = 0; w < R2; w++) {
      e[w * kCols] = x[w];
      la = max(la, qlen(x[w]) + qexp(factor(lk[(long)(R1 * w) * nkx])));
    }
    atomicMax(&s_len[ci], la);
  }
  __syncthreads();
  const int len = s_len[ci] + 1;
#pragma unroll 1
  for (int k1 = n; k1 < R1; k1 += T / kCols) {
    q2 *e = ex + k1 * R2 * kCols + ci;
    const double *lk = here(l) + (long)k1 * nkx;
    q2 y[R2];
#pragma unroll
    for (int w = 0; w < R2; w++) {
      y[w] = qscaled(e[w * kCols], factor(lk[(long)(R1 * w) * nkx]), kTgt - len);
      if (role != 1) y[w] = qrot<1>(y[w]);
    }
    Dft<R2, 1>::run(y);
#pragma unroll
    for (int w = 0; w < R2; w++) e[w * kCols] = qmul<false>(y[w], bf.bitw[w * k1]);
  }
  __syncthreads();
#pragma unroll 1
  for (int it = n; it < R2; it += T / kCols) rows_inverse<N>(ex, here(tw), nkx, it, ci);
  __syncthreads();
  const int eo = L::kShiftF + Plan<N>::shift + 2 - kN - kTgt - sr.weight() + len;
  const bool none = sr.bad || qrange(eo);
  const R nn = (R)nan("");
  if (!act || (role == 1 && i == 0 && k == 0)) return;
  if (mean) {
    R *mrf = (R *)bf.mrf + (long)b * 2 * N + cm;
    for (int j = n; j < N; j += T / kCols)
      mrf[2 * j] += none ? nn : qout<R>(ex[j * kCols + ci].x, eo);
    return;
  }
  V *dst = (V *)(role == 1 ? bf.V : bf.Gn) + off;
#pragma unroll 2
  for (int j = n; j < N; j += T / kCols) {
    const q2 z = ex[j * kCols + ci];
    const V d = dst[(long)j * ps];
    dst[(long)j * ps] = none ? mkv<R>(nn, nn) : mkv<R>(d.x + qout<R>(z.x, eo), d.y + qout<R>(z.y, eo));
  }
}
#endif

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <typename R, int N, int T, bool GEN>
static cudaError_t launch_n(const Grid &g, const Bufs &bf, int rk, cudaStream_t st, bool prep,
                            unsigned blocks, int role0) {
  if (prep)
    return cudaFuncSetAttribute(k_lineQ<R, N, T, GEN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)LineQ<N>::smem);
  k_lineQ<R, N, T, GEN><<<dim3(blocks, (unsigned)g.B), T, LineQ<N>::smem, st>>>(g, bf, rk, role0);
  return cudaGetLastError();
}
template <typename R, int N, bool GEN>
static cudaError_t launch_t(const Grid &g, const Bufs &bf, int rk, cudaStream_t st, bool prep) {
  constexpr int W = LineQ<N>::kWide, S = LineQ<N>::kNarrow;
  const unsigned per = (unsigned)(g.mz * ((g.nkx + kCols - 1) / kCols));
  cudaError_t e = cudaSuccess;
  // the velocity's roles, then the temperature's (its Lt is read by the former)
  for (int role0 = 0; e == cudaSuccess && role0 < (g.temp ? 6 : 3); role0 += 3) {
    const unsigned blocks = (role0 ? 1 : 2) * per + 1;
    bool narrow = false;
    if constexpr (W != S && (!GEN || S >= 64)) {
      narrow = (long)blocks * g.B >= 5 * 152;
      if (prep || narrow) e = launch_n<R, N, S, GEN>(g, bf, rk, st, prep, blocks, role0);
    }
    if (e == cudaSuccess && !narrow)
      e = launch_n<R, N, W, GEN>(g, bf, rk, st, prep, blocks, role0);
    if (prep && narrow) e = launch_n<R, N, W, GEN>(g, bf, rk, st, prep, blocks, role0);
  }
  return e;
}

#if !SB_GEN
template <typename R, int N, int T>
static cudaError_t launch_ln(const Grid &g, const Bufs &bf, int rk, cudaStream_t st, bool prep,
                             unsigned blocks) {
  constexpr int smem = (int)sizeof(q2) * N * kCols;
  if (prep)
    return cudaFuncSetAttribute(k_lineLQ<R, N, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  k_lineLQ<R, N, T><<<dim3(blocks, (unsigned)g.B), T, smem, st>>>(g, bf, rk);
  return cudaGetLastError();
}
template <typename R, int N>
static cudaError_t launch_lt(const Grid &g, const Bufs &bf, int rk, cudaStream_t st, bool prep) {
  const unsigned blocks = (unsigned)(2 * g.mz * ((g.nkx + kCols - 1) / kCols) + 1);
  return launch_ln<R, N, LineQ<N>::kWide>(g, bf, rk, st, prep, blocks);
}
#endif

#if SB_FLOAT_TU
typedef float UnitR;
#else
typedef double UnitR;
#endif
// les: k_lineLQ instead (in the units without SB_GEN)
cudaError_t SB_LINEQ_UNIT(SB_FLOAT_TU, SB_LEN, SB_GEN)(const Grid &g, const Bufs &bf, int rk,
                                                        cudaStream_t st, bool prep, bool les) {
#if SB_GEN
#define SB_CASE(N) \
  case N: return launch_t<UnitR, N, true>(g, bf, rk, st, prep);
#else
#define SB_CASE(N)                                                   \
  case N:                                                            \
    return les ? launch_lt<UnitR, N>(g, bf, rk, st, prep) : launch_t<UnitR, N, false>(g, bf, rk, st, prep);
#endif
  switch (g.my) {
#if SB_LEN == 0
    SB_CASE(32) SB_CASE(48) SB_CASE(64) SB_CASE(80)
#elif SB_LEN == 1
    SB_CASE(96) SB_CASE(128) SB_CASE(160) SB_CASE(192)
#else
    SB_CASE(256) SB_CASE(320) SB_CASE(384)
#endif
    default: return cudaErrorInvalidValue;
  }
#undef SB_CASE
}

#if !SB_FLOAT_TU && SB_LEN == 0 && !SB_GEN
// ---------------------------------------------------------------------------
// the phase tables of slot sn for a box: per (row or wave m, kx) the twist
// exp(-i psi m/my) and the symbols l1, l2 at t = (psi + 2 pi m)/my.  psi is
// -kx xofft as a fraction of a turn: an error of the phase itself matters no
// more than the rounding of exp(-i kx xofft), but the twists of the rows must
// agree with each other to better than FP64 (their noise would be amplified by
// (my/(dy k))^2 in a second derivative), hence the fixed-point qturn.  The
// symbols are written in sin and cos of t/2, taken from the nearer of 0 and
// pi, so that neither the long waves nor the ends of the spectrum cancel.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(64) k_bloch(Grid g, Bufs bf, int rk) {
  const int b = blockIdx.y;
  const Member &M = bf.mem[b];
  if (M.halted) return;
  const int N = g.my, nkx = g.nkx, sn = rk % 3;
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= (long)N * nkx) return;
  const int m = (int)(p / nkx), i = (int)(p - (long)m * nkx);
  constexpr double kPi = 3.14159265358979323846, kInv = 0.15915494309189533577;  // 1/(2 pi)
  double turn = 0.0;
  if (fabs(g.s) > 0.01) {
    const double arg = (-(g.alp * i)) * M.xwt[rk];
    const double n = rint(arg * kInv);
    double a = fma(-n, 6.283185307179586232, arg);
    a = fma(-n, 2.4492935982947064e-16, a);  // 2 pi less its double
    turn = a * kInv;
  }
  const ll X = __double2ll_rn(turn * 18446744073709551616.0);
  if (rk > 0) {
    // moving-frame phases exp(i kx y_j tau) (operators.f90:119-123), the work
    // array's with zeta_k (cross.f90:752-781)
    const double Dt = M.Deltat, ay = (g.alp * i) * ((double)m * g.dy - 0.5 * g.Ly);
    const double f1 = (rk == 1) ? -(kGama[0] * Dt * g.s) : -((kGama[1] + kZeta[0]) * Dt * g.s);
    const double f2 = (rk == 1) ? -(g.s * (kCa[0] * Dt)) : -(g.s * (kCa[rk - 1] - kCa[rk - 2]) * Dt);
    auto phase = [&](double f, double z) {
      const double t = ay * f * kInv;
      const qw w = qturn(__double2ll_rn((rint(t) - t) * 18446744073709551616.0), 1, 1, bf.bturn);
      return make_double2(z * fromfix((ll)((ull)(ll)w.hr << 32) + w.lr, -62),
                          z * fromfix((ll)((ull)(ll)w.hi << 32) + w.li, -62));
    };
    const long q = (long)b * N * nkx + p;
    bf.bm2[q] = phase(f2, 1.0);
    if (rk < 3) bf.bm1[q] = phase(f1, kZeta[rk - 1]);
  }
  const long o = ((long)sn * g.B + b) * N * nkx + p;
  bf.btw[o] = qturn(X, m, N, bf.bturn);
  // t/2 = pi (turn + ms)/N for |t| <= pi/2, else pi/2 less the rest
  const int ms = 2 * m > N ? m - N : m;
  const bool far = 4 * (ms < 0 ? -ms : ms) > N;
  const double sg = ms < 0 ? -1.0 : 1.0;
  const double h = far ? (0.5 * N - sg * ms) - sg * turn : (double)ms + turn;
  double s, c;
  sincos(kPi * h / (double)N, &s, &c);
  if (far) {
    const double t = s;
    s = sg * c;
    c = t;
  }
  const double s2 = s * s, c2 = c * c, st2 = 4.0 * s2 * c2;  // sin^2 t
  const double a3 = 3.0 - 4.0 * s2, b3 = 4.0 * c2 - 3.0;     // sin and cos of 3 t/2 over those of t/2
  const double n1 = 4.0 * s * c * (g.bn1p + 4.0 * (g.rh1[5] * c2 - g.rh1[6] * st2));
  const double p1 = g.bp1p + 4.0 * (g.bpr1[0] * c2 - g.bpr1[1] * st2 + g.bpr1[2] * (c2 * b3 * b3));
  const double n2 = g.bn20 - 4.0 * (g.rh2[4] * s2 + g.rh2[5] * st2 + g.rh2[6] * (s2 * a3 * a3));
  const double p2 = g.bp2p + 4.0 * (g.pr2[4] * c2 - g.pr2[5] * st2 + g.pr2[6] * (c2 * b3 * b3));
  bf.bl1[o] = n1 / p1;
  bf.bl2[o] = n2 / p2;
}

typedef cudaError_t LineQUnit(const Grid &, const Bufs &, int, cudaStream_t, bool, bool);
LineQUnit lineQ_unit0_1_0, lineQ_unit0_2_0, lineQ_unit1_0_0, lineQ_unit1_1_0, lineQ_unit1_2_0;
LineQUnit lineQ_unit0_0_1, lineQ_unit0_1_1, lineQ_unit0_2_1, lineQ_unit1_0_1, lineQ_unit1_1_1,
    lineQ_unit1_2_1;
static cudaError_t lineQ(const Grid &g, const Bufs &bf, int rk, cudaStream_t st, bool prep,
                         bool les) {
  static LineQUnit *const unit[2][2][3] = {
      {{lineQ_unit0_0_0, lineQ_unit0_1_0, lineQ_unit0_2_0},
       {lineQ_unit1_0_0, lineQ_unit1_1_0, lineQ_unit1_2_0}},
      {{lineQ_unit0_0_1, lineQ_unit0_1_1, lineQ_unit0_2_1},
       {lineQ_unit1_0_1, lineQ_unit1_1_1, lineQ_unit1_2_1}}};
  return unit[!les && (g.impl || g.temp) ? 1 : 0][g.prec ? 1 : 0][g.my < 96 ? 0 : g.my < 256 ? 1 : 2](g, bf, rk, st,
                                                                                 prep, les);
}

// the step, explicit (with or without LES) or semi-implicit,
// on the transform lengths; the y filter and dealiasing keep the banded solves
bool line_bloch_ok(const Grid &g) { return !g.ydeal && fix_length(g.my); }

cudaError_t launch_lineQ(const Grid &g, const Bufs &bf, int rk, cudaStream_t st) {
  return lineQ(g, bf, rk, st, false, false);
}
cudaError_t launch_lineLQ(const Grid &g, const Bufs &bf, int rk, cudaStream_t st) {
  return lineQ(g, bf, rk, st, false, true);
}
cudaError_t prepare_lineQ(const Grid &g, const Bufs &bf) {
  const cudaError_t e = g.les ? lineQ(g, bf, 0, 0, true, true) : cudaSuccess;
  return e != cudaSuccess ? e : lineQ(g, bf, 0, 0, true, false);
}
cudaError_t launch_bloch(const Grid &g, const Bufs &bf, int rk, cudaStream_t st) {
  const long n = (long)g.my * g.nkx;
  k_bloch<<<dim3((unsigned)((n + 63) / 64), (unsigned)g.B), 64, 0, st>>>(g, bf, rk);
  return cudaGetLastError();
}

#endif  // unit (0, 0, 0)

}  // namespace sb
