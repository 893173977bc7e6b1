// sb_krylov.cu -- device-resident Krylov spaces for the Newton-Krylov and
// Arnoldi searches, and the state <-> unknown-vector maps of a handle.
//
// The reference keeps its Krylov vectors on MPI rank 0 and forms every inner
// product, vector update and norm there (dotp, vecadd, norm, gmres_shear.f90:
// 3680-3919; the MGS loops of gmres_k_shear 1905-2207 and arnoldi_shear.f90:
// 222-330).  Here the vectors live in one device buffer of FP64 columns, the
// products of a block of columns are formed with fixed-order (deterministic)
// reductions, and only the small matrices of coefficients cross to the host,
// where the Hessenberg least-squares problems are solved.  The unknown vector
// is `throwing`'s (gmres_shear.f90:2229-2426, iuse_fou_mode 2): u00, w00 and,
// per y plane, the selected (kz, kx) entries of omega_y and phi; the period
// map reads and writes it on the device (sb_set_state_packed,
// sb_get_state_packed), so no state crosses the host during a search.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <string>

#include "../../include/shearbox.h"
#include "sb_common.cuh"
#include "sb_fix.cuh"
#include "sb_kernels.h"

namespace sb {
void set_error(const std::string &msg);
}

using sb::Grid;

namespace {

int kfail(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  sb::set_error(buf);
  return code;
}
#define KCK(x)                                                                    \
  do {                                                                            \
    cudaError_t e_ = (x);                                                         \
    if (e_ != cudaSuccess)                                                        \
      return kfail(3, "%s failed: %s (%s:%d)", #x, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

constexpr int kThreads = 256;
constexpr int kUThreads = 128;  // of the fixed-point update
constexpr int kTA = 4;  // columns of the left block per gram tile
constexpr int kTB = 8;  // columns of the right block per gram tile
constexpr int kMaxSrc = 8;

// ---------------------------------------------------------------------------
// C[a][b] = sum_r A[r, a0 + a] B[r, b0 + b] over rows [r0, r1): partial sums
// per row chunk, then a fixed-order sum over the chunks.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
k_gram(const double *__restrict__ V, long ld, long r0, long r1, long chunk, int a0, int m, int b0,
       int p, double *__restrict__ part) {
  const int ta = blockIdx.y * kTA, tb = blockIdx.z * kTB;
  const long lo = r0 + (long)blockIdx.x * chunk;
  const long hi = min(r1, lo + chunk);
  double acc[kTA][kTB];
#pragma unroll
  for (int a = 0; a < kTA; a++)
#pragma unroll
    for (int b = 0; b < kTB; b++) acc[a][b] = 0.0;
  const double *A[kTA];
  const double *B[kTB];
#pragma unroll
  for (int a = 0; a < kTA; a++) A[a] = V + (long)(a0 + min(ta + a, m - 1)) * ld;
#pragma unroll
  for (int b = 0; b < kTB; b++) B[b] = V + (long)(b0 + min(tb + b, p - 1)) * ld;
  for (long r = lo + threadIdx.x; r < hi; r += kThreads) {
    double va[kTA], vb[kTB];
#pragma unroll
    for (int a = 0; a < kTA; a++) va[a] = A[a][r];
#pragma unroll
    for (int b = 0; b < kTB; b++) vb[b] = B[b][r];
#pragma unroll
    for (int a = 0; a < kTA; a++)
#pragma unroll
      for (int b = 0; b < kTB; b++) acc[a][b] = fma(va[a], vb[b], acc[a][b]);
  }
  // block reduction in a fixed order: warp trees, then the warps in order
  __shared__ double s[kThreads / 32][kTA * kTB];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int a = 0; a < kTA; a++)
#pragma unroll
    for (int b = 0; b < kTB; b++) {
      double v = acc[a][b];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) s[w][a * kTB + b] = v;
    }
  __syncthreads();
  if (threadIdx.x < kTA * kTB) {
    const int a = threadIdx.x / kTB, b = threadIdx.x % kTB;
    double v = 0.0;
    for (int q = 0; q < kThreads / 32; q++) v += s[q][threadIdx.x];
    if (ta + a < m && tb + b < p) part[((long)blockIdx.x * m + ta + a) * p + tb + b] = v;
  }
}

// 32 products and 32 chunk lanes per block: each lane sums every 32nd chunk,
// then the lanes in order
__global__ void __launch_bounds__(1024)
k_gram_sum(const double *__restrict__ part, int nchunk, int m, int p, double *__restrict__ C) {
  __shared__ double s[32][33];
  const int q = blockIdx.x * 32 + threadIdx.x;
  double v = 0.0;
  if (q < m * p)
    for (int c = threadIdx.y; c < nchunk; c += 32) v += part[(long)c * m * p + q];
  s[threadIdx.y][threadIdx.x] = v;
  __syncthreads();
  for (int o = 16; o > 0; o >>= 1) {
    if ((int)threadIdx.y < o) s[threadIdx.y][threadIdx.x] += s[threadIdx.y + o][threadIdx.x];
    __syncthreads();
  }
  if (threadIdx.y == 0 && q < m * p) C[q] = s[0][threadIdx.x];
}

// ---------------------------------------------------------------------------
// The same products in block fixed point.  A column's 128 rows of a chunk share
// a power of two taken from their largest entry, |x| 2^p < 2^58, split into
// two signed halves at 2^30; a product keeps hi*hi and the two cross terms
// (three 32 x 32 + 64 bit multiply-adds, 6 issue cycles against 64 for one
// FP64 fused multiply-add) and drops lo*lo, 2^-59 of the largest product.  The
// chunk's sums are exact, |sum| < 2^123, kept to 2^60, and meet in FP64.  At
// most 16 rows meet in one cross sum (< 2^62) before its upper bits move to hi.
//
// A chunk is off by at most 80 x 2^60: each row's half units of both entries
// (2^58), its lo*lo (2^58), half a unit for each of up to 32 slices.  An FP64
// sum is off by units of 2^-53 of sum |x y|, so the integers stand where that
// is at least 2^kQSum = 2^114 (then the error is below 40 x 2^-53 of it, where
// 128 FP64 additions allow 128), and a pair of columns whose large entries do
// not meet takes the FP64 sum.  sum |x y| is bounded from below by |sum x y|
// and, where that is small, by the sum over the entries' upper 8 bits (four rows
// an instruction); the two largest entries meeting suffice (128 x 128 = 2^14).
// 187488 rows, 48 x 16: 161 us on normal entries, 202 on rows that fall by
// e^-0.25, 411 on entries over 40 decades, where most pairs take the FP64 sum
// (the FP64 kernel 490-510 on each; without the test 150, with errors up to
// 2^-48 of sum |x y| on the last and of any size on columns that hardly meet).
// Chunks that hold an infinity, a NaN or numbers beyond 2^+-400 take FP64 sums.
//
// Tile: 64 x 16 columns, 4 x 4 products per thread, the rows split over ks
// threads.  The chunk comes by asynchronous copies into shared memory and is
// converted in place, a warp per column: with the loads in registers instead a
// block waited for memory ten times a stage (187488 rows, 48 x 16: 200 us).
// ---------------------------------------------------------------------------
constexpr int kQBits = 58, kQLow = 30;
constexpr int kQA = 64, kQB = 16;  // columns of a tile
constexpr int kQR = 128;           // rows of a chunk
constexpr int kQS = kQR + 2;       // column stride: odd in 16-byte units
constexpr int kQLim = 400;
constexpr int kQSum = 114;           // of the smallest sum of |products| (see above)
constexpr int kQTop = kQBits - 8;    // of an entry's upper 8 bits
constexpr unsigned kQTops = 1u << (kQSum - 2 * kQTop);  // kQSum in products of those
constexpr int kQBS = kQR / 4 + 1;    // words of a column's upper bits, odd
constexpr int kQZero = 1 << 20;      // the power of two of a column of zeros

__device__ __forceinline__ int2 qsplit(long long x) {
  const int lo = ((int)x << (32 - kQLow)) >> (32 - kQLow);
  return make_int2(lo, (int)((x - lo) >> kQLow));
}
// the upper 8 bits of an entry's modulus
__device__ __forceinline__ unsigned qtop(int2 x) { return min((unsigned)abs(x.y) >> (kQTop - kQLow), 255u); }
// 8 bytes global -> shared, zeros where !on
__device__ __forceinline__ void copy8(void *dst, const void *src, bool on) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(on ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

__global__ void __launch_bounds__(kThreads, 2)
k_gramq(const double *__restrict__ V, long ld, long r0, long r1, int ks, int a0, int m, int b0,
        int p, double *__restrict__ part) {
  extern __shared__ __align__(16) int2 sx[];
  __shared__ int sp[kQA + kQB];  // the columns' powers of two
  __shared__ unsigned st[(kQA + kQB) * kQBS];  // upper bits of rows l, l + 32, l + 64, l + 96
  // the chunk's pairs of columns that take the FP64 sum
  __shared__ unsigned short s_pair[kQA * kQB];
  __shared__ double s_dot[kQA * kQB];
  __shared__ int s_low;
  if (threadIdx.x == 0) s_low = 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ta = blockIdx.y * kQA, tb = blockIdx.z * kQB;
  const int mt = min(kQA, m - ta), pt = min(kQB, p - tb), nc = mt + pt;
  const int GA = (mt + 3) / 4, GB = (pt + 3) / 4, nq = GA * GB;
  // product tile and row slice; for the sums over the slices (q, sl = product)
  const int q = tid % nq, sl = tid / nq;
  const int ga = q % GA, gb = q / GA;
  auto col = [&](int c) { return V + (long)(c < mt ? a0 + ta + c : b0 + tb + c - mt) * ld; };
  int pa[4], pb[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    pa[i] = min(ga + i * GA, mt - 1) * kQS;
    pb[i] = (mt + min(gb + i * GB, pt - 1)) * kQS;
  }
  double out[4] = {0.0, 0.0, 0.0, 0.0};
  for (long lo = r0 + (long)blockIdx.x * kQR; lo < r1; lo += (long)gridDim.x * kQR) {
    const int nr = (int)min((long)kQR, r1 - lo);
    for (int c = warp; c < nc; c += kThreads / 32) {
      const double *x = col(c) + lo;
#pragma unroll
      for (int r = lane; r < kQR; r += 32) copy8(sx + c * kQS + r, x + min(r, nr - 1), r < nr);
    }
    copy_wait();  // a warp converts the columns that it copied
    __syncwarp();
    bool bad = false;
#pragma unroll 2
    for (int c = warp; c < nc; c += kThreads / 32) {
      double x[kQR / 32];
      unsigned t = 0;
#pragma unroll
      for (int u = 0; u < kQR / 32; u++) {
        x[u] = *reinterpret_cast<const double *>(sx + c * kQS + lane + 32 * u);
        t = max(t, sb::hiword(x[u]));
      }
      t = __reduce_max_sync(0xffffffffu, t);
      const int E = (int)(t >> 20) - 1023;
      bad |= t != 0 && (E > kQLim || E < -kQLim);
      const sb::QScale sc = sb::qscale(t, kQBits);
      unsigned tops = 0;
#pragma unroll
      for (int u = 0; u < kQR / 32; u++) {
        const int2 v = qsplit(sb::tofix(x[u], sc));
        sx[c * kQS + lane + 32 * u] = v;
        tops |= qtop(v) << (8 * u);
      }
      st[c * kQBS + lane] = tops;
      if (lane == 0) sp[c] = t ? sc.p : kQZero;
    }
    if (__syncthreads_or(bad)) {
      for (int i = 0; i < 4; i++) {
        const int a = ga + i * GA, b = gb + sl * GB;
        if (sl < 4 && a < mt && b < pt) {
          const double *x = col(a) + lo, *y = col(mt + b) + lo;
          double v = 0.0;
          for (int r = 0; r < nr; r++) v = fma(x[r], y[r], v);
          out[i] += v;
        }
      }
      __syncthreads();
      continue;
    }
    long long hi[4][4], cr[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) hi[i][j] = cr[i][j] = 0;
    if (sl < ks) {
      for (int r = 2 * sl; r < nr;) {
        const int end = min(nr, r + 16 * ks);
#pragma unroll 2
        for (; r < end; r += 2 * ks) {
          int4 a[4], b[4];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            a[i] = *reinterpret_cast<const int4 *>(sx + pa[i] + r);
            b[i] = *reinterpret_cast<const int4 *>(sx + pb[i] + r);
          }
#pragma unroll
          for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
              hi[i][j] += (long long)a[i].y * b[j].y;
              cr[i][j] += (long long)a[i].x * b[j].y;
              cr[i][j] += (long long)a[i].y * b[j].x;
              hi[i][j] += (long long)a[i].w * b[j].w;
              cr[i][j] += (long long)a[i].z * b[j].w;
              cr[i][j] += (long long)a[i].w * b[j].z;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) {
            hi[i][j] += cr[i][j] >> kQLow;
            cr[i][j] &= (1 << kQLow) - 1;
          }
      }
    }
    __syncthreads();
    // the slices' sums, in integers (rounded: a bias would add up over the chunks)
    long long *red = reinterpret_cast<long long *>(sx);
    if (sl < ks)
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
          red[((sl * 4 + i) * 4 + j) * nq + q] = hi[i][j] + (cr[i][j] >> (kQLow - 1));
    __syncthreads();
    int low[4] = {-1, -1, -1, -1};
    if (sl < 4) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        long long t = 0;
        for (int k = 0; k < ks; k++) t += red[((k * 4 + i) * 4 + sl) * nq + q];
        const bool in = ga + i * GA < mt && gb + sl * GB < pt;
        const int a = min(ga + i * GA, mt - 1), b = min(gb + sl * GB, pt - 1);
        const int pab = sp[a] + sp[mt + b];
        if (in && abs(t) < 1ll << (kQSum - 2 * kQLow) && pab < kQZero / 2) {
          unsigned d = 0;
#pragma unroll 8
          for (int l = 0; l < kQR / 4; l++)
            d = __dp4a(st[a * kQBS + l], st[(mt + b) * kQBS + l], d);
          if (d < kQTops) {
            low[i] = atomicAdd(&s_low, 1);
            s_pair[low[i]] = (unsigned short)(a | b << 8);
          }
        }
        if (low[i] < 0) out[i] += sb::fromfix(t, 2 * kQLow - pab);
      }
    }
    __syncthreads();
    const int nlow = s_low;
    if (nlow == 0) continue;
    // the FP64 sums, L lanes a pair
    const int L = nlow > kThreads / 8 ? 4 : nlow > kThreads / 16 ? 8 : nlow > kThreads / 32 ? 16 : 32;
    for (int k = tid / L; k < (nlow + 31) / 32 * 32; k += kThreads / L) {
      double v = 0.0;
      if (k < nlow) {
        const int a = s_pair[k] & 255, b = s_pair[k] >> 8;
        const double *x = col(a) + lo, *y = col(mt + b) + lo;
#pragma unroll 4
        for (int r = tid % L; r < nr; r += L) v = fma(x[r], y[r], v);
      }
      for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (k < nlow && tid % L == 0) s_dot[k] = v;
    }
    __syncthreads();
    if (tid == 0) s_low = 0;
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (low[i] >= 0) out[i] += s_dot[low[i]];
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int a = ga + i * GA, b = gb + sl * GB;
    if (sl < 4 && a < mt && b < pt)
      part[((long)blockIdx.x * m + ta + a) * p + tb + b] = out[i];
  }
}

// W[r, b0 + b] += alpha * sum_a V[r, a0 + a] C[a][b] over rows [r0, r1)
__global__ void __launch_bounds__(kThreads)
k_update(double *__restrict__ V, long ld, long r0, long r1, int a0, int m, int b0, int p,
         const double *__restrict__ C, double alpha) {
  const long r = r0 + (long)blockIdx.x * kThreads + threadIdx.x;
  if (r >= r1) return;
  for (int g = 0; g < p; g += 8) {
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int nb = min(8, p - g);
    for (int a = 0; a < m; a++) {
      const double v = V[(long)(a0 + a) * ld + r];
      const double *c = C + (long)a * p + g;
#pragma unroll
      for (int b = 0; b < 8; b++)
        if (b < nb) acc[b] = fma(v, c[b], acc[b]);
    }
#pragma unroll
    for (int b = 0; b < 8; b++)
      if (b < nb) {
        double *w = V + (long)(b0 + g + b) * ld + r;
        *w = fma(alpha, acc[b], *w);
      }
  }
}

// a b + c, one instruction: left to itself the compiler widens the row's halves
// once and multiplies 64 x 64 bits (187488 rows, 48 x 16: 150 us against 95)
__device__ __forceinline__ long long qmad(int a, int b, long long c) {
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(c) : "r"(a), "r"(b));
  return c;
}

// The same update in block fixed point, NB columns of W per pass.  The
// coefficients come as 58-bit integers C'[a][b] 2^pc[b] in halves, where
// C' = C 2^-da[a] has entries of about one in every row, and the row's scaled
// entries V 2^da share a power of two, so that neither badly scaled columns
// nor the range over the rows (wavenumbers) lose digits.  Three multiply-adds
// a product as above; at most 64 products meet in one sum, off by at most
// 33 x 2^60 (a quarter for each product's roundings and for its lo*lo, one at
// the end).  As in k_gramq it stands where sum |v C'| is at least 2^kQSum by
// the upper bits of both, or W is so large, 2^(kQSum + 2), that its own rounding
// exceeds that; a column that picks small entries out of a row takes the FP64
// sum.  So do rows with an infinity, a NaN or numbers beyond 2^+-400.  The rows
// come by asynchronous copies, a thread its own, before the scale is taken.
// 187488 rows, 48 x 16: 121 us on normal entries and on rows that fall by
// e^-0.25, 281 on entries over 40 decades (FP64 263-277; without the test 108).
// MANY: for m > 64 the parts' sums are kept, so that W is rounded once.
template <int NB, bool MANY>
__global__ void __launch_bounds__(kUThreads, MANY ? 2 : 3)
k_updateq(double *__restrict__ V, long ld, long r0, long r1, int a0, int m, int b0, int p,
          const double *__restrict__ C, const int2 *__restrict__ CQ, const int *__restrict__ da,
          const int *__restrict__ pc, double alpha) {
  extern __shared__ __align__(16) int2 sx[];
  const int mx = min((m + 3) / 4 * 4, 64);
  int2 *sc = sx;                                 // coefficients [mx][NB]
  double *sv = (double *)(sx + mx * NB);         // rows of V [mx][kUThreads]
  unsigned *st = (unsigned *)(sv + mx * kUThreads);  // upper bits of four rows of them [mx/4][NB]
  int *sd = (int *)(st + mx / 4 * NB);           // exponents [mx]
  const int pp = (p + NB - 1) / NB * NB;
  const long r = r0 + (long)blockIdx.x * kUThreads + threadIdx.x;
  const int g = blockIdx.y * NB, nb = min(NB, p - g);
  const bool on = r < r1;
  double *w = V + (long)(b0 + g) * ld + (on ? r : r1 - 1);
  double sum[MANY ? NB : 1];  // over m > 64 columns of V: W is rounded once
#pragma unroll
  for (int b = 0; b < (MANY ? NB : 1); b++) sum[b] = 0.0;
  auto add = [&](int b, double x) {
    if constexpr (MANY) sum[b] += x;
    else w[(long)b * ld] = fma(alpha, x, w[(long)b * ld]);
  };
  for (int c0 = 0; c0 < m; c0 += 64) {
    const int mc = min(64, m - c0), m4 = (mc + 3) / 4 * 4;  // zeros from mc on
    const double *v = V + (long)(a0 + c0) * ld + (on ? r : r1 - 1);
    __syncthreads();
#pragma unroll 8
    for (int a = 0; a < m4; a++)
      copy8(sv + a * kUThreads + threadIdx.x, v + (long)min(a, mc - 1) * ld, on && a < mc);
    for (int k = threadIdx.x; k < m4 * NB; k += kUThreads) {
      const int a = k / NB;
      sc[k] = a < mc ? CQ[(long)(c0 + a) * pp + g + k % NB] : make_int2(0, 0);
    }
    for (int k = threadIdx.x; k < m4; k += kUThreads) sd[k] = k < mc ? da[c0 + k] : 0;
    copy_wait();
    __syncthreads();
    for (int k = threadIdx.x; k < m4 / 4 * NB; k += kUThreads) {
      const int2 *c = sc + k / NB * 4 * NB + k % NB;
      st[k] = qtop(c[0]) | qtop(c[NB]) << 8 | qtop(c[2 * NB]) << 16 | qtop(c[3 * NB]) << 24;
    }
    __syncthreads();
    const double *mv = sv + threadIdx.x;
    int top = -100000, raw = 0;
#pragma unroll 8
    for (int a = 0; a < mc; a++) {
      const int e = (int)(sb::hiword(mv[a * kUThreads]) >> 20);
      raw = max(raw, e);
      if (e) top = max(top, e + sd[a]);
    }
    bool plain = raw == 0x7ff || top > 1023 + kQLim || top < 1023 - kQLim;
    if (p > 1) {
      // a row with few entries near its largest would fall to FP64 in most
      // columns after the integers: a warp of those takes it at once
      int near = 0;
#pragma unroll 8
      for (int a = 0; a < mc; a++)
        near += (int)(sb::hiword(mv[a * kUThreads]) >> 20) + sd[a] > top - 8;
      plain |= __popc(__ballot_sync(0xffffffffu, on && 4 * near < mc)) > 16;
    }
    if (!on) continue;
    auto dot = [&](int b) {
      double acc = 0.0;
#pragma unroll 2
      for (int a = 0; a < mc; a++) acc = fma(mv[a * kUThreads], C[(long)(c0 + a) * p + g + b], acc);
      return acc;
    };
    if (plain) {
#pragma unroll
      for (int b = 0; b < NB; b += 4) {
        if (b >= nb) break;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        const double *c = C + (long)c0 * p + g + b;
#pragma unroll 4
        for (int a = 0; a < mc; a++) {
          const double x = mv[a * kUThreads];
#pragma unroll
          for (int q = 0; q < 4; q++) acc[q] = fma(x, c[(long)a * p + min(q, nb - b - 1)], acc[q]);
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (b + q < nb) add(b + q, acc[q]);
      }
      continue;
    }
    const int pr = kQBits - (top - 1022);
    long long hi[NB], cr[NB];
    unsigned tops[NB];
#pragma unroll
    for (int b = 0; b < NB; b++) {
      hi[b] = cr[b] = 0;
      tops[b] = 0;
    }
    for (int a = 0; a < m4;) {
      const int end = min(m4, a + 16);
#pragma unroll 1
      for (; a < end; a += 4) {
        unsigned xt = 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
          sb::QScale s;
          s.p = pr + sd[a + u];
          const int2 x = qsplit(sb::tofix(mv[(a + u) * kUThreads], s));
          xt |= qtop(x) << (8 * u);
#pragma unroll
          for (int b = 0; b < NB; b += 2) {
            const int4 c = *reinterpret_cast<const int4 *>(sc + (a + u) * NB + b);
            hi[b] = qmad(x.y, c.y, hi[b]);
            cr[b] = qmad(x.x, c.y, cr[b]);
            cr[b] = qmad(x.y, c.x, cr[b]);
            hi[b + 1] = qmad(x.y, c.w, hi[b + 1]);
            cr[b + 1] = qmad(x.x, c.w, cr[b + 1]);
            cr[b + 1] = qmad(x.y, c.z, cr[b + 1]);
          }
        }
#pragma unroll
        for (int b = 0; b < NB; b += 4) {
          const uint4 c = *reinterpret_cast<const uint4 *>(st + a / 4 * NB + b);
          tops[b] = __dp4a(xt, c.x, tops[b]);
          tops[b + 1] = __dp4a(xt, c.y, tops[b + 1]);
          tops[b + 2] = __dp4a(xt, c.z, tops[b + 2]);
          tops[b + 3] = __dp4a(xt, c.w, tops[b + 3]);
        }
      }
#pragma unroll
      for (int b = 0; b < NB; b++) {
        hi[b] += cr[b] >> kQLow;
        cr[b] &= (1 << kQLow) - 1;
      }
    }
    // hi < 2^(56 + bits of mc): the sum as one integer, 2^(60 - up)
    const int up = mc > 32 ? 0 : mc > 16 ? 1 : mc > 8 ? 2 : 3;
    // exponent field of a W that makes up for any error of the sum
    const int we = 1023 + kQSum + 2 + sb::qexp(alpha) + 1;
#pragma unroll
    for (int b = 0; b < NB; b++)
      if (b < nb) {
        const int pb = pr + pc[g + b];
        if (tops[b] < kQTops && (int)(sb::hiword(w[(long)b * ld]) >> 20) < we - pb) {
          add(b, dot(b));
        } else {
          const long long t = (hi[b] << up) + ((cr[b] + (1ll << (kQLow - 1 - up))) >> (kQLow - up));
          add(b, sb::fromfix(t, 2 * kQLow - up - pb));
        }
      }
  }
  if constexpr (MANY)
    if (on)
#pragma unroll
      for (int b = 0; b < NB; b++)
        if (b < nb) w[(long)b * ld] = fma(alpha, sum[b], w[(long)b * ld]);
}

// the coefficients' integers and exponents for k_updateq; false where a
// number is not finite or too far from one
bool fix_coefs(const double *C, int m, int p, int pp, int2 *q, int *da, int *pc) {
  int *top = pc;  // of the columns, then their powers of two
  for (int b = 0; b < p; b++) top[b] = -100000;
  for (int a = 0; a < m; a++) {
    int e = 0;
    for (int b = 0; b < p; b++) e = std::max(e, (int)(sb::hiword(C[(long)a * p + b]) >> 20));
    if (e && std::abs(e - 1023) > kQLim) return false;
    da[a] = e ? e - 1023 : -20000;  // a row of zeros weighs nothing
    for (int b = 0; b < p; b++) {
      const int x = (int)(sb::hiword(C[(long)a * p + b]) >> 20);
      if (x) top[b] = std::max(top[b], x - da[a]);
    }
  }
  for (int b = 0; b < p; b++) {
    if (top[b] < 0) top[b] = 1023;
    if (top[b] < 1023 - kQLim) return false;
    pc[b] = kQBits - (top[b] - 1022);
  }
  for (int a = 0; a < m; a++)
    for (int b = 0; b < pp; b++) {
      sb::QScale s{};
      if (b < p) s.p = pc[b] - da[a];
      const long long v = b < p && da[a] != -20000 ? sb::tofix(C[(long)a * p + b], s) : 0;
      const long long lo = ((v & ((1ll << kQLow) - 1)) ^ (1ll << (kQLow - 1))) - (1ll << (kQLow - 1));
      q[(long)a * pp + b] = make_int2((int)lo, (int)((v - lo) >> kQLow));
    }
  return true;
}

// W[r, b0 + b] = sum_a W[r, b0 + a] M[a][b] (in place, p <= 64 columns)
__global__ void __launch_bounds__(kThreads)
k_transform(double *__restrict__ V, long ld, long r0, long r1, int b0, int p,
            const double *__restrict__ M) {
  const long r = r0 + (long)blockIdx.x * kThreads + threadIdx.x;
  if (r >= r1) return;
  double x[64];
  for (int a = 0; a < p; a++) x[a] = V[(long)(b0 + a) * ld + r];
  for (int b = 0; b < p; b++) {
    double acc = 0.0;
    for (int a = 0; a < p; a++) acc = fma(x[a], M[(long)a * p + b], acc);
    V[(long)(b0 + b) * ld + r] = acc;
  }
}

struct Srcs {
  int n;
  int col[kMaxSrc];
  double coef[kMaxSrc];
};

// V[r, dst] = sum_k coef_k V[r, src_k]
__global__ void k_combine(double *__restrict__ V, long ld, long r0, long r1, int dst, Srcs s) {
  const long r = r0 + (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= r1) return;
  double v = 0.0;
  for (int k = 0; k < s.n; k++) v = fma(s.coef[k], V[(long)s.col[k] * ld + r], v);
  V[(long)dst * ld + r] = v;
}

// the representable finite-difference step of matvec_dns_disk3d (iuse_hej):
// V[dst] = x0 + ((x0 + e d) - x0), each operation rounded on its own
__global__ void k_perturb(double *__restrict__ V, long ld, long r0, long r1, int dst, int x0c,
                          int dc, double e) {
  const long r = r0 + (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= r1) return;
  const double x0 = V[(long)x0c * ld + r], d = V[(long)dc * ld + r];
  const double h = __dsub_rn(__dadd_rn(x0, __dmul_rn(e, d)), x0);
  V[(long)dst * ld + r] = __dadd_rn(x0, h);
}

// finite-difference products: order 1 (g0 - g1) / eps, order 2
// (g0 - g1) / (2 eps), order 4 (8 (g0 - g1) - (g2 - g3)) / (12 eps)
__global__ void k_fd(double *__restrict__ V, long ld, long r0, long r1, int dst, int order,
                     Srcs s, double eps) {
  const long r = r0 + (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= r1) return;
  const double a = V[(long)s.col[0] * ld + r], b = V[(long)s.col[1] * ld + r];
  double v;
  if (order == 1) {
    v = __ddiv_rn(__dsub_rn(a, b), eps);
  } else if (order == 2) {
    v = __ddiv_rn(__dsub_rn(a, b), __dmul_rn(2.0, eps));
  } else {
    const double c = V[(long)s.col[2] * ld + r], d = V[(long)s.col[3] * ld + r];
    v = __ddiv_rn(__dsub_rn(__dmul_rn(8.0, __dsub_rn(a, b)), __dsub_rn(c, d)),
                  __dmul_rn(12.0, eps));
  }
  V[(long)dst * ld + r] = v;
}

// ---------------------------------------------------------------------------
// state <-> unknown vector.  Complex entry sc of a y plane <-> (kz index k,
// kx index i): row k = 0 without i = 0, rows 1..nz all i, rows nz+1..mz-1
// without i = 0 (the conjugates of rows mz-k); x = [u00/su | w00/su | per
// plane j and entry sc: vor.re/sg, phi.re/sp, vor.im/sg, phi.im/sp].
// ---------------------------------------------------------------------------
__device__ __forceinline__ void entry_of(const Grid &g, int sc, int *k, int *i) {
  const int n0 = g.nkx - 1, n1 = g.nz * g.nkx;
  if (sc < n0) {
    *k = 0;
    *i = sc + 1;
  } else if (sc < n0 + n1) {
    const int s = sc - n0;
    *k = 1 + s / g.nkx;
    *i = s % g.nkx;
  } else {
    const int s = sc - n0 - n1;
    *k = g.nz + 1 + s / (g.nkx - 1);
    *i = 1 + s % (g.nkx - 1);
  }
}
__device__ __forceinline__ int index_of(const Grid &g, int k, int i) {
  if (k == 0) return i - 1;
  if (k <= g.nz) return (g.nkx - 1) + (k - 1) * g.nkx + i;
  return (g.nkx - 1) + g.nz * g.nkx + (k - g.nz - 1) * (g.nkx - 1) + (i - 1);
}

template <typename R>
__global__ void k_pack(Grid g, const R *__restrict__ vor, const R *__restrict__ phi,
                       const R *__restrict__ mu, double *__restrict__ x, double su, double sg,
                       double sp, double sx, double sz) {
  const int nselc = g.mz * g.nkx - 1 - g.nz;  // complex entries per plane
  const long nb = (long)g.my * nselc;
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < g.my) {
    x[t] = (double)mu[2 * t] / su;
    x[g.my + t] = (double)mu[2 * t + 1] / su;
  }
  if (t >= nb) return;
  const int j = (int)(t / nselc), sc = (int)(t - (long)j * nselc);
  int k, i;
  entry_of(g, sc, &k, &i);
  const long o = 2 * (((long)j * g.mz + k) * g.nkx + i);
  double vr = (double)vor[o], vi = (double)vor[o + 1];
  double pr = (double)phi[o], pi = (double)phi[o + 1];
  if (sx != 0.0 || sz != 0.0) {
    // phase_shift_fou: the mode times exp(-i kx sx) exp(-i kz sz)
    const double kz = g.gam * (double)(k <= g.nz ? k : k - g.mz);
    double s1, c1, s2, c2;
    sincos(g.alp * (double)i * sx, &s1, &c1);
    sincos(kz * sz, &s2, &c2);
    const double fr = c1 * c2 - s1 * s2, fi = -(s1 * c2 + c1 * s2);
    const double a = vr * fr - vi * fi, b = vr * fi + vi * fr;
    const double c = pr * fr - pi * fi, d = pr * fi + pi * fr;
    vr = a;
    vi = b;
    pr = c;
    pi = d;
  }
  double *o4 = x + 2 * (long)g.my + 4 * t;
  o4[0] = vr / sg;
  o4[1] = pr / sp;
  o4[2] = vi / sg;
  o4[3] = pi / sp;
}

template <typename R>
__global__ void k_unpack(Grid g, const double *__restrict__ x, R *__restrict__ vor,
                         R *__restrict__ phi, R *__restrict__ mu, double su, double sg,
                         double sp) {
  const int nselc = g.mz * g.nkx - 1 - g.nz;
  const long n = (long)g.my * g.mz * g.nkx;
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < g.my) {
    mu[2 * t] = (R)(x[t] * su);
    mu[2 * t + 1] = (R)(x[g.my + t] * su);
  }
  if (t >= n) return;
  const int i = (int)(t % g.nkx);
  const int k = (int)((t / g.nkx) % g.mz);
  const int j = (int)(t / ((long)g.nkx * g.mz));
  double vr = 0.0, vi = 0.0, pr = 0.0, pi = 0.0;
  if (i != 0 || k != 0) {
    const bool cj = (i == 0 && k > g.nz);  // set_conj: the conjugate of row mz-k
    const int sc = index_of(g, cj ? g.mz - k : k, i);
    const double *s4 = x + 2 * (long)g.my + 4 * ((long)j * nselc + sc);
    vr = s4[0] * sg;
    pr = s4[1] * sp;
    vi = s4[2] * sg;
    pi = s4[3] * sp;
    if (cj) {
      vi = -vi;
      pi = -pi;
    }
  }
  vor[2 * t] = (R)vr;
  vor[2 * t + 1] = (R)vi;
  phi[2 * t] = (R)pr;
  phi[2 * t + 1] = (R)pi;
}

// d/ds of the phase shift at s = 0 on a packed vector: every mode times
// -i kx (dir 0) or -i kz (dir 1); the mean profiles have no derivative
__global__ void k_tangent(Grid g, const double *__restrict__ x, double *__restrict__ out,
                          int dir) {
  const int nselc = g.mz * g.nkx - 1 - g.nz;
  const long nb = (long)g.my * nselc;
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 2L * g.my) out[t] = 0.0;
  if (t >= nb) return;
  const int sc = (int)(t % nselc);
  int k, i;
  entry_of(g, sc, &k, &i);
  const double kk = dir == 0 ? g.alp * (double)i : g.gam * (double)(k <= g.nz ? k : k - g.mz);
  const double *s4 = x + 2 * (long)g.my + 4 * t;
  double *o4 = out + 2 * (long)g.my + 4 * t;
  const double vr = s4[0], pr = s4[1], vi = s4[2], pi = s4[3];
  o4[0] = kk * vi;
  o4[1] = kk * pi;
  o4[2] = -kk * vr;
  o4[3] = -kk * pr;
}

long chunk_rows(long rows, long *nchunk) {
  long nc = (rows + 2047) / 2048;
  if (nc > 608) nc = 608;
  if (nc < 1) nc = 1;
  const long ch = (rows + nc - 1) / nc;
  *nchunk = (rows + ch - 1) / ch;
  return ch;
}

// the row split of k_gramq: slices of a chunk, blocks, shared memory
void gramq_plan(long rows, int m, int p, int *ks, int *nblk, size_t *smem) {
  const int mt = std::min(m, kQA), pt = std::min(p, kQB);
  const int nq = ((mt + 3) / 4) * ((pt + 3) / 4);
  // the fewest warp passes over a chunk's row pairs
  long best = 0;
  for (int k = 4; k <= 32 && k * nq <= kThreads; k++) {
    const long c = (long)((nq * k + 31) / 32) * ((kQR / 2 + k - 1) / k);
    if (!best || c < best) {
      best = c;
      *ks = k;
    }
  }
  const int tiles = ((m + kQA - 1) / kQA) * ((p + kQB - 1) / kQB);
  const long chunks = (rows + kQR - 1) / kQR, slots = std::max(1, 2 * 152 / tiles);
  // as many chunks to every block
  const long each = (chunks + slots - 1) / slots;
  *nblk = (int)((chunks + each - 1) / each);
  *smem = std::max(sizeof(int2) * (size_t)(mt + pt) * kQS, sizeof(long long) * 16 * nq * *ks);
}
constexpr int kGramSmem = (int)sizeof(int2) * (kQA + kQB) * kQS;
// shared memory of k_updateq for mx (a multiple of 4) columns at a time
size_t update_smem(int mx, int nb) {
  return (sizeof(int2) * nb + sizeof(double) * kUThreads + sizeof(int) * nb / 4 + sizeof(int)) * mx;
}
cudaError_t prepare_fixed() {
  constexpr auto A = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(k_gramq, A, kGramSmem);
#define SB_PREP(NB, MANY) \
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_updateq<NB, MANY>, A, (int)update_smem(64, NB))
  SB_PREP(4, false);
  SB_PREP(8, false);
  SB_PREP(16, false);
  SB_PREP(4, true);
  SB_PREP(8, true);
  SB_PREP(16, true);
#undef SB_PREP
  return e;
}
// The fixed-point forms from 16 coefficients on.  187488 rows, whole calls,
// FP64 against fixed point: products 48 x 16 492 -> 161 us, 32 x 1 182 -> 88,
// 16 x 2 120 -> 71, 4 x 4 the same (58); updates 263 -> 121, 110 -> 42,
// 64 -> 31, 30 -> 26.  Below, the conversions cost what the sums save.
bool fixed_ok(int m, int p) { return (long)m * p >= 16; }

}  // namespace

namespace sb {

long packed_length(const Grid &g) {
  const long nselc = (long)g.mz * g.nkx - 1 - g.nz;
  return 2L * g.my + 4L * g.my * nselc;
}

cudaError_t launch_pack(const Grid &g, const double *vor, const double *phi, const double *mu,
                        double *x, const double sca[3], double sx, double sz, cudaStream_t st) {
  const long nselc = (long)g.mz * g.nkx - 1 - g.nz;
  const long n = std::max((long)g.my * nselc, (long)g.my);
  const unsigned nb = (unsigned)((n + 255) / 256);
  if (g.prec)
    k_pack<float><<<nb, 256, 0, st>>>(g, (const float *)vor, (const float *)phi,
                                      (const float *)mu, x, sca[0], sca[1], sca[2], sx, sz);
  else
    k_pack<double><<<nb, 256, 0, st>>>(g, vor, phi, mu, x, sca[0], sca[1], sca[2], sx, sz);
  return cudaGetLastError();
}

cudaError_t launch_tangent(const Grid &g, const double *x, double *out, int dir,
                           cudaStream_t st) {
  const long nselc = (long)g.mz * g.nkx - 1 - g.nz;
  const long n = std::max((long)g.my * nselc, 2L * g.my);
  k_tangent<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, x, out, dir);
  return cudaGetLastError();
}

cudaError_t launch_unpack(const Grid &g, const double *x, double *vor, double *phi, double *mu,
                          const double sca[3], cudaStream_t st) {
  const long n = std::max((long)g.my * g.mz * g.nkx, (long)g.my);
  const unsigned nb = (unsigned)((n + 255) / 256);
  if (g.prec)
    k_unpack<float><<<nb, 256, 0, st>>>(g, x, (float *)vor, (float *)phi, (float *)mu, sca[0],
                                        sca[1], sca[2]);
  else
    k_unpack<double><<<nb, 256, 0, st>>>(g, x, vor, phi, mu, sca[0], sca[1], sca[2]);
  return cudaGetLastError();
}

}  // namespace sb

// ---------------------------------------------------------------------------
// the Krylov space object of the C-ABI
// ---------------------------------------------------------------------------
struct sb_kspace {
  long n = 0, ld = 0;
  int cols = 0;
  double *V = nullptr;     // cols columns of ld doubles (n used)
  double *part = nullptr;  // gram partial sums
  long part_cap = 0;
  double *small = nullptr;  // device copy of a coefficient matrix
  long small_cap = 0;
  double *hsmall = nullptr;  // pinned host staging of the same
  cudaStream_t st = nullptr;
  bool own_stream = false;
  int dev = 0;
};

namespace {

int check_rows(const sb_kspace *ks, long r0, long r1) {
  if (r0 < 0 || r1 > ks->n || r0 > r1) return kfail(1, "row range [%ld, %ld) outside [0, %ld)", r0, r1, ks->n);
  return 0;
}
int check_cols(const sb_kspace *ks, int c0, int m) {
  if (c0 < 0 || m < 0 || c0 + m > ks->cols)
    return kfail(1, "columns [%d, %d) outside [0, %d)", c0, c0 + m, ks->cols);
  return 0;
}
int ensure_small(sb_kspace *ks, long count) {
  if (count <= ks->small_cap) return 0;
  if (ks->small) cudaFree(ks->small);
  if (ks->hsmall) cudaFreeHost(ks->hsmall);
  ks->small = nullptr;
  ks->hsmall = nullptr;
  ks->small_cap = 0;
  KCK(cudaMalloc((void **)&ks->small, sizeof(double) * count));
  KCK(cudaMallocHost((void **)&ks->hsmall, sizeof(double) * count));
  ks->small_cap = count;
  return 0;
}

}  // namespace

extern "C" {

int sb_kspace_create(long n, int cols, void *stream, sb_kspace **out) {
  if (!out || n < 1 || cols < 1) return kfail(1, "sb_kspace_create: bad argument");
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return kfail(2, "no CUDA device");
  sb_kspace *ks = new sb_kspace;
  ks->n = n;
  ks->ld = (n + 31) / 32 * 32;  // 256-byte aligned columns
  ks->cols = cols;
  cudaGetDevice(&ks->dev);
  cudaError_t e = cudaMalloc((void **)&ks->V, sizeof(double) * (size_t)ks->ld * cols);
  if (e == cudaSuccess) e = cudaMemset(ks->V, 0, sizeof(double) * (size_t)ks->ld * cols);
  if (e == cudaSuccess) e = prepare_fixed();
  if (e == cudaSuccess && !stream) {
    e = cudaStreamCreateWithFlags(&ks->st, cudaStreamNonBlocking);
    ks->own_stream = true;
  } else {
    ks->st = (cudaStream_t)stream;
  }
  if (e != cudaSuccess) {
    sb_kspace_destroy(ks);
    return kfail(3, "sb_kspace_create: %s", cudaGetErrorString(e));
  }
  *out = ks;
  return 0;
}

int sb_kspace_destroy(sb_kspace *ks) {
  if (!ks) return 0;
  if (ks->st) cudaStreamSynchronize(ks->st);
  if (ks->V) cudaFree(ks->V);
  if (ks->part) cudaFree(ks->part);
  if (ks->small) cudaFree(ks->small);
  if (ks->hsmall) cudaFreeHost(ks->hsmall);
  if (ks->own_stream && ks->st) cudaStreamDestroy(ks->st);
  delete ks;
  return 0;
}

double *sb_kspace_col(sb_kspace *ks, int col) {
  if (!ks || col < 0 || col >= ks->cols) return nullptr;
  return ks->V + (size_t)col * ks->ld;
}

void *sb_kspace_stream(sb_kspace *ks) { return ks ? (void *)ks->st : nullptr; }

int sb_kspace_gram(sb_kspace *ks, long r0, long r1, int a0, int m, int b0, int p, double *C) {
  if (!ks || !C) return kfail(1, "null argument");
  int rc;
  if ((rc = check_rows(ks, r0, r1)) || (rc = check_cols(ks, a0, m)) || (rc = check_cols(ks, b0, p)))
    return rc;
  if (m == 0 || p == 0) return 0;
  const long rows = r1 - r0;
  const bool fixed = fixed_ok(m, p) && rows > 0;
  long nchunk, ch = 0;
  int slices = 0, qblk = 0;
  size_t smem = 0;
  if (fixed) {
    gramq_plan(rows, m, p, &slices, &qblk, &smem);
    nchunk = qblk;
  } else {
    ch = chunk_rows(rows > 0 ? rows : 1, &nchunk);
  }
  const long need = nchunk * (long)m * p;
  if (need > ks->part_cap) {
    if (ks->part) cudaFree(ks->part);
    ks->part = nullptr;
    ks->part_cap = 0;
    KCK(cudaMalloc((void **)&ks->part, sizeof(double) * need));
    ks->part_cap = need;
  }
  if ((rc = ensure_small(ks, (long)m * p))) return rc;
  const int ca = fixed ? kQA : kTA, cb = fixed ? kQB : kTB;
  const dim3 grid((unsigned)nchunk, (unsigned)((m + ca - 1) / ca), (unsigned)((p + cb - 1) / cb));
  if ((m + kTA - 1) / kTA > 65535 || (p + kTB - 1) / kTB > 65535)
    return kfail(1, "sb_kspace_gram: block too large");
  if (fixed)
    k_gramq<<<grid, kThreads, smem, ks->st>>>(ks->V, ks->ld, r0, r1, slices, a0, m, b0, p,
                                              ks->part);
  else
    k_gram<<<grid, kThreads, 0, ks->st>>>(ks->V, ks->ld, r0, r1, ch, a0, m, b0, p, ks->part);
  KCK(cudaGetLastError());
  k_gram_sum<<<(unsigned)((m * p + 31) / 32), dim3(32, 32), 0, ks->st>>>(ks->part, (int)nchunk, m,
                                                                         p, ks->small);
  KCK(cudaGetLastError());
  KCK(cudaMemcpyAsync(ks->hsmall, ks->small, sizeof(double) * m * p, cudaMemcpyDeviceToHost,
                      ks->st));
  KCK(cudaStreamSynchronize(ks->st));
  for (long q = 0; q < (long)m * p; q++) C[q] = ks->hsmall[q];
  return 0;
}

int sb_kspace_update(sb_kspace *ks, long r0, long r1, int a0, int m, int b0, int p,
                     const double *C, double alpha) {
  if (!ks || !C) return kfail(1, "null argument");
  int rc;
  if ((rc = check_rows(ks, r0, r1)) || (rc = check_cols(ks, a0, m)) || (rc = check_cols(ks, b0, p)))
    return rc;
  if (a0 < b0 + p && b0 < a0 + m) return kfail(1, "sb_kspace_update: overlapping column ranges");
  if (m == 0 || p == 0 || r1 == r0) return 0;
  const int nb = p > 8 ? 16 : p > 4 ? 8 : 4, pp = (p + nb - 1) / nb * nb;
  const bool fixed = fixed_ok(m, p) && pp / nb <= 65535;
  // the coefficients, and their integers (int2 [m][pp]), da [m] and pc [p]
  const long mp = (long)m * p, oq = (mp + 1) / 2 * 2, oe = oq + (long)m * pp;
  const long count = fixed ? oe + (m + p + 1) / 2 : mp;
  if ((rc = ensure_small(ks, count))) return rc;
  // the staging buffer may still feed an earlier update: wait for the stream
  KCK(cudaStreamSynchronize(ks->st));
  for (long q = 0; q < mp; q++) ks->hsmall[q] = C[q];
  int *he = (int *)(ks->hsmall + oe);
  const bool fix = fixed && fix_coefs(C, m, p, pp, (int2 *)(ks->hsmall + oq), he, he + m);
  KCK(cudaMemcpyAsync(ks->small, ks->hsmall, sizeof(double) * (fix ? count : mp),
                      cudaMemcpyHostToDevice, ks->st));
  if (fix) {
    const dim3 grid((unsigned)((r1 - r0 + kUThreads - 1) / kUThreads), (unsigned)(pp / nb));
    const int *e = (const int *)(ks->small + oe);
    const int2 *cq = (const int2 *)(ks->small + oq);
    const size_t smem = update_smem(std::min((m + 3) / 4 * 4, 64), nb);
#define SB_UPD(NB, MANY)                                                                       \
  k_updateq<NB, MANY><<<grid, kUThreads, smem, ks->st>>>(ks->V, ks->ld, r0, r1, a0, m, b0, p,    \
                                                         ks->small, cq, e, e + m, alpha)
#define SB_UPDM(NB) \
  if (m > 64) SB_UPD(NB, true); \
  else SB_UPD(NB, false)
    if (nb == 16) {
      SB_UPDM(16);
    } else if (nb == 8) {
      SB_UPDM(8);
    } else {
      SB_UPDM(4);
    }
#undef SB_UPDM
#undef SB_UPD
  } else {
    k_update<<<(unsigned)((r1 - r0 + kThreads - 1) / kThreads), kThreads, 0, ks->st>>>(
        ks->V, ks->ld, r0, r1, a0, m, b0, p, ks->small, alpha);
  }
  KCK(cudaGetLastError());
  return 0;
}

int sb_kspace_transform(sb_kspace *ks, long r0, long r1, int b0, int p, const double *M) {
  if (!ks || !M) return kfail(1, "null argument");
  int rc;
  if ((rc = check_rows(ks, r0, r1)) || (rc = check_cols(ks, b0, p))) return rc;
  if (p > 64) return kfail(1, "sb_kspace_transform: at most 64 columns");
  if (p == 0 || r1 == r0) return 0;
  if ((rc = ensure_small(ks, (long)p * p))) return rc;
  KCK(cudaStreamSynchronize(ks->st));
  for (long q = 0; q < (long)p * p; q++) ks->hsmall[q] = M[q];
  KCK(cudaMemcpyAsync(ks->small, ks->hsmall, sizeof(double) * p * p, cudaMemcpyHostToDevice,
                      ks->st));
  k_transform<<<(unsigned)((r1 - r0 + kThreads - 1) / kThreads), kThreads, 0, ks->st>>>(
      ks->V, ks->ld, r0, r1, b0, p, ks->small);
  KCK(cudaGetLastError());
  return 0;
}

int sb_kspace_combine(sb_kspace *ks, long r0, long r1, int dst, int nsrc, const int *src,
                      const double *coef) {
  if (!ks || (nsrc > 0 && (!src || !coef))) return kfail(1, "null argument");
  if (nsrc < 0 || nsrc > kMaxSrc) return kfail(1, "sb_kspace_combine: 0..%d sources", kMaxSrc);
  int rc;
  if ((rc = check_rows(ks, r0, r1)) || (rc = check_cols(ks, dst, 1))) return rc;
  Srcs s{};
  s.n = nsrc;
  for (int k = 0; k < nsrc; k++) {
    if ((rc = check_cols(ks, src[k], 1))) return rc;
    s.col[k] = src[k];
    s.coef[k] = coef[k];
  }
  if (r1 == r0) return 0;
  k_combine<<<(unsigned)((r1 - r0 + 255) / 256), 256, 0, ks->st>>>(ks->V, ks->ld, r0, r1, dst, s);
  KCK(cudaGetLastError());
  return 0;
}

int sb_kspace_perturb(sb_kspace *ks, long r0, long r1, int dst, int x0, int d, double e) {
  if (!ks) return kfail(1, "null argument");
  int rc;
  if ((rc = check_rows(ks, r0, r1)) || (rc = check_cols(ks, dst, 1)) || (rc = check_cols(ks, x0, 1)) ||
      (rc = check_cols(ks, d, 1)))
    return rc;
  if (r1 == r0) return 0;
  k_perturb<<<(unsigned)((r1 - r0 + 255) / 256), 256, 0, ks->st>>>(ks->V, ks->ld, r0, r1, dst, x0,
                                                                    d, e);
  KCK(cudaGetLastError());
  return 0;
}

int sb_kspace_fd(sb_kspace *ks, long r0, long r1, int dst, int order, const int *g, double eps) {
  if (!ks || !g) return kfail(1, "null argument");
  if (order != 1 && order != 2 && order != 4) return kfail(1, "order must be 1, 2 or 4");
  int rc;
  if ((rc = check_rows(ks, r0, r1)) || (rc = check_cols(ks, dst, 1))) return rc;
  Srcs s{};
  s.n = order == 4 ? 4 : 2;
  for (int k = 0; k < s.n; k++) {
    if ((rc = check_cols(ks, g[k], 1))) return rc;
    s.col[k] = g[k];
  }
  if (r1 == r0) return 0;
  k_fd<<<(unsigned)((r1 - r0 + 255) / 256), 256, 0, ks->st>>>(ks->V, ks->ld, r0, r1, dst, order,
                                                               s, eps);
  KCK(cudaGetLastError());
  return 0;
}

int sb_kspace_set(sb_kspace *ks, int col, long off, long len, const double *host) {
  if (!ks || (!host && len > 0)) return kfail(1, "null argument");
  int rc;
  if ((rc = check_cols(ks, col, 1)) || (rc = check_rows(ks, off, off + len))) return rc;
  if (len == 0) return 0;
  KCK(cudaMemcpyAsync(ks->V + (size_t)col * ks->ld + off, host, sizeof(double) * len,
                      cudaMemcpyHostToDevice, ks->st));
  KCK(cudaStreamSynchronize(ks->st));
  return 0;
}

int sb_kspace_get(sb_kspace *ks, int col, long off, long len, double *host) {
  if (!ks || (!host && len > 0)) return kfail(1, "null argument");
  int rc;
  if ((rc = check_cols(ks, col, 1)) || (rc = check_rows(ks, off, off + len))) return rc;
  if (len == 0) return 0;
  KCK(cudaMemcpyAsync(host, ks->V + (size_t)col * ks->ld + off, sizeof(double) * len,
                      cudaMemcpyDeviceToHost, ks->st));
  KCK(cudaStreamSynchronize(ks->st));
  return 0;
}

int sb_kspace_sync(sb_kspace *ks) {
  if (!ks) return kfail(1, "null argument");
  KCK(cudaStreamSynchronize(ks->st));
  return 0;
}

}  // extern "C"
