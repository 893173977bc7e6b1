"""The 64-bit fixed-point transforms (csrc/sb_fix.cuh, csrc/sb_bloch.cu) on the
host: transforms of every length and direction against an extended-precision
DFT, no worse than an FP64 transform of the same data; conversions; the phase
twists; the scaled products.  The header's device code compiles for the host."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HARNESS = r"""
#include <cstring>
#include <vector>
#include "sb_fix.cuh"
#include "sb_host.h"
using namespace sb;
template <int N, int S> static void run(const double *in, double *out) {
  typedef Plan<N> P;
  constexpr int R1 = P::R1, R2 = P::R2;
  const std::vector<int> t = sbh::fix_twiddles(N, S, false);
  const qw *tw = (const qw *)t.data();
  unsigned top = 0;
  for (int i = 0; i < 2 * N; i++) top = hiword(in[i]) > top ? hiword(in[i]) : top;
  const QScale s = qscale(top, P::bits);
  std::vector<q2> y(N);
  for (int n2 = 0; n2 < R2; n2++) {
    q2 v[R1];
    for (int n1 = 0; n1 < R1; n1++) {
      const int n = n2 + R2 * n1;
      v[n1] = mkq(tofix(in[2 * n], s), tofix(in[2 * n + 1], s));
    }
    Dft<R1, S>::run(v);
    for (int k = 0; k < R1; k++) y[k * R2 + n2] = qmul<false>(v[k], tw[n2 * k]);
  }
  for (int k1 = 0; k1 < R1; k1++) {
    Dft<R2, S>::run(&y[k1 * R2]);
    for (int k2 = 0; k2 < R2; k2++) {
      const int k = k1 + R1 * k2, e = P::shift - s.p;
      out[2 * k] = fromfix(y[k1 * R2 + k2].x, e);
      out[2 * k + 1] = fromfix(y[k1 * R2 + k2].y, e);
    }
  }
}
extern "C" {
int fix_fft(int N, int S, const double *in, double *out) {
#define C(n) case n: if (S < 0) run<n, -1>(in, out); else run<n, 1>(in, out); return 0;
  switch (N) { C(32) C(48) C(64) C(80) C(96) C(128) C(160) C(192) C(256) C(320) C(384) }
  return 1;
}
double fix_round(double x, double big, int bits) {
  const QScale s = qscale(hiword(x) > hiword(big) ? hiword(x) : hiword(big), bits);
  return fromfix(tofix(x, s), -s.p);
}
float fix_roundf(float x, float big, int bits) {
  const QScale s = qscale(hiword(x) > hiword(big) ? hiword(x) : hiword(big), bits);
  return fromfixf(tofix(x, s), -s.p);
}
int fix_flags(double x) { const QScale s = qscale(hiword(x), 57); return s.bad + 2 * (s.p == kZeroScale); }
double fix_out(long long v, int t) { return fromfix(v, t); }
void fix_turn(long long X, int j, int N, int *o) {
  static const std::vector<int> t = sbh::fix_twiddles(1024, -1, false);
  const qw w = qturn(X, j, N, (const qw *)t.data());
  memcpy(o, &w, 16);
}
void fix_scaled(long long x, long long y, double c, int s0, long long *o) {
  const q2 z = qscaled(mkq(x, y), c, s0);
  o[0] = z.x; o[1] = z.y;
  o[2] = qlen(mkq(x, y)); o[3] = qexp(c);
}
}
"""
LENGTHS = (32, 48, 64, 80, 96, 128, 160, 192, 256, 320, 384)
CSRC = os.path.join(ROOT, "shear_nnf_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("fix")
    src, so = d / "fix.cpp", d / "fix.so"
    src.write_text(HARNESS)
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-Wno-unknown-pragmas", "-fsanitize=undefined",
                           "-fno-sanitize-recover=signed-integer-overflow", "-shared", "-fPIC", "-I",
                           CSRC, "-o", str(so), str(src), os.path.join(CSRC, "sb_host.cpp")])
    L = ctypes.CDLL(str(so))
    dp = np.ctypeslib.ndpointer(np.float64)
    L.fix_fft.argtypes = [ctypes.c_int, ctypes.c_int, dp, dp]
    L.fix_round.argtypes = [ctypes.c_double, ctypes.c_double, ctypes.c_int]
    L.fix_round.restype = ctypes.c_double
    L.fix_roundf.argtypes = [ctypes.c_float, ctypes.c_float, ctypes.c_int]
    L.fix_roundf.restype = ctypes.c_float
    L.fix_flags.argtypes = [ctypes.c_double]
    L.fix_out.argtypes = [ctypes.c_longlong, ctypes.c_int]
    L.fix_out.restype = ctypes.c_double
    L.fix_turn.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int,
                           np.ctypeslib.ndpointer(np.int32)]
    L.fix_scaled.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_double, ctypes.c_int,
                             np.ctypeslib.ndpointer(np.int64)]
    return L


def _dft(n, sign, x):
    k = np.arange(n)
    ang = 2 * np.arccos(np.longdouble(-1)) * sign * (np.outer(k, k) % n).astype(np.longdouble) / n
    c, s = np.cos(ang), np.sin(ang)
    xr, xi = x.real.astype(np.longdouble), x.imag.astype(np.longdouble)
    return c @ xr - s @ xi, s @ xr + c @ xi


def _inputs(n, rng):
    """White rows (a line in y), the largest coherent inputs (the overflow
    bound), one wave, entries of twelve orders of magnitude."""
    w = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    one = np.zeros(n, complex)
    one[5] = 0.7 - 0.3j
    top = 1 - 2.0 ** -53
    sg = np.sign(rng.standard_normal((2, n)))
    return {"white": w, "one": one, "const": np.full(n, top * (1 + 1j)),
            "signs": top * (sg[0] + 1j * sg[1]), "wide": w * 10.0 ** rng.uniform(-12, 0, n)}


@pytest.mark.parametrize("n", LENGTHS)
def test_transforms_no_worse_than_fp64(lib, n):
    """Error bound: 2^-53 relative in the 2-norm, an FP64 transform's unit (its
    own error is about twice that); overflow would show as an error of order
    one, or stop the sanitized build."""
    rng = np.random.default_rng(n)
    for sign in (-1, 1):
        for kind, x in _inputs(n, rng).items():
            out = np.zeros(2 * n)
            assert lib.fix_fft(n, sign, np.ascontiguousarray(x).view(np.float64), out) == 0
            r, i = _dft(n, sign, x)
            z = out.view(np.complex128)
            err = np.sqrt(np.sum((z.real - r) ** 2 + (z.imag - i) ** 2) / np.sum(r * r + i * i))
            assert err < 2.0 ** -53 * (1.5 if kind == "wide" else 1.0), (kind, sign, float(err))


def test_conversions(lib):
    """To the nearest multiple of 2^-bits of the block's largest value and
    back; zeros, signs, tiny and non-finite blocks."""
    rng = np.random.default_rng(0)
    for _ in range(4000):
        big = float(np.ldexp(rng.uniform(0.5, 1), int(rng.integers(-300, 300))))
        x = float(big * rng.uniform(-1, 1) * 10.0 ** -rng.integers(0, 22))
        assert abs(lib.fix_round(x, big, 57) - x) <= 2.0 ** -57 * 2 * big + 2.0 ** -53 * abs(x)
        xf, bf = np.float32(np.clip(x, -1e37, 1e37)), np.float32(min(big, 1e37))
        if bf > 1e-37:
            got = lib.fix_roundf(xf, bf, 57)
            assert abs(float(got) - float(xf)) <= 2.0 ** -57 * 2 * float(bf) + 1e-38
    for x in (0.0, -0.0, 1.0, -1.0, 1.5e308, 2.0 ** -900):
        assert lib.fix_round(x, 0.0, 57) == x
    assert lib.fix_flags(float("nan")) == 1 and lib.fix_flags(float("inf")) == 1
    assert lib.fix_flags(0.0) == 2 and lib.fix_flags(1e-300) == 2 and lib.fix_flags(1e-280) == 0
    # below the range: no size
    assert abs(lib.fix_out(-(1 << 60), -1200)) < 2.0 ** -900
    assert lib.fix_out((1 << 54) - 1, 0) == float((1 << 54) - 1)
    assert lib.fix_out(-(2 ** 63 - 1), 0) == -float(2 ** 63)


@pytest.mark.parametrize("n", LENGTHS)
def test_twists(lib, n):
    """exp(-2 pi i X j/(n 2^64)) to 2^-60, for phases of both signs and the
    half turn."""
    rng = np.random.default_rng(n)
    two_pi = 2 * np.arccos(np.longdouble(-1))
    o = np.zeros(4, np.int32)
    for X in [0, 1, -1, 2 ** 63 - 1, -2 ** 63] + [int(v) for v in rng.integers(-2 ** 63, 2 ** 63, 12)]:
        for j in (0, 1, n // 2, n - 1, int(rng.integers(0, n))):
            lib.fix_turn(X, j, n, o)
            q, r = divmod(X * j, n)  # exact turns at 2^64, less whole ones
            t = (np.longdouble(q % 2 ** 64) + np.longdouble(r) / n) / np.longdouble(2) ** 64
            w = [np.longdouble(int(o[k])) / 2 ** 30 + np.longdouble(int(o[k + 1])) / np.longdouble(2) ** 62
                 for k in (0, 2)]
            assert abs(w[0] - np.cos(two_pi * t)) < 2.0 ** -60 and abs(w[1] + np.sin(two_pi * t)) < 2.0 ** -60


def test_scaled_products(lib):
    """x c 2^s0 within two units and the last bit of c, for factors over the
    whole range; a zero factor gives nothing."""
    rng = np.random.default_rng(1)
    o = np.zeros(4, np.int64)
    for _ in range(3000):
        x, y = (int(v) >> int(rng.integers(0, 60)) for v in rng.integers(-2 ** 61, 2 ** 61, 2))
        c = float(rng.standard_normal() * 10.0 ** rng.integers(-12, 12))
        lib.fix_scaled(x, y, c, 0, o)
        s0 = 57 - int(o[2]) - int(o[3]) - 1 - int(rng.integers(0, 30))
        lib.fix_scaled(x, y, c, s0, o)
        for v, z in ((x, int(o[0])), (y, int(o[1]))):
            exact = np.longdouble(v) * np.longdouble(c) * np.longdouble(2) ** s0
            assert abs(np.longdouble(z) - exact) <= 2.0 + 2.0 ** -52 * abs(exact) and abs(z) < 2 ** 57 + 2
    lib.fix_scaled(1 << 60, 1 << 60, 0.0, 0, o)
    assert o[0] == 0 and o[1] == 0
