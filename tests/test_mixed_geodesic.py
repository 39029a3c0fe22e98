"""The mixed march's acceleration (CPU): geodesic_accel_1 is geodesic_accel_at with the roundings spelled out, and no further
from extended precision."""
from __future__ import annotations

import os
import subprocess

from tests.conftest import ROOT

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include "geodesic.cuh"
using namespace phx;
using L = long double;

int main() {
  srand(11);
  auto u = [] { return rand() / (double)RAND_MAX; };
  // mean square error of both forms, away from the axis, within 0.1 and within 1e-3 of it; largest difference
  double at[3] = {0, 0, 0}, one[3] = {0, 0, 0}, worst = 0;
  const int n = 150000;
  for (int t = 0; t < n; t++) {
    const int reg = t % 3;
    const double a = 0.9375, hs = 0.25, x1 = std::log(1.4) + u() * std::log(30.0);
    double x2 = reg == 0 ? 0.15 + u() * (kPi - 0.3) : reg == 1 ? 0.005 + 0.095 * u() : 1e-5 + 1e-3 * u();
    if (u() < 0.5) x2 = kPi - x2;
    const KerrPt<double> p = kerr_point(a, hs, x1, x2);
    double k[4] = {1, (2 * u() - 1) / p.r, (2 * u() - 1) / (p.r * p.tp), (2 * u() - 1) / (p.r * p.s)}, F[4] = {0, 0, 0, 0};
    normalize_null(cov_metric(p, a), k);
    if (!std::isfinite(k[0])) continue;
    // the same r, sin, cos for all three, the rest of the point in each one's arithmetic
    double d[4], dF[4], e[4];
    geodesic_accel_at<double, false>(a, p, k, F, d, dF);
    geodesic_accel_1(a, KsPt<double>{p.r, p.s, p.c, p.tp, p.tpp}, k, e);
    KerrPt<L> q;
    q.r = p.r, q.s = p.s, q.c = p.c, q.tp = p.tp, q.tpp = p.tpp, q.s2 = q.s * q.s;
    q.sig = q.r * q.r + (L)a * a * q.c * q.c;
    q.isig = 1 / q.sig;
    q.q = 2 * q.r * q.isig;
    Cov<L> D1, D2;
    cov_derivs<L>(q, a, &D1, &D2);
    const L ir = 1 / q.r, ip = q.isig / (q.tp * q.tp * q.s2);
    const Contra<L> g = {-(1 + q.q), 2 * q.isig, q.isig * ((q.r - 2) * q.r + (L)a * a) * ir * ir, a * q.isig * ir,
                         ip * q.s2, ip * q.tp * q.tp};
    L kl[4], P[4], Q[4], f[4], o[4], s1 = 0, s2 = 0;
    for (int i = 0; i < 4; i++) kl[i] = k[i];
    symv(D1, kl, P);
    symv(D2, kl, Q);
    for (int i = 0; i < 4; i++) s1 += P[i] * kl[i], s2 += Q[i] * kl[i], f[i] = kl[1] * P[i] + kl[2] * Q[i];
    f[1] -= s1 / 2;
    f[2] -= s2 / 2;
    raise(g, f, o);
    const L sc[4] = {1, q.r, q.r * q.tp, q.r * q.s};
    L big = 0;
    for (int i = 0; i < 4; i++) big = fmaxl(big, fabsl(o[i] * sc[i]));
    double ea = 0, eb = 0;
    for (int i = 0; i < 4; i++) {
      ea = std::fmax(ea, (double)fabsl((d[i] + o[i]) * sc[i] / big));
      eb = std::fmax(eb, (double)fabsl((e[i] + o[i]) * sc[i] / big));
      worst = std::fmax(worst, (double)fabsl((d[i] - e[i]) * sc[i] / big));
    }
    at[reg] += ea * ea;
    one[reg] += eb * eb;
  }
  for (int r = 0; r < 3; r++) std::printf("%.4e %.4e ", std::sqrt(at[r] / (n / 3)), std::sqrt(one[r] / (n / 3)));
  std::printf("%.3e\n", worst);
  return 0;
}
"""


def test_no_further_from_extended_precision(tmp_path):
    """About 10^2 operations of 1.1e-16 each bound the difference of the two by 5e-14 of the largest component (terms that
    cancel reach a few times it).  Fewer roundings (fused sums): the error of the mean may not be larger than that of
    geodesic_accel_at without contraction, beyond the 1% to which 5 x 10^4 points a region fix it."""
    src, exe = tmp_path / "a.cpp", tmp_path / "a"
    src.write_text(SRC)
    core = os.path.join(ROOT, "phoenix_b200", "csrc", "core")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + core, str(src), "-o", str(exe)])
    v = [float(x) for x in subprocess.check_output([str(exe)]).decode().split()]
    assert v[6] <= 5e-14, v
    for at, one in ((v[0], v[1]), (v[2], v[3]), (v[4], v[5])):
        assert one <= 1.01 * at, v


QUOT_SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstdint>
#include "kerr.cuh"
using namespace phx;

int main() {
  uint64_t s = 0x9E3779B97F4A7C15ull;
  auto u01 = [&]() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return (double)(s >> 11) / 9007199254740992.0; };
  int off = 0, far = 0, plain = 0;
  for (int i = 0; i < 4000000; i++) {
    // offsets in a block over its cell size
    const double dx = std::exp(-12 + 12 * u01()), a = (i % 16 ? u01() * 64 : 1e-6 * u01()) * dx;
    const double ib = geo_rcp<double, true>(dx), q = geo_quot<double, true>(a, dx, ib), e = a / dx;
    off += q != e;
    far += std::fabs(q - e) > std::nextafter(std::fabs(e), 1e308) - std::fabs(e);
    plain += a * ib != e;
  }
  // an exact multiple of the cell size stays one
  int whole = 0;
  for (int n = 0; n < 4096; n++) {
    const double dx = std::ldexp(1.0, -n % 40);
    whole += geo_quot<double, true>(n * dx, dx, geo_rcp<double, true>(dx)) != n;
  }
  std::printf("%d %d %d %d\n", off, far, whole, plain);
  return 0;
}
"""


def test_cell_weights_quotient(tmp_path):
    """The quotient from a reciprocal within an ulp is off by at most one ulp, and only where a/b lies next to the middle of
    two numbers: the remainder's correction errs by about 2^-53 ulp x 2^52, so one in some thousands."""
    src, exe = tmp_path / "q.cpp", tmp_path / "q"
    src.write_text(QUOT_SRC)
    core = os.path.join(ROOT, "phoenix_b200", "csrc", "core")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + core, str(src), "-o", str(exe)])
    off, far, whole, plain = map(int, subprocess.check_output([str(exe)]).decode().split())
    assert far == 0 and whole == 0 and off <= 4000 and plain > 400000, (off, far, whole, plain)
