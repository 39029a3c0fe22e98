"""The segment operator with and without pivoting (CPU): the same bits wherever the march leaves the pivoting out."""
from __future__ import annotations

import os
import subprocess

import pytest

from tests.conftest import ROOT

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "transfer.cuh"
using namespace phx;

template <class R>
int run() {
  srand(5);
  auto u = [] { return rand() / (double)RAND_MAX; };
  int bad = 0, n = 0;
  for (int t = 0; t < 200000; t++) {
    Coeffs<R> c{};
    const double chi = 6.2831853 * u();
    // the coefficients' sum from far below the limit up to exactly on it, one of them alone now and then
    double v[4] = {u(), u(), u(), u()};
    if (t % 5 < 4) for (int i = 0; i < 4; i++) if (i != t % 5) v[i] = 0;
    const double s = v[0] + v[1] + v[2] + v[3];
    const double top = t % 3 ? 0.5 * std::exp(-20 * u()) : 0.5;
    c.aQ = R(v[0] / s * top * (u() < 0.5 ? -1 : 1)), c.aV = R(v[1] / s * top), c.rQ = R(v[2] / s * top);
    c.rV = R(v[3] / s * top * (u() < 0.5 ? -1 : 1));
    c.aI = R(t % 7 ? top * u() * 3 : 0), c.jI = R(u()), c.jQ = R(u()), c.jV = R(u());
    const R h = R(1);
    if (!(h * (fabs_t(c.aQ) + fabs_t(c.aV) + fabs_t(c.rQ) + fabs_t(c.rV)) <= R(0.5))) continue;
    R K[4][4], j[4], E[4][4], S[4], F[4][4], T[4];
    build_K(c, R(std::cos(chi)), R(std::sin(chi)), K, j);
    segment_operator<R, true>(K, j, h, E, S);
    segment_operator<R, false>(K, j, h, F, T);
    bad += std::memcmp(E, F, sizeof E) != 0 || std::memcmp(S, T, sizeof S) != 0;
    n++;
  }
  return n > 100000 ? bad : -1;
}

int main() {
  std::printf("%d %d\n", run<float>(), run<double>());
  return 0;
}
"""


@pytest.mark.parametrize("contract", ["off", "fast"])
def test_same_bits_without_pivoting(tmp_path, contract):
    src, exe = tmp_path / "s.cpp", tmp_path / "s"
    src.write_text(SRC)
    core = os.path.join(ROOT, "phoenix_b200", "csrc", "core")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=" + contract, "-I" + core, str(src), "-o", str(exe)])
    assert subprocess.check_output([str(exe)]).split() == [b"0", b"0"]
