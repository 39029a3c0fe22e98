"""Images of several frequencies against single-frequency renders (needs a GPU).

A frequency's records do not depend on the other frequencies of the image: the geodesic and the fluid are shared, the
coefficients, the segment operator and the sums are per frequency.  The kernels of 1, 4 and 32 frequency slots are
different instantiations, so their FP32 arithmetic may round differently in the coefficients and the operator (a few
ulp each, 6e-8) and in the sums of about 10^3 samples: 1e-5 of the largest value bounds FP32 and mixed.  FP64 is
compiled without contraction and gives the same value: 1e-12.
"""
from __future__ import annotations

import numpy as np
import pytest

import phoenix_b200 as P
from tests.golden.cases import case_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-5), ("mixed", 1e-5), ("fp64", 1e-12)])
@pytest.mark.parametrize("n", [2, 4, 5, 32])
def test_each_frequency_as_alone(gpu_snapshots, precision, tol, n):
    snap = gpu_snapshots["small"]
    freqs = [86e9 * 4.0 ** (k / (n - 1)) for k in range(n)]
    kw = dict(case_params("edge"), img_width=13, img_height=9)
    res, _ = snap.render(P.make_params(**dict(kw, precision=precision, frequencies=freqs)))
    for k in {0, 1, n // 2, n - 1}:
        one, _ = snap.render(P.make_params(**dict(kw, precision=precision, frequencies=[freqs[k]])))
        for part in (slice(0, 4), slice(4, 5), slice(5, 6)):
            a, b = res[:, :, k, part], one[:, :, 0, part]
            assert np.abs(a - b).max() <= tol * np.abs(b).max(), (n, k, part)
