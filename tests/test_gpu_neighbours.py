"""A ray does not depend on the rays beside it (needs a GPU).

The plasma stage takes the segment operator with or without pivoting by what any lane of the warp needs.  Images of thick
plasma, whose samples lie on both sides of that limit, in several job orders and refill policies: bit for bit the same."""
from __future__ import annotations

import numpy as np
import pytest

import phoenix_b200 as P
from tests.golden.cases import CASES, case_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,nfreqs,tau_fp64", [("fp32", 1, 0.0), ("fp32", 3, 0.0), ("fp32", 7, 0.0), ("mixed", 1, 1e9),
                                                       ("mixed", 3, 1e9), ("mixed", 7, 1e9)])
@pytest.mark.parametrize("pipeline", [False, True])
def test_thick_plasma_in_any_order(gpu_snapshots, precision, nfreqs, tau_fp64, pipeline):
    snap = gpu_snapshots[CASES["thick"]["snapshot"]]
    kw = dict(case_params("thick"), frequencies=[43e9 * 2.0 ** k for k in range(nfreqs)], m_unit=1e20, precision=precision)
    W, H = kw["img_width"], kw["img_height"]
    rng = np.random.default_rng(1)
    orders = [np.arange(W * H, dtype=np.int32), rng.permutation(W * H).astype(np.int32), P.schedule_morton(W, H)]
    out = []
    for order in orders:
        for refill in (0,) if pipeline else (1, 24):
            p = P.make_params(**kw)
            p.refill_lanes, p.tau_fp64 = refill, tau_fp64
            out.append(snap.render(p, jobs=order)[0])
    assert np.abs(out[0]).max() > 0
    for other in out[1:]:
        assert np.array_equal(out[0], other)
