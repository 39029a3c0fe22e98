"""Batches and servers of more than 4 frequencies (needs a GPU): the 32-slot queue kernels, at every register cap, in
128-thread blocks and in whole-SM ones, against single renders.  Separate compilations round the FP32
coefficients and the operator differently (a few ulp of 6e-8, sums of about 10^3 samples): 1e-5 of the largest value."""
from __future__ import annotations

import numpy as np
import pytest

import phoenix_b200 as P
from tests.golden.cases import case_params

pytestmark = pytest.mark.gpu


def _params(nfreqs, side, precision="fp32", **kw):
    freqs = [86e9 * 4.0 ** (k / max(1, nfreqs - 1)) for k in range(nfreqs)]
    return P.make_params(**dict(case_params("edge"), img_width=side, img_height=side, precision=precision, frequencies=freqs,
                                **kw))


def _close(a, b):
    for part in (slice(0, 4), slice(4, 5), slice(5, 6)):
        assert np.abs(a[..., part] - b[..., part]).max() <= 1e-5 * np.abs(b[..., part]).max()


@pytest.mark.parametrize("bps,block", [(1, 128), (3, 384), (4, 512)])
@pytest.mark.parametrize("nfreqs,side", [(5, 20), (32, 20), (5, 280), (32, 280)])
def test_batches(gpu_snapshots, bps, block, nfreqs, side):
    snap = gpu_snapshots["small"]
    p = _params(nfreqs, side)
    ref, _ = snap.render(p)
    with P.Batch([(snap, p)], blocks_per_sm=bps) as b:
        b.run()
        res, info = b.result(0)
    assert info["block"] == (block if side == 280 else 128)
    _close(res, ref)


def test_autotuned_batch(gpu_snapshots):
    """Three register caps x three refill policies, then the five other tile shapes."""
    snap = gpu_snapshots["small"]
    p = _params(6, 40)
    with P.Batch([(snap, p)], autotune=True, sample_stride=2) as b:
        t = b.tuning()
        b.run()
        res, _ = b.result(0)
    assert sorted({c["blocks_per_sm"] for c in t["candidates"][:9]}) == [1, 3, 4] and t["ncand"] == 14
    _close(res, snap.render(p)[0])


@pytest.mark.parametrize("bps", [1, 3, 4])
def test_server(gpu_snapshots, bps):
    snap = gpu_snapshots["small"]
    ps = [_params(n, 24, inclination=float(i)) for n, i in ((5, 20), (32, 75), (1, 120), (17, 163))]
    with P.Server([snap], "fp32", max_freqs=32, blocks_per_sm=bps, arena_bytes=1 << 26) as srv:
        ids = [srv.submit(0, p) for p in ps]
        for i in ids:
            srv.wait(i, 100.0)
        out = [srv.result(i)[0] for i in ids]
    for p, res in zip(ps, out):
        _close(res, snap.render(p)[0])
