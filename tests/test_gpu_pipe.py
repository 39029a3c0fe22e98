"""The pipelined march of small launches (needs a GPU): the same images as the plain kernel, at the edges of its blocks.

A render with default launch parameters and few rays runs in the pipelined kernel; naming a refill policy other than
the default keeps the plain one (24 finished lanes).  The rays are the same step for step.  FP64 is compiled without
contraction and gives the same bits.  FP32 and mixed may round the coefficients and the operator differently in the
two kernels (a few ulp of 6e-8 each, over about 10^3 samples of a sum): 1e-5 of the largest value.
"""
from __future__ import annotations

import numpy as np
import pytest

import phoenix_b200 as P
from tests.golden.cases import case_params

pytestmark = pytest.mark.gpu


def _render(snap, precision, nfreqs, W, H, jobs=None, **kw):
    freqs = [86e9 * 4.0 ** (k / max(1, nfreqs - 1)) for k in range(nfreqs)]
    p = dict(case_params("edge"), img_width=W, img_height=H, precision=precision, frequencies=freqs, **kw)
    out = np.full((W, H, nfreqs, 6), -7.0)
    return snap.render(P.make_params(**p), jobs=jobs, out=out)


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-5), ("mixed", 1e-5), ("fp64", 0.0)])
@pytest.mark.parametrize("nfreqs", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("W,H", [(1, 1), (31, 1), (8, 4), (11, 3), (17, 23)])
def test_same_image_as_the_plain_kernel(gpu_snapshots, precision, tol, nfreqs, W, H):
    snap = gpu_snapshots["small"]
    a, ia = _render(snap, precision, nfreqs, W, H)
    b, ib = _render(snap, precision, nfreqs, W, H, refill_lanes=24)
    assert ia["block"] != ib["block"]
    for key in ("steps", "nplasma", "bad"):
        assert ia[key] == ib[key], key
    for part in (slice(0, 4), slice(4, 5), slice(5, 6)):
        assert np.abs(a[..., part] - b[..., part]).max() <= tol * np.abs(b[..., part]).max()


def test_job_subsets_and_more_rays_than_blocks(gpu_snapshots):
    """A job list of part of the image leaves the other pixels alone; a launch of more rays than resident blocks takes
    several rounds of the job queue."""
    snap = gpu_snapshots["small"]
    jobs = np.arange(5, 300, 7, dtype=np.int32)
    a, _ = _render(snap, "fp64", 1, 20, 17, jobs=jobs)
    b, _ = _render(snap, "fp64", 1, 20, 17)
    flat_a, flat_b = a.reshape(-1, 6), b.reshape(-1, 6)
    rest = np.setdiff1d(np.arange(340), jobs)
    assert np.array_equal(flat_a[jobs], flat_b[jobs]) and (flat_a[rest] == -7.0).all()
    big, ib = _render(snap, "fp32", 1, 240, 250)
    plain, ip = _render(snap, "fp32", 1, 240, 250, refill_lanes=24)
    assert ib["blocks"] * 32 < 240 * 250 and ib["steps"] == ip["steps"] and ib["nplasma"] == ip["nplasma"]
    assert np.abs(big - plain)[..., :4].max() <= 1e-5 * np.abs(plain[..., :4]).max()
