"""Per-pixel counts of the pipelined and the plain kernel (needs a GPU): the same, for every form of job list.

A snapshot with NaN densities in one corner makes bad samples (a NaN segment is left out and counted).  A pixel that is in the
job list several times has the counts of one ray, as each of its rays stores its own."""
from __future__ import annotations

import math

import numpy as np
import pytest

import phoenix_b200 as P

pytestmark = pytest.mark.gpu

W, H = 24, 20


@pytest.fixture(scope="module")
def torn_snapshot():
    """One uniform block, its inner quarter without a density."""
    n = 8
    lo, hi = [math.log(1.2), 0.0, 0.0], [math.log(100.0), math.pi, 2.0 * math.pi]
    prim = np.zeros((1, n, n, n, 8), np.float32)
    prim[..., 0], prim[..., 1], prim[..., 5], prim[..., 6] = 1.0, 0.03, 0.05, 0.02
    prim[:, :, :, :3, 0] = np.nan  # x1 is the fastest index
    with P.Snapshot.from_arrays(nx=[n] * 3, ng=[1, 1, 1], nlevels=1, a=0.9375, hslope=0.25, gam=13.0 / 9.0, x_lo=lo, x_hi=hi,
                                lb=np.array([lo]), dxc=np.array([[(h - l) / n for l, h in zip(lo, hi)]]),
                                level_maps=[np.zeros((1, 1, 1), np.int32)], prim_f32=prim.reshape(1, n ** 3, 8)) as snap:
        yield snap


def _counts(snap, precision, nfreqs, refill, jobs):
    import torch
    p = P.make_params(img_width=W, img_height=H, precision=precision, sigma_cut=1e30, rt_outer=50.0,
                      frequencies=[86e9 * 2.0 ** k for k in range(nfreqs)])
    p.refill_lanes = refill
    d_jobs = torch.from_numpy(jobs).cuda()
    res = torch.zeros(W * H * nfreqs * 6, dtype=torch.float64, device="cuda")
    ps = torch.full((W * H, 3), -7, dtype=torch.int32, device="cuda")
    ctr = torch.zeros(P.NUM_COUNTERS, dtype=torch.int64, device="cuda")
    snap.render_async(p, d_jobs.data_ptr(), jobs.size, res.data_ptr(), ctr.data_ptr(), ps.data_ptr(),
                      stream=torch.cuda.current_stream().cuda_stream)
    return ps.cpu().numpy(), int(ctr[P.CTR["bad"]])


@pytest.mark.parametrize("precision", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("nfreqs", [1, 3, 7])
@pytest.mark.parametrize("jobs", ["each", "twice", "in one warp"])
def test_counts(torn_snapshot, precision, nfreqs, jobs):
    each = np.arange(W * H, dtype=np.int32)
    half = each[W * H // 4:-W * H // 4]
    jobs = {"each": each, "twice": np.concatenate([half, half[::-1]]), "in one warp": np.repeat(half[100:130], 16)}[jobs].copy()
    a, bad_a = _counts(torn_snapshot, precision, nfreqs, 0, jobs)
    b, bad_b = _counts(torn_snapshot, precision, nfreqs, 24, jobs)
    assert (b[:, 2] > 0).any() and (b[jobs, 2] >= 0).all()
    assert np.array_equal(a, b) and bad_a == bad_b
