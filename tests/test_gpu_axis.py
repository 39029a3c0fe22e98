"""Mixed images at the axis (needs a GPU): the central column of an image of odd width.

Its rays have no angular momentum and pass the poles at 1e-11, where FP64 holds the distance to the south pole to 1e-5
only: any change of the geodesic's roundings moves what they cross behind the pole, by up to 1e-2 of the image's scale at a
pixel.  The values in golden/axis.npz (optical depth and Faraday depth of three frequencies, cfg1 snapshot) are those of
the kernels whose geodesic had its roundings from the compiler, before they were spelled out.  Neither depends on the
segment operator: what may differ is the rounding of the FP32 coefficients (a few ulp of 6e-8) in sums of some
hundred samples of one sign, so 5e-7 of the column's largest value.  Every kernel has to give them: plain, pipelined,
batch, and of 1, 4 and 32 frequency slots.
"""
from __future__ import annotations

import os

import numpy as np
import pytest

import phoenix_b200 as P
from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu

W, H = 33, 41
COLUMN = np.arange(W // 2 * H, (W // 2 + 1) * H, dtype=np.int32)


@pytest.mark.parametrize("kernel,nfreqs", [("pipeline", 1), ("pipeline", 3), ("pipeline", 7), ("plain", 1), ("plain", 3),
                                           ("plain", 7), ("batch", 1), ("batch", 3)])
@pytest.mark.parametrize("incl", [20, 130])
def test_column_over_the_poles(gpu_snapshots, incl, nfreqs, kernel):
    ref = np.load(os.path.join(GOLDEN, "axis.npz"))[f"i{incl}"].astype(np.float64)
    p = P.make_params(img_width=W, img_height=H, inclination=float(incl), phi=33.0, m_unit=1e19, precision="mixed",
                      frequencies=[86e9 * 2.0 ** k for k in range(nfreqs)])
    snap = gpu_snapshots["cfg1"]
    if kernel == "batch":
        with P.Batch([(snap, p, COLUMN)]) as b:
            b.run()
            res, _ = b.result(0)
    else:
        p.refill_lanes = 24 if kernel == "plain" else 0
        res, _ = snap.render(p, jobs=COLUMN)
    n = min(nfreqs, 3)
    got = res[W // 2, :, :n, 4:]
    assert (np.abs(got - ref[:, :n]).max(axis=0) <= 5e-7 * np.abs(ref[:, :n]).max(axis=0)).all()


@pytest.mark.parametrize("incl", [20.0, 75.0])
def test_pipelined_and_plain_sample_alike(gpu_snapshots, incl):
    """An image of odd width and three frequencies, 488 rays an SM: the same samples in every pixel, Faraday depths to 1e-5
    of the largest (the bound of separately compiled coefficients, far below what one sample more or less moves)."""
    import torch
    snap, W, H = gpu_snapshots["cfg1"], 333, 217
    jobs = torch.from_numpy(P.schedule_morton(W, H)).cuda()
    out = []
    for refill in (0, 24):
        p = P.make_params(img_width=W, img_height=H, inclination=incl, phi=33.0, m_unit=1e19, precision="mixed",
                          frequencies=[86e9, 172e9, 344e9])
        p.refill_lanes = refill
        res = torch.zeros(W * H, 3, 6, dtype=torch.float64, device="cuda")
        ps = torch.zeros(W * H, 3, dtype=torch.int32, device="cuda")
        ctr = torch.zeros(P.NUM_COUNTERS, dtype=torch.int64, device="cuda")
        snap.render_async(p, jobs.data_ptr(), W * H, res.data_ptr(), ctr.data_ptr(), ps.data_ptr(),
                          stream=torch.cuda.current_stream().cuda_stream)
        out.append((res.cpu().numpy(), ps.cpu().numpy()))
    (a, pa), (b, pb) = out
    assert np.array_equal(pa, pb)
    assert (np.abs(a[..., 5] - b[..., 5]).max(axis=0) <= 1e-5 * np.abs(b[..., 5]).max(axis=0)).all()
