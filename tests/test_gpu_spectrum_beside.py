"""Device spectra beside other work, and their rounding (needs a GPU)."""
from __future__ import annotations

import math
import time

import numpy as np
import pytest

import phoenix_b200 as P
from tests.golden.cases import case_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,side", [("fp32", 64), ("fp32", 96), ("mixed", 64), ("fp64", 64)])
def test_starts_beside_a_small_render(gpu_snapshots, precision, side):
    """A render that leaves part of every SM free does not hold a spectrum on another stream up: the spectrum (tens of
    microseconds) takes less than a tenth of the render (10 ms and more) that runs meanwhile; waiting for SMs of its own, it
    took a third."""
    import torch
    p = P.make_params(**dict(case_params("cfg1"), img_width=side, img_height=side, precision=precision))
    q = P.make_params(img_width=256, img_height=256, frequencies=[1e11, 2e11])
    jobs = torch.from_numpy(P.schedule_morton(side, side)).cuda()
    res = torch.zeros(side, side, 1, 6, dtype=torch.float64, device="cuda")
    img = torch.rand(256, 256, 2, 6, dtype=torch.float64, device="cuda")
    spec = torch.zeros(2, 8, dtype=torch.float64, device="cuda")
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    share = []
    for _ in range(4):  # the first loads the kernels
        ctr = torch.zeros(P.NUM_COUNTERS, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        gpu_snapshots["cfg1"].render_async(p, jobs.data_ptr(), jobs.numel(), res.data_ptr(), ctr.data_ptr(), stream=a.cuda_stream)
        time.sleep(1e-3)
        t0 = time.perf_counter()
        P.device_spectrum(q, img.data_ptr(), spec.data_ptr(), b.cuda_stream)
        b.synchronize()
        t1 = time.perf_counter()
        a.synchronize()
        share.append((t1 - t0) / (time.perf_counter() - t0))
    assert min(share) < 0.1
    np.testing.assert_allclose(spec[:, 4].cpu().numpy(), img[..., 4].mean(dim=(0, 1)).cpu().numpy(), rtol=1e-12)


@pytest.mark.parametrize("npix", [1, 255, 4097, 20481, 300 * 300])
def test_totals_against_the_exact_sum(npix):
    """Sums of positive numbers of a like size: the threads' partial sums average their roundings out, the rest is
    compensated.  Left are the roundings of the total, of its product with the solid angle or its division, and of the
    same on this side: 4 x 1.1e-16."""
    import torch
    rng = np.random.default_rng(npix)
    res = rng.lognormal(size=(npix, 1, 2, 6))
    p = P.make_params(img_width=npix, img_height=1, frequencies=[1e11, 2e11])
    d_res = torch.from_numpy(res).cuda()
    d_spec = torch.zeros((2, 8), dtype=torch.float64, device="cuda")
    P.device_spectrum(p, d_res.data_ptr(), d_spec.data_ptr(), torch.cuda.current_stream().cuda_stream)
    spec = d_spec.cpu().numpy()
    for f in range(2):
        exact = [math.fsum(res[:, 0, f, k]) for k in range(6)]
        jy = P.pixel_solid_angle(p) * P.JANSKY
        want = [e * jy for e in exact[:4]] + [e / npix for e in exact[4:]]
        assert np.abs(spec[f, :6] / want - 1.0).max() <= 4.5e-16
