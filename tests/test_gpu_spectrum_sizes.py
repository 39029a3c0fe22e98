"""Device spectra at the edges of the reduction's rounds (needs a GPU).

A cluster of 16 CTAs of 512 threads takes 8,192 pixels a step and six steps a round.  The sums are of positive numbers
in FP64, in another order than numpy's: at most n roundings of 1.1e-16 on each side bound the difference, and pairwise
partial sums keep it far below 1e-12."""
from __future__ import annotations

import numpy as np
import pytest

import phoenix_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npix", [511, 8191, 8193, 49151, 49152, 49153, 331 * 297])
@pytest.mark.parametrize("F", [1, 2, 5])
def test_totals(npix, F):
    import torch
    rng = np.random.default_rng(npix + F)
    res = rng.lognormal(size=(npix, 1, F, 6))
    res[npix // 2, 0, F - 1, 3] = np.nan
    p = P.make_params(img_width=npix, img_height=1, frequencies=[100e9 * (f + 1) for f in range(F)])
    d_res = torch.from_numpy(res).cuda()
    d_spec = torch.zeros((F, 8), dtype=torch.float64, device="cuda")
    P.device_spectrum(p, d_res.data_ptr(), d_spec.data_ptr(), torch.cuda.current_stream().cuda_stream)
    spec = d_spec.cpu().numpy()
    counts = d_spec.cpu()[:, 6:].contiguous().view(torch.int64).numpy()
    r = res.reshape(npix, F, 6)
    for f in range(F):
        ok = np.isfinite(r[:, f].sum(-1))
        np.testing.assert_allclose(spec[f, :4], r[ok, f, :4].sum(0) * P.pixel_solid_angle(p) * P.JANSKY, rtol=1e-12)
        np.testing.assert_allclose(spec[f, 4:6], r[ok, f, 4:].mean(0), rtol=1e-12)
        assert (counts[f] == ok.sum()).all()
