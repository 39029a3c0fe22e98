"""Which kernel a default launch takes (needs a GPU): the pipelined one below the measured break-even, the plain one above.

The break-even lies lower without a line of rays along the axis (even widths) and with one frequency more than the plasma
warps share evenly; images between the two limits ran up to a fifth longer in the pipeline."""
from __future__ import annotations

import numpy as np
import pytest

import phoenix_b200 as P
from tests.golden.cases import case_params

pytestmark = pytest.mark.gpu

PIPE = {1: 64, 2: 96, 3: 96, 4: 96, 5: 160, 8: 160}


@pytest.mark.parametrize("precision,nfreqs,rays,odd,pipe", [
    ("fp32", 1, 640, 0, True), ("fp32", 1, 670, 0, False), ("fp32", 1, 690, 1, True), ("fp32", 1, 710, 1, False),
    ("fp32", 3, 440, 0, True), ("fp32", 3, 480, 0, False), ("fp32", 3, 490, 1, True), ("fp32", 4, 490, 0, True),
    ("fp32", 5, 310, 0, True), ("mixed", 1, 640, 0, True), ("mixed", 1, 670, 0, False), ("mixed", 1, 840, 1, True),
    ("mixed", 2, 410, 0, True), ("mixed", 2, 440, 0, False), ("mixed", 3, 350, 0, True), ("mixed", 3, 390, 0, False),
    ("mixed", 3, 490, 0, False), ("mixed", 3, 490, 1, True), ("mixed", 5, 230, 0, True), ("mixed", 5, 260, 0, False),
    ("mixed", 8, 290, 0, True), ("fp64", 3, 130, 0, True), ("fp64", 3, 150, 0, False)])
def test_kernel_taken(gpu_snapshots, precision, nfreqs, rays, odd, pipe):
    """The rays that count are those of the job list; few steps (max_steps) keep the launches short."""
    snap = gpu_snapshots["small"]
    freqs = [86e9 * 4.0 ** (k / max(1, nfreqs - 1)) for k in range(nfreqs)]
    kw = dict(case_params("edge"), precision=precision, frequencies=freqs, max_steps=3)
    sms = snap.render(P.make_params(**dict(kw, img_width=4, img_height=4)))[1]["sms"]
    p = P.make_params(**dict(kw, img_width=400 + odd, img_height=400))
    _, info = snap.render(p, jobs=np.arange(rays * sms, dtype=np.int32))
    assert (info["block"] == PIPE[nfreqs]) == pipe, info["block"]


@pytest.mark.parametrize("pa,W,H,pipe", [(0.0, 401, 400, True), (0.0, 400, 401, False), (90.0, 400, 401, True),
                                         (90.0, 401, 400, False), (30.0, 401, 401, False), (180.0, 401, 400, True)])
def test_line_along_the_axis(gpu_snapshots, pa, W, H, pipe):
    snap = gpu_snapshots["small"]
    p = P.make_params(**dict(case_params("edge"), precision="mixed", img_width=W, img_height=H, pa=pa, max_steps=3))
    _, info = snap.render(p, jobs=np.arange(800 * snap.render(p, jobs=np.arange(4))[1]["sms"], dtype=np.int32))
    assert (info["block"] == PIPE[1]) == pipe
