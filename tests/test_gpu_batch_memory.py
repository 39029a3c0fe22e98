"""Host memory of a batch (needs a GPU): its job lists, 4 bytes a ray, are not kept once it is created."""
from __future__ import annotations

import os

import pytest

import phoenix_b200 as P
from tests.golden.cases import case_params

pytestmark = pytest.mark.gpu


def _resident_bytes():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGE_SIZE")


def test_job_lists_are_released(gpu_snapshots):
    """Two images of 2048^2: 33.6 MB of job lists.  The first batch of the process loads the kernels."""
    p = P.make_params(**dict(case_params("edge"), img_width=2048, img_height=2048, precision="fp32"))
    items = [(gpu_snapshots["small"], p)] * 2
    P.Batch(items).close()
    before = _resident_bytes()
    with P.Batch(items):
        kept = _resident_bytes() - before
    assert kept < 2 * 2048 * 2048 * 4 // 2
