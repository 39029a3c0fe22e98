"""The plain kernel where default launches of small images no longer take it (needs a GPU): the thick case against the oracle,
and default images of whole-SM blocks against a part of their pixels in the pipelined kernel.  Separate compilations
round the FP32 coefficients and the operator differently (a few ulp of 6e-8, sums of about 10^3 samples): 1e-5 of the
largest value."""
from __future__ import annotations

import numpy as np
import pytest

import phoenix_b200 as P
from tests.golden.cases import CASES, case_params
from tests.test_gpu_freq_slots import _close, _params
from tests.test_gpu_parity import TOL, flux_errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "mixed", "fp64"])
def test_plain_kernel_matches_oracle(gpu_snapshots, oracle_results, precision):
    """The plain kernel of 4 slots on the thick case, whose default launch is pipelined."""
    ref, _, _ = oracle_results("thick")
    p = P.make_params(precision=precision, **case_params("thick"))
    p.refill_lanes = 24
    res, info = gpu_snapshots[CASES["thick"]["snapshot"]].render(p)
    assert info["block"] == 128
    err = flux_errors(res, ref, p)
    t = TOL[precision]
    assert err[:, 0].max() <= t["flux"] and err[:, 1:].max() <= t.get("pol", t["flux"])
    assert np.abs(res[..., :4] - ref[..., :4]).sum() <= t["l1"] * np.abs(ref[..., :4]).sum()


@pytest.mark.parametrize("precision,nfreqs,block", [("fp32", 1, 512), ("fp32", 3, 512), ("fp32", 6, 512), ("mixed", 1, 512),
                                                    ("mixed", 3, 384), ("mixed", 6, 384)])
def test_large_image(gpu_snapshots, precision, nfreqs, block):
    """A default image of whole-SM blocks against a part of its pixels, which run pipelined."""
    snap = gpu_snapshots["small"]
    side = 384
    p = _params(nfreqs, side, precision)
    full, info = snap.render(p)
    assert info["block"] == block and info["blocks"] == info["sms"]
    jobs = np.arange(11, side * side, 97, dtype=np.int32)
    part, pinfo = snap.render(p, jobs=jobs)
    assert pinfo["block"] < 192 and pinfo["block"] != 128
    _close(part.reshape(-1, nfreqs, 6)[jobs], full.reshape(-1, nfreqs, 6)[jobs])
