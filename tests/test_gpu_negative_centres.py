"""Gaussian lines whose centre is below zero (the width is a constant, so the
profile is defined there) reach the bins that they reach in the FP64 oracle,
on a grid that begins at zero and on one that begins below."""
import numpy as np
import pytest
import torch

from gexs_b200 import Job, LineList, _capi as capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu_start", [0.0, -20.0])
@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32])
def test_gaussian_lines_below_zero(gpu_ctx, nu_start, precision):
    rng = np.random.Generator(np.random.PCG64(5))
    n, g = 70, 4000
    L = {"nu": np.sort(rng.uniform(-12.0, -1.1, n)), "elow": rng.uniform(0.0, 2000.0, n),
         "aif": 10.0 ** rng.uniform(-2, 1, n), "gns": np.full(n, 3, dtype=np.int32)}
    out = torch.zeros(g, dtype=torch.float64, device="cuda")
    job = Job(LineList.from_dict(L), out, convention=capi.CONV_PHYSICAL, profile=capi.GAUSSIAN,
              temperature=900.0, pressure=0.2, partition=100.0, mass=18.0, nu_start=nu_start,
              dnu=0.01, grid_points=g, precision=precision, cutoff=25.0, half_width=0.5)
    gpu_ctx.run([job])
    gpu_ctx.check()
    want, got = H.oracle_of(job, L), out.cpu().numpy()
    assert np.max(np.abs(want)) > 0.0
    if precision == capi.FP64:
        worst, nbad = H.fp64_mismatch(got, want, abs_floor=1e-14 * np.max(np.abs(want)))
        assert nbad == 0, worst
    else:
        rel, _ = H.fp32_errors(got, want)
        assert rel <= H.FP32_REL, rel
