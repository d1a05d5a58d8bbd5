"""FP32 Doppler/Gaussian tiles split into parts (items of 128 bins) against
the same launch without parts: gexs_run splits a job of few, well filled
tiles, gexs_run_noalloc never does; the two give the same bits, at grid ends
around a part and a tile, and match the FP64 oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

from gexs_b200 import Job, LineList, _capi as capi
from gexs_b200._capi import check, lib
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profile", [capi.DOPPLER, capi.GAUSSIAN])
@pytest.mark.parametrize("points", [1, 127, 129, 513, 1000, 2047])
def test_parts_are_bitwise_the_whole_tile(gpu_ctx, profile, points):
    rng = np.random.Generator(np.random.PCG64(points))
    n, dnu = 6000, 0.01
    L = {"nu": np.sort(rng.uniform(2990.0, 3025.0, n)), "elow": rng.uniform(0.0, 2000.0, n),
         "aif": 10.0 ** rng.uniform(-2, 1, n), "gns": np.full(n, 3, dtype=np.int32)}
    lines = LineList.from_dict(L)
    jobs = []
    for _ in range(2):
        out = torch.full((points,), 3.0, dtype=torch.float64, device="cuda")
        jobs.append(Job(lines, out, convention=capi.CONV_PHYSICAL, profile=profile,
                        temperature=900.0, pressure=1.0, partition=30.0, mass=18.0,
                        nu_start=3000.0, dnu=dnu, grid_points=points, precision=capi.FP32,
                        cutoff=25.0, half_width=0.03))
    gpu_ctx.run([jobs[0]])
    gpu_ctx.check()
    arr = (capi.GexsJob * 1)(jobs[1].c)
    check(lib().gexs_run_noalloc(arr, 1, None, None), "noalloc")
    torch.cuda.synchronize()
    a, b = (j.out.cpu().numpy() for j in jobs)
    assert np.array_equal(a.view(np.int64), b.view(np.int64))
    rel, band = H.fp32_errors(a, H.oracle_of(jobs[0], L))
    assert rel <= H.FP32_REL and band <= H.FP32_BAND, (rel, band)
