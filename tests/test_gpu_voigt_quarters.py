"""FP32 Voigt launches of few tiles take quarters of a tile as work items; the
same job next to a large one takes whole tiles.  Both give the same bits, at
grid ends around a quarter and a tile, with slices (more than 16384 lines in
a tile), window edges inside a quarter and accumulation, and match the FP64
oracle."""
import numpy as np
import pytest
import torch

from gexs_b200 import Job, LineList, _capi as capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _job(lines, points, out, dnu=0.01, cutoff=25.0, accumulate=0):
    return Job(lines, out, convention=capi.CONV_PHYSICAL, profile=capi.VOIGT, temperature=900.0,
               pressure=0.3, partition=30.0, mass=18.0, nu_start=3000.0, dnu=dnu,
               grid_points=points, precision=capi.FP32, cutoff=cutoff, accumulate=accumulate)


@pytest.mark.parametrize("points,n,cutoff", [
    (1, 500, 25.0), (127, 500, 25.0), (129, 3000, 1.7), (385, 3000, 25.0), (513, 40000, 25.0),
    (2047, 3000, 4.0)])
def test_quarters_are_bitwise_the_whole_tile(gpu_ctx, points, n, cutoff):
    rng = np.random.Generator(np.random.PCG64(points))
    L = {"nu": np.sort(rng.uniform(2995.0, 3025.0, n)), "elow": rng.uniform(0.0, 2000.0, n),
         "aif": 10.0 ** rng.uniform(-2, 1, n), "gns": np.full(n, 3, dtype=np.int32),
         "gamma": rng.uniform(0.03, 0.1, n), "n": rng.uniform(0.4, 0.8, n)}
    lines = LineList.from_dict(L)
    init = rng.uniform(0.0, 1e-24, points)
    for accumulate in (0, 1):
        outs = [torch.as_tensor(init.copy(), device="cuda") for _ in range(2)]
        a, b = (_job(lines, points, o, cutoff=cutoff, accumulate=accumulate) for o in outs)
        big = _job(lines, 400000, torch.zeros(400000, dtype=torch.float64, device="cuda"), 0.002)
        gpu_ctx.run([a])
        gpu_ctx.run([big, b])
        gpu_ctx.check()
        ra, rb = (o.cpu().numpy() for o in outs)
        assert np.array_equal(ra.view(np.int64), rb.view(np.int64))
        want = H.oracle_of(a, L, out=init.copy() if accumulate else None)
        rel, band = H.fp32_errors(ra, want)
        assert rel <= H.FP32_REL and band <= H.FP32_BAND, (rel, band)
