"""The FP64 Gauss-Hermite sum's three forms (asymptotic series at |x| >= 32,
node sum with refined reciprocals, IEEE node sum) on either side of the
lines between them, against the FP64 CPU oracle within 1e-10 per bin: widths
that put |x| = 32 inside a warp's bins, y from 0 and 1e-120 to 1e4, windows
that end inside a tile."""
import numpy as np
import pytest
import torch

from gexs_b200 import Job, LineList, _capi as capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [16, 32])
@pytest.mark.parametrize("nu0,dnu,gamma", [
    (3000.0, 0.002, 0.05), (3000.0, 0.01, 1e-7), (800.0, 0.05, 0.0), (3000.0, 0.01, 1e-122),
    (200.0, 0.02, 3.0), (9000.0, 0.1, 0.08), (9000.0, 0.0003, 0.01)])
def test_forms_match_oracle(gpu_ctx, nodes, nu0, dnu, gamma):
    rng = np.random.Generator(np.random.PCG64(nodes))
    n, g = 37, 2111
    L = {"nu": np.sort(nu0 + g * dnu * rng.uniform(-0.3, 1.3, n)), "elow": np.full(n, 100.0),
         "aif": 10.0 ** rng.uniform(-2, 1, n), "gns": np.full(n, 5, dtype=np.int32),
         "gamma": gamma * rng.uniform(0.5, 1.0, n), "n": np.full(n, 0.5)}
    out = torch.zeros(g, dtype=torch.float64, device="cuda")
    job = Job(LineList.from_dict(L), out, convention=capi.CONV_PHYSICAL,
              profile=capi.VOIGT_QUAD, temperature=700.0, pressure=1.0, partition=50.0, mass=18.0,
              nu_start=nu0, dnu=dnu, grid_points=g, precision=capi.FP64, quad_nodes=nodes,
              cutoff=0.4 * g * dnu)
    gpu_ctx.run([job])
    gpu_ctx.check()
    want = H.oracle_of(job, L)
    worst, nbad = H.fp64_mismatch(out.cpu().numpy(), want, abs_floor=1e-300)
    assert nbad == 0, worst
