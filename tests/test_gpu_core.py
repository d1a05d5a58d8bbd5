"""The Voigt core kernel (Humlicek regions II-IV) at the sizes where its
walk over a line's bins changes form: ranges of no bin, of a few bins
(several lane groups, private strips), of more than 32 and of hundreds of
bins (several passes, ranges cut by tile edges), groups of lines too far
apart for the strips, line counts around a group of 32 and a slice of 2048.
FP32 and FP64 forms against the FP64 CPU oracle with the suite's tolerances
(1e-4 on bins above 1e-6 of the peak and 1e-6 on the band for FP32, 1e-10
per bin for FP64)."""
import numpy as np
import pytest
import torch

from gexs_b200 import Job, LineList, _capi as capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


# lines, first centre, span of the centres, spacing, T, P
CASES = [
    (1, 500.0, 0.0, 0.1, 100.0, 1e-5),
    (31, 900.0, 40.0, 0.1, 100.0, 1e-5),        # ranges of 0-1 bins, sparse
    (33, 3000.0, 0.3, 0.01, 1500.0, 0.01),      # ranges of ~20 bins, dense
    (400, 3000.0, 120.0, 0.01, 1500.0, 1.0),    # sparse: wider than a strip
    (4100, 2000.0, 2.0, 0.01, 1500.0, 1.0),     # three slices of one tile
    (65, 8000.0, 2.0, 0.001, 3000.0, 1e-4),     # ranges of hundreds of bins
    (2049, 20000.0, 8.0, 0.004, 3000.0, 0.03),
    (97, 150.0, 3.0, 0.002, 296.0, 10.0),       # y above 15: no core
]


@pytest.mark.parametrize("case", CASES, ids=[str(i) for i in range(len(CASES))])
def test_core_ranges_match_oracle(gpu_ctx, case):
    n, nu0, span, dnu, T, P = case
    rng = np.random.Generator(np.random.PCG64(n))
    nu = np.sort(nu0 + span * rng.random(n))
    L = {"nu": nu, "elow": rng.uniform(0.0, 2000.0, n), "aif": 10.0 ** rng.uniform(-2, 1, n),
         "gns": (2 * rng.integers(0, 40, n) + 1).astype(np.int32),
         "gamma": rng.uniform(0.03, 0.1, n), "n": rng.uniform(0.4, 0.8, n)}
    lines = LineList.from_dict(L)
    lo, g = nu0 - 1.3, int((span + 2.6) / dnu) + 1
    for precision in (capi.FP32, capi.FP64):
        out = torch.full((g,), 7.0, dtype=torch.float64, device="cuda")
        job = Job(lines, out, convention=capi.CONV_PHYSICAL, profile=capi.VOIGT, temperature=T,
                  pressure=P, partition=100.0, mass=18.0, nu_start=lo, dnu=dnu, grid_points=g,
                  precision=precision, cutoff=25.0)
        gpu_ctx.run([job])
        gpu_ctx.check()
        want = H.oracle_of(job, L)
        got = out.cpu().numpy()
        if precision == capi.FP64:
            worst, nbad = H.fp64_mismatch(got, want)
            assert nbad == 0, worst
        else:
            rel, band = H.fp32_errors(got, want)
            assert rel <= H.FP32_REL and band <= H.FP32_BAND, (rel, band)


@pytest.mark.parametrize("dop,gamma", [(None, -0.02), (1e-58, 0.05), (1e-70, 0.05), (1e-70, 0.0)])
def test_fp64_general_tier(gpu_ctx, dop, gamma):
    """FP64 lines outside the fast tiers: y < 0 (the whole line per bin), |x|
    or y near and beyond 1e60 (IEEE divisions, no x^4 overflow)."""
    rng = np.random.Generator(np.random.PCG64(5))
    n, g = 70, 1500
    L = {"nu": np.sort(rng.uniform(1000.0, 1012.0, n)), "elow": rng.uniform(0.0, 2000.0, n),
         "aif": 10.0 ** rng.uniform(-2, 1, n), "gns": np.full(n, 3, dtype=np.int32),
         "gamma": np.where(np.arange(n) % 3 == 0, gamma, 0.04), "n": np.full(n, 0.5)}
    out = torch.zeros(g, dtype=torch.float64, device="cuda")
    job = Job(LineList.from_dict(L), out, convention=capi.CONV_PHYSICAL, profile=capi.VOIGT,
              temperature=900.0, pressure=0.2, partition=100.0, mass=18.0, nu_start=998.0,
              dnu=0.01, grid_points=g, precision=capi.FP64, cutoff=25.0)
    if dop is not None:
        job.c.dop_coef = dop
    gpu_ctx.run([job])
    gpu_ctx.check()
    want = H.oracle_of(job, L)
    assert np.isfinite(want).all()
    worst, nbad = H.fp64_mismatch(out.cpu().numpy(), want, abs_floor=1e-13 * np.max(np.abs(want)))
    assert nbad == 0, worst


@pytest.mark.parametrize("profile", [capi.VOIGT, capi.VOIGT_QUAD])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_fp64_infinite_line_stays_in_its_window(gpu_ctx, profile, bad):
    """A line whose intensity is infinite or not a number makes the bins of
    its window so, and no others, as in the oracle."""
    n, g = 700, 3000
    rng = np.random.Generator(np.random.PCG64(11))
    L = {"nu": np.sort(rng.uniform(1000.0, 1030.0, n)), "elow": np.full(n, 50.0),
         "aif": 10.0 ** rng.uniform(-2, 1, n), "gns": np.full(n, 3, dtype=np.int32),
         "gamma": np.full(n, 0.05), "n": np.full(n, 0.5)}
    L["aif"][n // 2] = bad
    out = torch.zeros(g, dtype=torch.float64, device="cuda")
    job = Job(LineList.from_dict(L), out, convention=capi.CONV_PHYSICAL, profile=profile,
              temperature=900.0, pressure=0.2, partition=100.0, mass=18.0, nu_start=1000.0,
              dnu=0.01, grid_points=g, precision=capi.FP64, cutoff=2.3)
    gpu_ctx.run([job])
    gpu_ctx.check()
    want, got = H.oracle_of(job, L), out.cpu().numpy()
    fine = np.isfinite(want)
    assert 0 < fine.sum() < g
    assert np.array_equal(got[~fine], want[~fine], equal_nan=True)
    worst, nbad = H.fp64_mismatch(got[fine], want[fine])
    assert nbad == 0, worst
