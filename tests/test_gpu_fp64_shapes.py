"""FP64 results have the same bits for every launch shape: sparse lists (the
core kernel walks line by line), dense ones (lane groups), cores in every
region, tiles cut into slices, |x| = 32 of the quadrature inside a warp's
bins."""
import pytest
import torch

from gexs_b200 import Job, LineList, synth, _capi as capi

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4, 0), (2, 4, 0), (8, 4, 0), (2, 8, 0), (4, 8, 0), (8, 8, 0)]


# profile, lines, first and last wavenumber, spacing, T, P
CASES = [
    (capi.VOIGT, 2000, 2000.0, 2400.0, 0.005, 1500.0, 0.01),
    (capi.VOIGT, 40000, 2000.0, 2040.0, 0.01, 1500.0, 1.0),
    (capi.VOIGT, 3000, 9000.0, 9100.0, 0.002, 2500.0, 0.1),
    (capi.DOPPLER, 2000, 2000.0, 2400.0, 0.005, 2500.0, 0.01),
    (capi.VOIGT_QUAD, 8000, 2000.0, 2400.0, 0.01, 1500.0, 0.1),
    (capi.VOIGT_QUAD, 3000, 2000.0, 2400.0, 0.05, 2500.0, 1.0),
]


@pytest.mark.parametrize("case", CASES, ids=[str(i) for i in range(len(CASES))])
def test_bits_are_those_of_every_shape(gpu_ctx, case):
    profile, n, lo, hi, dnu, t, p = case
    d = synth.make_lines_torch(synth.make_states(20000, 40, 71), n, lo, hi, 72, 73)
    lines = LineList(d["nu"], d["elow"], d["aif"], d["gns"], d["gamma"], d["n"])
    g = int(round((hi - lo) / dnu)) + 1
    for cfg, nodes in [(c, k) for k in ((16, 32) if profile == capi.VOIGT_QUAD else (16,))
                       for c in SHAPES]:
        out = torch.zeros(g, dtype=torch.float64, device="cuda")
        job = Job(lines, out, convention=capi.CONV_PHYSICAL, profile=profile, temperature=t,
                  pressure=p, partition=1e3, mass=18.0, nu_start=lo, dnu=dnu, grid_points=g,
                  precision=capi.FP64, cutoff=25.0, quad_nodes=nodes)
        gpu_ctx.run([job], cfg=cfg)
        gpu_ctx.check()
        bits = out.view(torch.int64)
        assert float(out.max()) > 0.0
        if cfg == SHAPES[0]:
            first = bits
        bad = int((bits != first).sum())
        assert bad == 0, (cfg, nodes, bad)
