"""The core kernel's line slices depend on the job alone: a cross-section of a
long list on a grid of few tiles has the same bits alone and in a launch
whose partial rows pass 1 GiB (they are then taken in rounds), in both
precisions; and a request for a band of one tile does not reserve rows for
the whole list."""
import numpy as np
import pytest
import torch

from gexs_b200 import Job, LineList, synth, _capi as capi
from gexs_b200.engine import Server
from tests import helpers as H

pytestmark = pytest.mark.gpu

LO, HI, DNU = 2000.0, 2700.0, 0.01


@pytest.fixture(scope="module")
def long_list():
    st = synth.make_states(20000, 40, 61)
    return st, synth.make_lines_torch(st, 10000000, LO, HI, 62, 63)


def _job(lines, precision, temperature):
    g = int(round((HI - LO) / DNU)) + 1                   # 137 tiles of 512 bins
    out = torch.zeros(g, dtype=torch.float64, device="cuda")
    return Job(lines, out, convention=capi.CONV_PHYSICAL, profile=capi.VOIGT,
               temperature=temperature, pressure=1e-3, partition=1e3, mass=18.0, nu_start=LO,
               dnu=DNU, grid_points=g, precision=precision, cutoff=0.3)


def test_bits_alone_and_with_others(gpu_ctx, long_list):
    d = long_list[1]
    lines = LineList(d["nu"], d["elow"], d["aif"], d["gns"], d["gamma"], d["n"])
    temps = [300.0, 700.0, 1500.0, 2100.0, 2900.0]
    res = {}
    for precision in (capi.FP64, capi.FP32):
        alone = [_job(lines, precision, t) for t in temps]
        for j in alone:
            gpu_ctx.run([j])
        mixed = [_job(lines, precision, t) for t in temps]
        gpu_ctx.run(mixed)
        gpu_ctx.check()
        for a, m in zip(alone, mixed):
            assert torch.equal(a.out.view(torch.int64), m.out.view(torch.int64)), precision
        res[precision] = [j.out.cpu().numpy() for j in mixed]
    for a, b in zip(res[capi.FP32], res[capi.FP64]):
        rel, band = H.fp32_errors(a, b)
        assert rel <= H.FP32_REL and band <= H.FP32_BAND, (rel, band)


def test_band_request_is_admitted_within_its_scratch(long_list):
    """Prep arrays (24 B a line) and a few rows, not rows for each 256 lines
    of the list."""
    st, d = long_list
    n = d["nu"].numel()
    srv = Server(0, hbm_budget=24 * n + 24 * n + (160 << 20))
    try:
        lid = srv.add_list(d, st.energy, st.g, 18.0, compact=True)
        t = srv.submit(srv.request(lid, capi.VOIGT, 700.0, 1e-3, 2300.0, DNU, 500, cutoff=1.0))
        out, _ = srv.wait(t, 500)
        assert np.isfinite(out).all() and out.max() > 0.0
    finally:
        srv.close()
