"""FP64 tiles of 2048 bins (8 bins x 8 warps) are cut into slices like narrower
ones: a dense band takes about as long as with 1024 bins, and has the same
bits, at grid ends around a sub-tile of 1024 bins."""
import pytest
import torch

from gexs_b200 import Job, LineList, synth, _capi as capi

pytestmark = pytest.mark.gpu


def _run(gpu_ctx, lines, profile, points, cfg, repeat=1):
    out = torch.zeros(points, dtype=torch.float64, device="cuda")
    job = Job(lines, out, convention=capi.CONV_PHYSICAL, profile=profile, temperature=1500.0,
              pressure=0.1, partition=1e3, mass=18.0, nu_start=2000.0, dnu=0.01,
              grid_points=points, precision=capi.FP64, cutoff=25.0)
    best = float("inf")
    for _ in range(repeat):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        gpu_ctx.run([job], cfg=cfg)
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    gpu_ctx.check()
    return out, best


@pytest.mark.parametrize("profile", [capi.DOPPLER, capi.VOIGT])
def test_dense_band(gpu_ctx, profile):
    d = synth.make_lines_torch(synth.make_states(20000, 40, 71), 300000, 2000.0, 2080.0, 72, 73)
    lines = LineList(d["nu"], d["elow"], d["aif"], d["gns"], d["gamma"], d["n"])
    for points in (8001, 1, 1023, 1025, 2049):
        narrow, t0 = _run(gpu_ctx, lines, profile, points, (4, 8, 0), 3)
        wide, t1 = _run(gpu_ctx, lines, profile, points, (8, 8, 0), 3)
        assert torch.equal(narrow.view(torch.int64), wide.view(torch.int64)), points
        if points == 8001:
            assert t1 < 5.0 * t0, (t0, t1)      # about 1.1; 12 to 70 in one piece
