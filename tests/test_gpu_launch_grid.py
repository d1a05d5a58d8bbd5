"""ctas_per_sm of a launch configuration holds for the kernel that computes the
profile, in both precisions (grids as the profiler records them)."""
import json

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from gexs_b200 import Job, LineList, synth, _capi as capi

pytestmark = pytest.mark.gpu

MAIN = {(capi.DOPPLER, capi.FP64): "core_kernel", (capi.DOPPLER, capi.FP32): "tile_kernel",
        (capi.VOIGT, capi.FP64): "tile_kernel", (capi.VOIGT, capi.FP32): "voigt_ws_kernel"}


@pytest.mark.parametrize("prof,precision", list(MAIN))
def test_ctas_per_sm(gpu_ctx, tmp_path, prof, precision):
    d = synth.make_lines_torch(synth.make_states(2000, 40, 71), 200000, 2000.0, 2400.0, 72, 73)
    lines = LineList(d["nu"], d["elow"], d["aif"], d["gns"], d["gamma"], d["n"])
    out = torch.zeros(400001, dtype=torch.float64, device="cuda")
    job = Job(lines, out, convention=capi.CONV_PHYSICAL, profile=prof, temperature=1500.0,
              pressure=0.1, partition=1e3, mass=18.0, nu_start=2000.0, dnu=0.001,
              grid_points=400001, precision=precision, cutoff=25.0)
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    gpu_ctx.run([job], cfg=(4, 4, 1))
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        gpu_ctx.run([job], cfg=(4, 4, 1))
        torch.cuda.synchronize()
    path = str(tmp_path / "trace.json")
    p.export_chrome_trace(path)
    with open(path) as f:
        grids = [e["args"]["grid"] for e in json.load(f)["traceEvents"]
                 if e.get("cat") == "kernel" and MAIN[(prof, precision)] in e["name"]]
    assert grids and all(g[0] == nsm for g in grids), grids
