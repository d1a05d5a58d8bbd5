"""The last segment of a long manager pass: its region-I kernel starts after the
segment before has finished (both kernels' times as the profiler records
them, to some microseconds), and the result is that of one launch, bit for bit."""
import json

import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from gexs_b200 import Context, Job, LineList, synth, _capi as capi
from gexs_b200.engine import Manager

pytestmark = pytest.mark.gpu


def test_long_last_segment_waits(tmp_path):
    n, g, lo, dnu = 2200000, 200001, 2000.0, 0.002
    d = synth.make_lines_torch(synth.make_states(20000, 40, 71), n, lo, 2400.0, 72, 73)
    h = {k: v.cpu().pin_memory().numpy() for k, v in d.items()}
    n = len(h["nu"])
    freq = lo + np.arange(g) * dnu
    m = Manager(capi.VOIGT, 0, capi.CONV_REF_GPU, capi.FP32, 8 * g + 44 * (n + 4096))
    try:
        m.initialize_vectors(g, 1)
        m.initialize_constants(0.0, 1500.0, 1e4, dnu, 18.0, 1.0, 296.0, 1.0)
        out = np.zeros(g)

        def step():
            out[:] = 0.0
            m.transfer_freq(freq, np.zeros(g))
            m.transfer_vectors(h["elow"], h["nu"], h["aif"], h["gns"], h["gamma"], h["n"])
            m.execute(g, n, 0, 1500.0, 1.0, 1e4)
            m.transfer_results(None, out, 0)

        step()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            step()
    finally:
        m.close()
    path = str(tmp_path / "trace.json")
    p.export_chrome_trace(path)
    with open(path) as f:
        ev = [e for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel"]
    main = {e["args"]["stream"]: e for e in ev if "voigt_ws_kernel" in e["name"]}
    core = {e["args"]["stream"]: e for e in ev if "core_kernel" in e["name"]}
    streams = sorted(main)               # one per segment, created in order
    assert len(streams) >= 3 and streams == sorted(core)
    before, last = core[streams[-2]], main[streams[-1]]
    assert before["ts"] + before["dur"] <= last["ts"] + 20.0, \
        (before["ts"] - last["ts"], before["dur"])

    one = torch.zeros(g, dtype=torch.float64, device="cuda")
    job = Job(LineList(d["nu"], d["elow"], d["aif"], d["gns"], d["gamma"], d["n"]), one,
              convention=capi.CONV_REF_GPU, profile=capi.VOIGT, temperature=1500.0, pressure=1.0,
              partition=1e4, mass=18.0, nu_start=lo, dnu=dnu, grid_points=g,
              precision=capi.FP32)
    ctx = Context(0)                     # untuned: the manager's launch shape
    ctx.run([job])
    ctx.check()
    assert np.array_equal(one.cpu().numpy().view(np.int64), out.view(np.int64))
