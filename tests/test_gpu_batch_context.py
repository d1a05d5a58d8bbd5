"""A batch keeps its context: dropping the caller's own reference first leaves
the batch usable, and its destruction touches no freed context."""
import gc
import weakref

import pytest
import torch

from gexs_b200 import Context, Job, LineList, _capi as capi
from gexs_b200.engine import Batch

pytestmark = pytest.mark.gpu


def test_batch_outlives_the_callers_context(small_lines):
    ctx = Context(0)
    out = torch.zeros(2000, dtype=torch.float64, device="cuda")
    job = Job(LineList.from_dict(small_lines), out, convention=capi.CONV_PHYSICAL,
              profile=capi.VOIGT, temperature=900.0, pressure=1.0, partition=1e3, mass=18.0,
              nu_start=1000.0, dnu=0.01, grid_points=2000, precision=capi.FP32, cutoff=25.0)
    batch = Batch(ctx, [job])
    alive = weakref.ref(ctx)
    del ctx
    gc.collect()
    assert alive() is not None
    batch.launch()
    alive().check()
    assert float(out.max()) > 0.0
    del batch
    gc.collect()
    assert alive() is None
