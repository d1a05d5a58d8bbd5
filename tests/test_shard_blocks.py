"""Line ranges of shards begin at multiples of the block of lines that the FP64
form sums, and FP64 shards computed from them have the bits of the unsplit
cross-section (one GPU, one shard after another)."""
import numpy as np
import pytest

from gexs_b200 import shard


def test_ranges_begin_at_line_blocks():
    nu = np.sort(np.random.default_rng(3).exponential(4000.0, 60000) + 100.0)
    seen = 0
    for world in (2, 3, 8):
        b, lo, hi = shard.plan(nu, 100.0, 0.01, 0, 2990001, 25.0, world)
        assert np.all(lo % 512 == 0)
        for r in range(world):
            a, c = shard.line_range(nu, 100.0, 0.01, int(b[r]), int(b[r + 1] - b[r]), 25.0)
            assert a % 512 == 0 and a <= lo[r] + 512 and c >= hi[r]
            seen += lo[r] > 0
    assert seen > 0


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["plan", "line_range"])
def test_fp64_shards_have_the_bits_of_one_launch(gpu_ctx, how):
    import torch
    from gexs_b200 import Job, LineList, synth, _capi as capi
    st = synth.make_states(5000, 40, 81)
    L = synth.make_lines(st, 60000, 2000.0, 2400.0, 82, broadening_seed=83)
    g, lo, dnu, cut = 40001, 2000.0, 0.01, 25.0
    b, los, his = shard.plan(L["nu"], lo, dnu, 0, g, cut + 1.0, 3)

    def run(profile, part, a, n, out):
        j = Job(LineList.from_dict(part), out, convention=capi.CONV_PHYSICAL, profile=profile,
                temperature=1500.0, pressure=0.3, partition=1e3, mass=18.0, nu_start=lo, dnu=dnu,
                grid_points=g, start_idx=a, n_points=n, precision=capi.FP64, cutoff=cut)
        gpu_ctx.run([j])
        gpu_ctx.check()

    for profile in (capi.VOIGT, capi.VOIGT_QUAD, capi.DOPPLER):
        whole, parts = (torch.zeros(g, dtype=torch.float64, device="cuda") for _ in range(2))
        run(profile, L, 0, g, whole)
        for r in range(3):
            a, n = int(b[r]), int(b[r + 1] - b[r])
            l0, l1 = (int(los[r]), int(his[r])) if how == "plan" else \
                shard.line_range(L["nu"], lo, dnu, a, n, cut)
            run(profile, {k: np.ascontiguousarray(v[l0:l1]) for k, v in L.items()}, a, n, parts)
        assert float(whole.max()) > 0.0
        bad = int((whole.view(torch.int64) != parts.view(torch.int64)).sum())
        assert bad == 0, (profile, bad)
