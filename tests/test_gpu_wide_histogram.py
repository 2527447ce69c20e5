"""Speed histograms of more than 2^31 entries (needs a B200 and 64 GB of host memory).

255 x 255 x 34 cells of 1024 bins are 2.26e9 entries, 18 GB: every count has to land in its own cell,
as it does in the same solve with 16 bins."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hop_cap", [20_000, 19_999])   # the histogram loop, the general loop
def test_counts_beyond_two_to_the_31_entries(N, hop_cap):
    import psutil
    if psutil.virtual_memory().available < 64 << 30:
        pytest.skip("18 GB of histograms are read back")
    from dsmc_suite_b200 import Context
    ico = N.Icosphere(3)
    S = N.SurfaceInputs(ico=ico, face_T=ico.face_temperature())
    p = N.params_config(N.RUNNER_BALLISTIC, hd=34)
    p.ftd = p.ffd = 255
    p.hop_step_cap = hop_cap
    per_cell = []
    with Context(0) as ctx:
        for bins in (16, 1024):
            p.n_speed_bins, p.speed_bin_width = bins, 1600.0 / bins
            ctx.solve(N.PATH_FAST_FP32, p, S, 2000)
            per_cell.append(ctx.speed_hist().sum(1))
    few, many = per_cell
    assert few[2**31 // 1024:].any()
    np.testing.assert_array_equal(many, few)
