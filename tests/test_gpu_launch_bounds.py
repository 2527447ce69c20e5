"""What one launch of a solve takes on (needs a B200).

A launch advances a particle by the launch shape's steps (the step loops' 8 or 12 unrolled ones where
the shape asks for fewer), however long the life is, so that no launch runs for longer than the
caller's shape says."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 500, 8192])
def test_particle_without_a_position_takes_a_launch_at_a_time(N, K):
    """The first particle of test_particle_without_a_position: it deposits its weight into one cell
    until its life cap, here 20,000 steps, over as many launches as other particles would take."""
    from dsmc_suite_b200 import Context
    p = N.params_config(N.RUNNER_BALLISTIC, 1737e3, 4.90e12, 50, 20261203)
    ico = N.Icosphere(3)
    with Context(0) as ctx:
        ctx.set_launch_shape(128, 0, K, 1)
        ctx.setup(p, N.SurfaceInputs(ico=ico, face_T=ico.face_temperature()))
        ctx.enable_particle_outputs(1)
        ctx.run(N.PATH_FAST_FP32, 287_594, 1)
        ctx.sync()
        d = ctx.density()
        _, fate, steps = ctx.particle_outputs(1)
        assert d[0, 22, 48] == 20_000 << 24 and np.count_nonzero(d) == 1
        assert fate[0] == N.FATE_STEP_CAP and steps[0] == 20_000 == ctx.stats()["total_steps"]
        assert ctx.launch_info()[0] >= 20_000 // max(K, 12)
