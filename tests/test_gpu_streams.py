"""One context on several streams (needs a B200).

Asynchronous work stays on the stream it was issued on; what a later call takes over on another stream
(the rows, the grids, the tables of a set-up) it takes over after that work."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_rows_enabled_on_another_stream_are_clear(N):
    torch = pytest.importorskip("torch")
    from dsmc_suite_b200 import Context
    n = 20_000
    ico = N.Icosphere(3)
    streams = [torch.cuda.Stream() for _ in range(2)]
    with Context(0) as ctx:
        ctx.setup(N.params_config(N.RUNNER_BALLISTIC), N.SurfaceInputs(ico=ico, face_T=ico.face_temperature()))
        ctx.enable_particle_outputs(n)
        for k in range(4):
            ctx.set_stream(streams[k % 2].cuda_stream)
            ctx.run(N.PATH_PLAIN_FP64, 0, n)              # tens of milliseconds, not waited for
            ctx.set_stream(streams[1 - k % 2].cuda_stream if k < 3 else None)
            ctx.enable_particle_outputs(n)
            torch.cuda.synchronize()
            ttime, fate, steps = ctx.particle_outputs(n)
            assert not ttime.any() and not fate.any() and not steps.any()
