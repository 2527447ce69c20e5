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


def test_setup_beside_a_capture_of_another_thread(N):
    """A context is set up and solved on one thread while another captures a stream of its own (as a
    server does when it opens): neither call disturbs the other."""
    import threading
    torch = pytest.importorskip("torch")
    from dsmc_suite_b200 import Context
    ico = N.Icosphere(3)
    problem = N.params_config(N.RUNNER_BALLISTIC), N.SurfaceInputs(ico=ico, face_T=ico.face_temperature())
    x = torch.zeros(4, device="cuda")
    got = []
    with Context(0) as ctx:
        want = ctx.solve(N.PATH_FAST_FP32, *problem, 500)["density"]

        def solve():
            try:
                got.append(ctx.solve(N.PATH_FAST_FP32, *problem, 500)["density"])
            except Exception as e:   # the assertion below shows it
                got.append(e)

        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode="thread_local"):
            x.add_(1)
            t = threading.Thread(target=solve)
            t.start()
            t.join()
            x.add_(1)
        graph.replay()
        torch.cuda.synchronize()
    assert isinstance(got[0], np.ndarray), got[0]
    assert np.array_equal(got[0], want) and x.tolist() == [2.0] * 4
