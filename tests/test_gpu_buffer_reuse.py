"""Device buffers that a context keeps from one call for the next (needs a B200).

A set-up takes over the blocks of the problem before it, and the synchronous calls share one
scratch block; every call clears or fills what it reads. Problems of other sizes, models and tables
in turn on one context give what each gives on a fresh context."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import cold_T

pytestmark = pytest.mark.gpu


def test_one_context_through_unlike_calls_equals_fresh_contexts(N):
    from dsmc_suite_b200 import Context
    from dsmc_suite_b200 import workloads as W
    ico = N.Icosphere(3)
    S = N.SurfaceInputs(ico=ico, face_T=ico.face_temperature())
    spot, facet = W.cratered_mesh(3, depth=0.3)
    normal = N.mesh_normals(spot, facet)["normal"]
    rng = np.random.default_rng(1)
    hist = rng.integers(0, 50, size=(3000, 40)).astype(np.uint64)

    def config(hd, bins, n, path, rows):
        def call(ctx):
            p = N.params_config(N.RUNNER_BALLISTIC, hd=hd)
            p.n_speed_bins = bins
            r = ctx.solve(path, p, S, n, outputs=rows)
            return [r["density"], r["horizon"], list(r["stats"].values())] + (
                [r["ttime"], r["fate"], r["steps"]] if rows else []) + ([ctx.speed_hist()] if bins else [])
        return call

    def reference(ctx):
        p = N.params_reference(N.RUNNER_BALLISTIC, 36, 72)
        r = ctx.solve(N.PATH_FAST_FP32, p, N.SurfaceInputs(T_map=cold_T(N)), 300, outputs=True)
        return [r["density"], r["horizon"], r["ttime"], *ctx.velocity_record(200, per_bucket=5)]

    def push(ctx):
        ctx.setup(N.params_config(N.RUNNER_BALLISTIC), S)
        return ctx.push(N.PATH_PLAIN_FP64, np.full((50, 3), 3e5), np.full((50, 3), 10.0), 40)

    calls = [config(50, 0, 2000, N.PATH_FAST_FP32, True), config(9, 16, 500, N.PATH_PLAIN_FP64, False), reference,
             lambda ctx: ctx.fit_hist(hist, 25.0, 6), config(60, 64, 300, N.PATH_FAST_FP64, True), push,
             lambda ctx: ctx.thermal(7, 11), lambda ctx: [ctx.shadow_flux(spot, facet, normal, 0.3, 3, 9)],
             config(50, 0, 2000, N.PATH_FAST_FP32, True), reference, lambda ctx: ctx.fit_hist(hist[:70], 25.0, 4)]
    with Context(0) as ctx:
        together = [call(ctx) for call in calls]
    for call, got in zip(calls, together):
        with Context(0) as ctx:
            alone = call(ctx)
        assert len(alone) == len(got)
        for a, b in zip(alone, got):
            np.testing.assert_array_equal(np.asarray(a), np.asarray(b))
