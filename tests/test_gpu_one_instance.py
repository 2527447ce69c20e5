"""A solve of one instance against the kernels of the served queue (needs a B200).

A solve in the default launch shape runs loops that take the instance with the launch, start few
particles on a lane spread, switch to the loops for few particles below a particle count and pack
the live slots once the queue is empty; a 256-thread shape runs the general loops of the served queue over
descriptors in device memory. A particle's trajectory, random stream and deposits are functions of
its id alone, so both give the same grids, rows and counters bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import cold_T

pytestmark = pytest.mark.gpu

BODIES = {"ceres": (470e3, 6.26e10), "moon": (1737e3, 4.90e12)}
# edges of a warp, of one warp per scheduler, of the ranges of the loops for few particles and of the
# slots (640 per SM), on a GPU of 148 SMs
SIZES = [1, 33, 593, 18_944, 18_945, 59_200, 59_201, 94_719, 94_721, 200_003]


def _problem(N, kind):
    if kind == "reference":
        p = N.params_reference(N.RUNNER_BALLISTIC, 36, 72)
        return p, N.SurfaceInputs(T_map=cold_T(N))
    R, GM = BODIES[kind.split("_")[0]]
    p = N.params_config(N.RUNNER_BALLISTIC, R, GM, 41, 77)
    if kind.endswith("_hist"):
        p.n_speed_bins = 24
        p.speed_bin_width = 40.0
    if kind.endswith("_cap"):   # the hop cap below the life cap: the general loop
        p.hop_step_cap = 111
    ico = N.Icosphere(3)
    return p, N.SurfaceInputs(ico=ico, face_T=ico.face_temperature())


@pytest.mark.parametrize("kind,n", [(k, n) for k in ("ceres", "moon") for n in SIZES] +
                         [(k, n) for k in ("ceres_hist", "ceres_cap") for n in (33, 94_721)] +
                         [("reference", n) for n in (33, 5_000)])
def test_one_instance_equals_served_kernels(N, kind, n):
    from dsmc_suite_b200 import Context
    p, S = _problem(N, kind)
    res = []
    for shape in (None, (256, 2, 3000, 2)):
        with Context(0) as ctx:
            if shape:
                ctx.set_launch_shape(*shape)
            r = ctx.solve(N.PATH_FAST_FP32, p, S, n, outputs=True)
            if p.n_speed_bins:
                r["hist"] = ctx.speed_hist()
            res.append(r)
    a, b = res
    assert a["stats"] == b["stats"] and a["stats"]["n_finished"] == n
    for key in a:
        if key != "stats":
            assert np.array_equal(a[key], b[key]), key


@pytest.fixture(scope="module")
def collisional(N):
    """The config model's collisional problem, and the reference model's with every third cell's fit
    invalid (a path integral then passes its threshold where no collision can follow)."""
    from dsmc_suite_b200 import Context
    from dsmc_suite_b200 import workloads as W
    with Context(0) as ctx:
        P = W.collisional_problem(ctx, "col", *BODIES["ceres"], 50, 7, W.sun_vector(0.0), 235.0, 50_000, 0)
    c = P.collision
    valid = c.valid.copy()
    valid[::3] = 0
    q = N.params_reference(N.RUNNER_ADVANCED, 36, 72)
    q.lifetime /= 60.0
    q.wdecay = float(np.exp(-q.dt_step / q.lifetime))
    n_bg = np.full(q.ncell, 2e13)
    n_bg[1::7] = -1.0
    ref = N.CollisionInputs(n_bg, c.coef, c.box, c.total, valid, c.struct.cdf_degree)
    return {"config": (P.params, P.surface, c), "reference": (q, N.SurfaceInputs(T_map=cold_T(N)), ref)}


@pytest.mark.parametrize("kind,n", [("config", 33), ("config", 2001), ("config", 59_200), ("config", 59_201),
                                    ("reference", 33), ("reference", 400)])
def test_collisions_equal_served_kernels(N, collisional, kind, n):
    from dsmc_suite_b200 import Context
    p, S, col = collisional[kind]
    res = []
    for shape in (None, (256, 2, 3000, 2)):
        with Context(0) as ctx:
            if shape:
                ctx.set_launch_shape(*shape)
            res.append(ctx.solve(N.PATH_FAST_FP32, p, S, n, collision=col, outputs=True))
    a, b = res
    assert a["stats"] == b["stats"] and a["stats"]["n_collisions"] > 0
    for key in a:
        if key != "stats":
            assert np.array_equal(a[key], b[key]), key


def test_particle_without_a_position(N):
    """Two particles of one stream draw an infinite launch speed (an FP32 uniform of exactly 1),
    one at its first launch, one after 23 hops: from then on each deposits its weight into the cell
    it launched from until its life cap. The first has unit weight, so its deposit is known; the
    second is compared with the general loop, which steps such a particle like any other."""
    from dsmc_suite_b200 import Context
    R, GM = BODIES["moon"]
    p = N.params_config(N.RUNNER_BALLISTIC, R, GM, 50, 20261203)
    ico = N.Icosphere(3)
    S = N.SurfaceInputs(ico=ico, face_T=ico.face_temperature())

    def one(pid, hop_cap):
        q = p.copy()
        q.hop_step_cap = hop_cap
        with Context(0) as ctx:
            ctx.setup(q, S)
            ctx.enable_particle_outputs(1)
            ctx.run(N.PATH_FAST_FP32, pid, 1)
            ctx.sync()
            ttime, _, steps = ctx.particle_outputs(1)
            assert np.isnan(ttime[1, 0]) and steps[0] == 20_000
            return ctx.density(), ttime[3, 0]

    d, w = one(287_594, 20_000)
    assert w == 1.0 and d[0, 22, 48] == 20_000 << 24 and np.count_nonzero(d) == 1
    a, wa = one(200_964, 20_000)
    b, wb = one(200_964, 19_999)   # a hop cap below the life cap: the general loop
    assert wa == wb < 1.0 and np.array_equal(a, b)
