"""The loops of a solve in launch shapes and sizes that the default shape does not reach (needs a B200).

A trajectory, its random stream and its deposits are functions of the particle's id, so every shape and
every split of the ids gives the same grids, rows and counters bit for bit. The shapes cut launches in
the middle of a hop and of an unrolled block of steps (steps per launch below 8 and 12, and no multiple
of them), with 4 and 5 blocks per SM; the sizes put the reference model's loops above the few particles
per SM where the loops for few take over. Each is compared with the general loop of the served queue."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import cold_T

pytestmark = pytest.mark.gpu

GENERAL = (256, 2, 3000, 2)


def _same(a, b):
    assert a["stats"] == b["stats"]
    for key in a:
        if key != "stats":
            assert np.array_equal(a[key], b[key]), key


def _solve(N, shape, path, p, S, n, col=None):
    from dsmc_suite_b200 import Context
    with Context(0) as ctx:
        if shape:
            ctx.set_launch_shape(*shape)
        r = ctx.solve(path, p, S, n, collision=col, outputs=True)
        if p.n_speed_bins:
            r["hist"] = ctx.speed_hist()
        return r


def _config(N, body="ceres"):
    R, GM = {"ceres": (470e3, 6.26e10), "moon": (1737e3, 4.90e12)}[body]
    ico = N.Icosphere(3)
    return N.params_config(N.RUNNER_BALLISTIC, R, GM, 41, 77), N.SurfaceInputs(ico=ico, face_T=ico.face_temperature())


def _reference(N, runner):
    p = N.params_reference(runner, 36, 72)
    p.lifetime /= 60.0
    p.wdecay = float(np.exp(-p.dt_step / p.lifetime))
    return p, N.SurfaceInputs(T_map=cold_T(N))


@pytest.fixture(scope="module")
def fits(N):
    """Collision tables of the config model's pipeline on the 36 x 72 x 50 grid."""
    from dsmc_suite_b200 import Context
    from dsmc_suite_b200 import workloads as W
    with Context(0) as ctx:
        return W.collisional_problem(ctx, "col", 470e3, 6.26e10, 50, 7, W.sun_vector(0.0), 235.0, 50_000, 0)


def _problem(N, fits, kind):
    if kind.endswith(" bins"):   # histograms where the general loop is the only one
        p, S, col = _problem(N, fits, kind[:-5])
        p = p.copy()
        p.n_speed_bins, p.speed_bin_width = 24, 40.0
        return p, S, col
    if kind in ("ceres", "moon"):
        return (*_config(N, kind), None)
    if kind == "hist":
        p, S = _config(N)
        p.n_speed_bins, p.speed_bin_width = 24, 40.0
        return p, S, None
    if kind == "reference":
        return (*_reference(N, N.RUNNER_BALLISTIC), None)
    c = fits.collision
    if kind == "collisions":
        return fits.params, fits.surface, c
    p, S = _reference(N, N.RUNNER_ADVANCED)
    return p, S, N.CollisionInputs(np.full(p.ncell, 2e13), c.coef, c.box, c.total, c.valid, c.struct.cdf_degree)


@pytest.mark.parametrize("kind", ["ceres", "moon", "hist", "reference", "collisions", "reference collisions",
                                  "reference bins", "collisions bins", "reference collisions bins"])
def test_shapes_that_cut_hops_and_blocks_of_steps(N, fits, kind):
    p, S, col = _problem(N, fits, kind)
    n = 300
    want = _solve(N, GENERAL, N.PATH_FAST_FP32, p, S, n, col)
    assert want["stats"]["n_finished"] == n
    for shape in ((128, 0, 8192, 1), (128, 4, 301, 1), (128, 5, 7, 64), (128, 4, 13, 3), (64, 0, 100, 8), (96, 5, 1000, 1)):
        _same(_solve(N, shape, N.PATH_FAST_FP32, p, S, n, col), want)


@pytest.mark.parametrize("kind", ["ceres", "reference", "collisions", "reference collisions", "hist"])
@pytest.mark.parametrize("shape", [None, (128, 4, 1001, 4), (128, 5, 301, 16)])
def test_bulk_loops_equal_the_general_loop(N, fits, kind, shape):
    p, S, col = _problem(N, fits, kind)
    n = 120_000   # 811 per SM: a full start, a refilled queue and a packed tail
    _same(_solve(N, shape, N.PATH_FAST_FP32, p, S, n, col), _solve(N, GENERAL, N.PATH_FAST_FP32, p, S, n, col))


@pytest.mark.parametrize("body", ["ceres", "moon"])
def test_fp64_loops_agree(N, body):
    """FAST_FP64's loops for few and for many particles, at 3, 4 and 5 blocks per SM."""
    p, S = _config(N, body)
    n = 120_000
    want = _solve(N, (128, 3, 8192, 1), N.PATH_FAST_FP64, p, S, n)
    for shape in (None, (128, 4, 1001, 1), (128, 5, 8192, 1)):
        _same(_solve(N, shape, N.PATH_FAST_FP64, p, S, n), want)
    from dsmc_suite_b200 import Context
    with Context(0) as ctx:   # 59,200 are few by the loops' line, 400 per SM; parts of 40,000 more so
        ctx.setup(p, S)
        grids = []
        for k in range(0, n, 40_000):
            ctx.zero()
            ctx.run(N.PATH_FAST_FP64, k, 40_000)
            ctx.sync()
            grids.append(ctx.density())
    assert np.array_equal(sum(grids), want["density"])


def test_contexts_on_two_threads(N):
    """Thermal solves of unlike depths and solves of unlike bodies side by side, a context a thread."""
    from dsmc_suite_b200 import Context
    works = []
    for body, depth, grid in (("ceres", 0.05, (36, 72)), ("moon", 0.02, (12, 24))):
        p, S = _config(N, body)
        tp = N.ThermalParams.default()
        tp.depth = depth
        works.append((p, S, tp, grid))
    got, want = [[], []], []

    def work(k, times, out):
        p, S, tp, grid = works[k]
        try:
            with Context(0) as ctx:
                for _ in range(times):
                    out.append([ctx.thermal(*grid, tp)[0], ctx.solve(N.PATH_FAST_FP32, p, S, 3000)["density"]])
        except Exception as e:   # the comparison below shows it
            out.append(e)

    for k in range(2):
        work(k, 1, want)
    threads = [threading.Thread(target=work, args=(k, 40, got[k])) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert len(got[k]) == 40
        for r in got[k]:
            assert not isinstance(r, Exception), r
            assert all(np.array_equal(a, b) for a, b in zip(r, want[k]))
