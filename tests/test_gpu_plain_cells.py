"""PLAIN_FP64's cell limits at the sizes where they can go wrong (needs a B200).

Most steps of the plain path keep the last cell while the position is well inside its limits and
evaluate the reference's index formulas (asin, atan2, log) otherwise; the oracle evaluates them on
every step. Grids, fates and step counts are compared exactly for grids of one and two columns or
rows (limits that never hold, half-plane columns), of many thin shells, uniform and exponential,
and for an inconsistent shell constant, which the formulas define and the limits must follow. The
velocity record is compared with a per-bucket cap of a few records, where most particles have
none."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import cold_T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ftd,ffd,hd,exp_grid,log1p_scale", [
    (36, 72, 50, 1, 1.0), (1, 1, 3, 1, 1.0), (2, 2, 5, 0, 1.0), (1, 3, 400, 0, 1.0), (255, 255, 120, 1, 1.0),
    (36, 72, 50, 1, 0.5), (7, 5, 40, 1, -1.0)])
def test_plain_cells_match_the_formulas(ctx, N, O, ftd, ffd, hd, exp_grid, log1p_scale):
    p = N.params_config(N.RUNNER_BALLISTIC, hd=hd)
    p.ftd, p.ffd, p.use_exp_grid = ftd, ffd, exp_grid
    if not exp_grid:
        p.unih = 0.3 * p.Radii / hd   # the top shells end below the escape radius
    p.log1p_alpha2 *= log1p_scale
    ico = N.Icosphere(3)
    S = N.SurfaceInputs(ico=ico, face_T=ico.face_temperature())
    n = 300
    g = ctx.solve(N.PATH_PLAIN_FP64, p, S, n, outputs=True)
    o = O.run(p, S, n, nthreads=4)
    assert np.array_equal(g["fate"], o["fate"]) and np.array_equal(g["steps"], o["steps"])
    assert np.array_equal(g["density"].ravel(), np.asarray(o["density"]).ravel())
    assert np.array_equal(g["horizon"].ravel(), np.asarray(o["horizon"]).ravel())


@pytest.mark.parametrize("per_bucket,total_cap", [(1, 50_000), (3, 50_000), (3, 100)])
def test_velocity_record_with_few_records_per_bucket(ctx, N, O, per_bucket, total_cap):
    p = N.params_reference(N.RUNNER_BALLISTIC, 36, 72)
    S = N.SurfaceInputs(T_map=cold_T(N))
    n = 120
    ctx.setup(p, S)
    full = ctx.velocity_record(n, per_bucket=200, total_cap=1_000_000)
    few = ctx.velocity_record(n, per_bucket=per_bucket, total_cap=total_cap)
    # the first per_bucket records of every (td, ht) bucket, in the record's own order
    seen, keep = {}, []
    for k in range(len(full[0])):
        b = (int(full[1][k]), int(full[3][k]))
        seen[b] = seen.get(b, 0) + 1
        if seen[b] <= per_bucket:
            keep.append(k)
    keep = keep[:total_cap]
    for a, b in zip(few, full):
        assert np.array_equal(a, b[keep])


def test_velocity_record_of_buckets_with_more_than_two_to_the_31_visits(ctx, N):
    """The first records of a bucket stay its first, however often particles come back to it."""
    p = N.params_reference(N.RUNNER_BALLISTIC, 6, 12)
    p.hd, p.unih = 1, p.max_height - p.Radii
    S = N.SurfaceInputs(T_map=N.latlon_temperature(6, 12, T_ss=235.0, T_floor=150.0))
    p.n_speed_bins, p.speed_bin_width = 1, 1e6   # one bin: the deposits of each cell
    n = 2_000_000
    ctx.solve(N.PATH_PLAIN_FP64, p, S, n)
    assert ctx.speed_hist().reshape(6, 12).sum(1).max() > 2**31
    p.n_speed_bins = 0
    ctx.setup(p, S)
    few, many = (ctx.velocity_record(m, per_bucket=4) for m in (2000, n))
    assert len(few[0]) == 6 * 4
    for a, b in zip(few, many):
        assert np.array_equal(a, b)
