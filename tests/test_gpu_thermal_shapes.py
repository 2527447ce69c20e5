"""The thermal column kernels where their choice and their loops turn (needs a B200).

Both kernels (profiles in shared memory with 8 lanes a column, profiles in device memory with one
thread a column) follow the oracle's FP64 operation order; the bar is the one of the thermal model:
99 % of the cells bit-identical (CUDA's log10 / pow may round the sublimation term differently in
the last place), every cell within 0.02 K. The sizes put the depth at its minimum of 3, at one less
and one more than the read-ahead of 8, and at both sides of the shared-memory limits of 8 and 4
columns a block; the column counts at one, at a part of a block, and past one wave of blocks."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ftd,ffd,n_sub,depth_points", [
    (1, 1, 1, 3), (1, 3, 2, 3), (3, 3, 2, 9), (3, 3, 2, 10), (3, 3, 2, 11), (5, 5, 3, 18), (2, 7, 1, 1520),
    (2, 7, 1, 1540), (2, 7, 1, 2630), (2, 7, 1, 2660), (72, 72, 2, 467), (96, 100, 1, 300)])
def test_thermal_shapes_match_oracle(ctx, N, O, ftd, ffd, n_sub, depth_points):
    tp = N.ThermalParams.default()
    tp.n_substep = n_sub
    dt = 9.07417 * 3600.0 / ffd / n_sub
    dr = np.sqrt(0.1 * 2.0 * dt * tp.conductivity / tp.density / tp.Cp)
    tp.depth = dr * (depth_points - 0.5)
    rng = np.random.default_rng(5)
    flux = rng.uniform(0.0, 200.0, size=(ftd, ffd)) * (rng.random((ftd, ffd)) < 0.7)
    flux.flat[0] = 1e6   # the bracket has to widen
    T, h = ctx.thermal(ftd, ffd, tp, flux)
    To, ho = O.thermal(ftd, ffd, tp, flux)
    assert h == ho == depth_points
    assert np.mean(T == To) >= 0.99, np.mean(T == To)
    assert np.abs(T - To).max() <= 0.02
