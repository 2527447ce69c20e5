"""The eight lanes of a column of the thermal kernel read and overwrite one shared profile.

The kernel's source is compiled for the host with every lane a fiber (thermal_lanes.cpp) and run with
each lane taken to its next warp-wide call before the next lane starts, first to last and last to
first. CUDA orders the lanes of a warp no further than that, so the result has to be that of the
kernel with one lane a column, bit for bit: both do the same operations on the same values."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lanes(tmp_path_factory):
    d = tmp_path_factory.mktemp("thermal_lanes")
    src = (ROOT / "dsmc_suite_b200" / "csrc" / "kernel_thermal.cu").read_text()
    head, tail = src.split("cudaError_t launch_thermal(")
    assert tail and '#include "dsmc_kernels.h"' in head
    (d / "thermal_lanes.inc").write_text(head.replace('#include "dsmc_kernels.h"', "") + "\n}\n")
    so = d / "thermal_lanes.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{d}", "-o", str(so),
                    str(ROOT / "tests" / "thermal_lanes.cpp")], check=True, capture_output=True)
    f = C.CDLL(str(so)).thermal_lanes
    f.restype = C.c_int
    return f


@pytest.mark.parametrize("h", [3, 4, 9, 10, 11, 40])
@pytest.mark.parametrize("ncol", [1, 4, 6])
def test_lanes_of_a_column_in_any_order(lanes, N, h, ncol):
    tp = N.ThermalParams.default()
    R, dr, n_sub = 0.05, 2e-4, 3
    cp, piv = np.zeros(h), np.ones(h)
    for i in range(1, h):
        a, b, c = (-R, 1 + 2 * R, -R) if i < h - 1 else (-1 / dr, 1 / dr, 0.0)
        piv[i] = b - a * cp[i - 1]
        cp[i] = c / piv[i]
    flux = np.linspace(0.0, 180.0, ncol)
    T_init = np.where(flux > 0, (flux / 5.6704e-8) ** 0.25, 100.0)
    ptr = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))
    vec = lambda *x: np.ascontiguousarray(x, dtype=np.float64)
    p, LH = vec(*tp.p_mat), vec(*tp.LH_mat)
    consts = vec(tp.tran_unit_p, tp.tran_unit_LH, 18e-3 / 6.02e23)
    rcp = 1.0 / piv

    def run(shared, reverse):
        out = np.zeros(ncol)
        assert lanes(shared, reverse, ncol, h, n_sub, C.c_double(R), C.c_double(6e-4 / dr), C.c_double(-1 / dr),
                     ptr(p), ptr(LH), ptr(consts), ptr(flux), ptr(T_init), ptr(cp), ptr(piv), ptr(rcp), ptr(out)) == 0
        return out

    want = run(0, 0)
    assert np.all(np.isfinite(want)) and np.array_equal(run(0, 1), want)
    assert np.array_equal(run(1, 0), want)
    assert np.array_equal(run(1, 1), want)
