"""The library's host code on a fake CUDA runtime (fake_cudart.cpp): which streams, allocations and
attributes a call uses, and what it does when an allocation fails. No kernel runs, so nothing here
looks at results; the GPU tests do."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def fake_lib(built, tmp_path_factory):
    """The built objects linked with the fake runtime, as a library of their own."""
    from dsmc_suite_b200 import _native as N
    from dsmc_suite_b200 import build as B
    so = tmp_path_factory.mktemp("fake") / "libdsmc_fake.so"
    objs = [str(B.OBJ / (s + ".o")) for s in [*B.CUDA_SOURCES, *B.C_SOURCES]]
    # -Bsymbolic: the library's calls go to the fake even where a real runtime is loaded
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include",
                    "-o", str(so), str(ROOT / "tests" / "fake_cudart.cpp"), *objs, "-lm", "-lpthread"],
                   check=True, capture_output=True)
    L = C.CDLL(str(so))
    for name, res, args in N.SIGNATURES:
        f = getattr(L, name)
        f.restype, f.argtypes = res, args
    for name in ("allocs", "loops", "reads", "races", "device_syncs", "lowered"):
        getattr(L, "fake_" + name).restype = C.c_longlong
    L.fake_held.restype = C.c_size_t
    L.fake_stream.restype = C.c_void_p
    L.fake_limit.argtypes = [C.c_size_t]
    L.fake_fail_at.argtypes = L.fake_finish_after.argtypes = [C.c_longlong]
    return L


@pytest.fixture
def fake(fake_lib, N, monkeypatch):
    monkeypatch.setattr(N, "_lib", fake_lib)
    fake_lib.fake_reset()
    return fake_lib


@pytest.fixture
def context(fake):
    from dsmc_suite_b200 import Context
    with Context(0) as c:
        yield c


@pytest.fixture(scope="module")
def problem(N):
    ico = N.Icosphere(2)
    return N.params_config(N.RUNNER_BALLISTIC, hd=20), N.SurfaceInputs(ico=ico, face_T=ico.face_temperature())


def test_rows_are_cleared_after_the_run_that_writes_them(fake, context, N, problem):
    """A plain run is asynchronous; the same rows enabled again on another stream are cleared only
    after it, whether that stream is the context's own or one more of the caller's."""
    context.setup(*problem)
    context.enable_particle_outputs(100)
    for stream in (fake.fake_stream(), None, fake.fake_stream(), fake.fake_stream()):
        context.run(N.PATH_PLAIN_FP64, 0, 100)
        context.set_stream(stream)
        context.enable_particle_outputs(100)
        assert fake.fake_races() == 0


def test_setup_waits_for_its_own_work_alone(fake, context, N, problem):
    """A set-up reuses the blocks of the problem before it once that problem's work has ended, on
    every stream the context was given; it does not wait for the device, which CUDA refuses while
    another thread captures a stream (as a server does when it opens)."""
    from dsmc_suite_b200 import Context
    fake.fake_capturing(1)
    context.setup(*problem)
    for stream in (fake.fake_stream(), fake.fake_stream(), None):
        context.run(N.PATH_PLAIN_FP64, 0, 100)
        context.set_stream(stream)
        before = fake.fake_allocs()
        context.setup(*problem)
        assert fake.fake_allocs() == before and fake.fake_races() == 0
    with Context(0) as other:
        other.setup(*problem)
        other.run(N.PATH_PLAIN_FP64, 0, 100)
        context.setup(*problem)
        assert fake.fake_races() > 0   # the other context's kernel still runs, and is not waited for
    assert fake.fake_device_syncs() == 0


@pytest.mark.parametrize("path", ["PATH_FAST_FP32", "PATH_FAST_FP64"])
def test_a_run_of_no_particles_leaves_no_work_behind(fake, context, N, problem, path):
    """The next set-up, on another stream, takes over the tables that such a run was given."""
    context.setup(*problem)
    context.set_stream(fake.fake_stream())
    context.run(getattr(N, path), 0, 0)
    assert context.launch_info()[0] == 0
    context.set_stream(None)
    context.setup(*problem)
    assert fake.fake_races() == 0


def test_setup_leaves_grids_it_handed_out(fake, context, N, problem):
    """The caller may be reading a grid whose device address it was given, on a stream the context
    does not know: those blocks are freed, which waits for the device, and not written again."""
    context.setup(*problem)
    before = fake.fake_allocs()
    context.setup(*problem)
    assert fake.fake_allocs() == before
    context.density_device()
    context.setup(*problem)
    assert fake.fake_allocs() > before
    before = fake.fake_allocs()
    context.setup(*problem)
    assert fake.fake_allocs() == before


def test_thermal_calls_leave_the_shared_memory_limit_alone(fake, context, N):
    """The limit belongs to the function on the device, not to the call: a call of a shallow column
    on one thread must not lower it between another thread's setting and its launch."""
    from dsmc_suite_b200 import Context
    tp = N.ThermalParams.default()
    with Context(0) as other:
        for ctx, depth in ((context, 0.05), (other, 0.02), (context, 0.12), (other, 0.05)):
            tp.depth = depth
            ctx.thermal(6, 12, tp)
    assert fake.fake_lowered() == 0


@pytest.mark.parametrize("n", [200, 200_000])   # fewer particles than slots, and more
def test_a_solve_after_one_whose_allocation_failed(fake, N, problem, n):
    """Every device allocation of a first solve fails in turn: that call reports it, and the next call
    on the same context solves as a first one does."""
    from dsmc_suite_b200 import Context
    for path in (N.PATH_FAST_FP32, N.PATH_FAST_FP64):
        failed = 0
        for k in range(64):
            with Context(0) as ctx:
                ctx.setup(*problem)
                fake.fake_fail_at(k)
                fake.fake_finish_after(2)
                status = N.lib().dsmc_run(ctx.h, path, 0, n)
                fake.fake_fail_at(-1)
                if status == 0:
                    break
                assert status == -4
                failed += 1
                fake.fake_finish_after(2)
                ctx.run(path, 0, n)
        assert failed >= 3   # slots, counters, tables


def test_large_thermal_solves_keep_their_device_block(fake, context, N):
    """A thermal solve above the 256 MB that every call's scratch is kept up to allocates once per
    context, also with other calls between."""
    tp = N.ThermalParams.default()
    tp.n_substep, tp.depth = 8, 0.1
    h = context.thermal(120, 180, tp)[1]
    assert 120 * 180 * h * 16 > 256 << 20
    before, held = fake.fake_allocs(), fake.fake_held()
    for k in range(3):
        context.thermal(120, 180, tp)
        context.fit_hist(np.ones((50, 8), dtype=np.uint64), 25.0, 3)
        context.thermal(7, 9)
    assert fake.fake_allocs() == before and fake.fake_held() == held


@pytest.mark.parametrize("call", ["rows", "solve", "solve64", "setup", "fit", "record"])
def test_kept_blocks_make_room_when_memory_is_short(fake, N, problem, call):
    """A context that keeps spare blocks and scratch gives them back before a call of its own fails for
    want of the memory that they hold."""
    from dsmc_suite_b200 import Context
    p, surface = problem
    wide = p.copy()
    wide.n_speed_bins = 200   # 83 MB of histograms
    with Context(0) as ctx:
        ctx.setup(wide, surface)
        ctx.setup(p, surface)                                        # the histograms' block is spare
        ctx.fit_hist(np.ones((400_000, 60), dtype=np.uint64), 25.0, 3)   # 230 MB of scratch
        do = {
            "rows": lambda: ctx.enable_particle_outputs(3_000_000),                    # 252 MB
            "solve": lambda: ctx.run(N.PATH_FAST_FP32, 0, 100),                        # 14 MB
            "solve64": lambda: ctx.run(N.PATH_FAST_FP64, 0, 100),
            "setup": lambda: (setattr(wide, "n_speed_bins", 600), ctx.setup(wide, surface)),  # 249 MB
            "record": lambda: ctx.velocity_record(200_000, per_bucket=2),   # 256 MB of rows, or 64 MB at a time
            "fit": lambda: ctx.fit_hist(np.ones((500_000, 60), dtype=np.uint64), 25.0, 3),    # 294 MB
        }[call]
        assert fake.fake_held() > 300_000_000
        fake.fake_limit(fake.fake_held() + (1 << 20) - (250_000_000 if call == "record" else 0))
        do()


def test_a_setup_takes_over_blocks_of_about_its_size(fake, context, N, problem):
    """A block of an earlier problem that is taken over may be larger than asked for, by 16 MB at most."""
    p, surface = problem
    wide = p.copy()
    cells = p.hd * p.ftd * p.ffd
    for bins in (200, 150, 130, 60, 58):
        wide.n_speed_bins = bins
        context.setup(wide, surface)
        spare = fake.fake_held()
        context.setup(wide, surface)      # the spare blocks too large for it stay spare, within their bound
        assert fake.fake_held() == spare
        fake.fake_limit(fake.fake_held())
        with pytest.raises(N.DsmcError):  # gives every spare block back, and fails
            context.enable_particle_outputs(10_000_000)
        fake.fake_limit(1 << 36)
        assert fake.fake_held() < cells * (bins + 2) * 8 + (20 << 20)


def test_a_solve_too_large_for_the_memory_is_refused_once(fake, context, N, problem):
    """With nothing left to give back the call reports the lack of memory, and does so without a
    launch."""
    context.setup(*problem)
    fake.fake_limit(fake.fake_held() + (1 << 20))
    assert N.lib().dsmc_run(context.h, N.PATH_FAST_FP32, 0, 100) == -4
    assert fake.fake_loops() == 0
    with pytest.raises(N.DsmcError):
        context.enable_particle_outputs(1_000_000)


@pytest.mark.parametrize("K,G,group", [(64, 16, 16), (1024, 8, 8), (1024, 100, 8), (8192, 8, 1), (100_000, 8, 1), (64, 1, 1)])
def test_short_launches_are_issued_in_groups(fake, context, N, problem, K, G, group):
    """A solve looks at its counters once for every launches_per_graph launches, but no later than after
    the 8192 steps of the default launch; the default shape looks after each launch."""
    context.set_launch_shape(128, 5, K, G)
    context.setup(*problem)
    for n in (100, 1_000_000):   # fewer particles than slots, and more
        fake.fake_reset()
        fake.fake_finish_after(6 * group)
        context.run(N.PATH_FAST_FP32, 0, n)
        rounds = fake.fake_reads()
        assert 6 <= rounds <= 7 and fake.fake_loops() == group * rounds == context.launch_info()[0]


def test_thermal_grids_up_to_the_limit(fake, context, N):
    """Inputs, profiles and results of 2^30 doubles are accepted: 3 ncol + 2 h + 2 ncol h, to the depth."""
    tp = N.ThermalParams.default()
    tp.n_substep = 1
    dr = np.sqrt(0.1 * 2.0 * (9.07417 * 3600.0 / 100) * tp.conductivity / tp.density / tp.Cp)
    most = (2**30 - 3 * 1000) // (2 + 2 * 1000)
    tp.depth = dr * (most - 0.5)
    assert context.thermal(10, 100, tp)[1] == most
    tp.depth = dr * (most + 0.5)
    with pytest.raises(N.DsmcError, match="too large"):
        context.thermal(10, 100, tp)


def test_shadow_flux_without_threads(built, tmp_path):
    """Subtrees of a mesh are built on threads of their own from 2000 triangles on, where there are any to
    be had; a process that can make none gets its flux all the same."""
    from dsmc_suite_b200 import build as B
    exe = tmp_path / "no_threads"
    objs = [str(B.OBJ / (s + ".o")) for s in [*B.CUDA_SOURCES, *B.C_SOURCES]]
    subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", f"-I{ROOT / 'include'}", "-o", str(exe),
                    str(ROOT / "tests" / "no_threads.cpp"), str(ROOT / "tests" / "fake_cudart.cpp"), *objs, "-lm", "-lpthread"],
                   check=True, capture_output=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
