"""The library's host code without a GPU: its objects linked with a runtime that
looks at launches instead of running them (fake_cuda/runtime.cu).  Layouts,
tuner trials and scratch of the solves are held against the buffers that the
launches get, and a solve leaves its number where it would write."""
import ctypes
import glob
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

import cupic_gb300 as cg
from cupic_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="session")
def fake_path(tmp_path_factory):
    build.build()
    out = tmp_path_factory.mktemp("fake")
    obj, lib = str(out / "runtime.o"), str(out / "libcupic_fake.so")
    subprocess.run([build.nvcc()] + build.common_flags() + ["-I", build.CSRC, "-D__CUDA_DEVICE_RUNTIME_API_H__", "-c",
                   os.path.join(HERE, "fake_cuda", "runtime.cu"), "-o", obj], check=True)
    objs = [os.path.join(build.OUT, os.path.splitext(s)[0] + ".o") for s in build.SOURCES]
    subprocess.run(["g++", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-o", lib, obj,
                    os.path.join(HERE, "fake_cuda", "new.cpp")] + objs + ["-lpthread"], check=True)
    return lib


@pytest.fixture
def fake(fake_path, monkeypatch):
    """cupic_gb300 on a library of its own on that runtime (nothing tuned yet)."""
    copy = fake_path + f".{len(glob.glob(fake_path + '*'))}"
    shutil.copyfile(fake_path, copy)  # one handle each
    for name in ("CTAS", "DEPTH", "TUNE", "NOSTRIP", "SCALAR"):
        monkeypatch.delenv("CUPIC_JACOBI_" + name, raising=False)
    monkeypatch.setattr(cg, "_LIB", None)
    monkeypatch.setattr(cg, "library_path", lambda: copy)
    L = cg.load_library()
    L.fake_allocated.restype = ctypes.c_uint64
    L.fake_raise.restype = ctypes.c_uint64
    L.fake_raise.argtypes = [ctypes.c_uint64]
    return L


def faults(L):
    text = ctypes.create_string_buffer(1 << 16)
    L.fake_faults(text, len(text))
    return text.value.decode().splitlines()


def params(ncx, ncy, **over):
    return cg.workload_params("tiny", ncx=ncx, ncy=ncy, n=2.0, **over)


def test_raised_shared_memory_counts_the_static_part(fake):
    """48 KB without an opt-in are static and dynamic shared memory together: a
    kernel's dynamic part is raised from there on, not from 48 KB on, and never
    lowered again."""
    for n in (1000, 48 * 1024 - 720, 48 * 1024 - 719, 48 * 1024, 100000):
        assert fake.fake_raise(n) >= n
    # rows of 200 cells take 48,768 bytes of the push, beside its static 640
    with cg.Sim(params(200, 40)) as sim:
        sim.init_plasma()
        sim.step(2)
    assert faults(fake) == []


def two_columns(p, value=0.5):
    """A potential whose columns 0 and nnx-1 differ."""
    phi = np.full((p.nny, p.nnx), 1.25)
    phi[1:-1, -1] += value
    return phi


MESHES = [(256, 1024), (300, 700), (128, 512), (200, 300), (512, 512), (512, 2048), (64, 90), (3, 5)]


@pytest.mark.parametrize("ncx,ncy", MESHES)
def test_two_seam_columns_keep_launches_inside_their_buffers(fake, ncx, ncy):
    """A potential with two different columns at the seam takes the precision form
    off the register tiles: the launches timed and made after that are of their
    own layout, in scratch of that layout."""
    p = params(ncx, ncy, refine_every=32, max_sweeps=320)
    with cg.Sim(p) as sim:
        sim.init_plasma()
        assert faults(fake) == []
        sim.set_phi(two_columns(p))
        assert faults(fake) == []
        sim.poisson_solver(1e-9, 1, 320, 32)
        sim.step(2)
        assert fake.fake_launches(b"k_jacobi") > 0
        assert faults(fake) == []


@pytest.mark.parametrize("ncx,ncy", MESHES)
def test_two_seam_columns_change_the_potential_alone(fake, ncx, ncy):
    """The tuner's trials after such a potential leave the field, the report and
    the potential just set alone."""
    p = params(ncx, ncy, refine_every=32, max_sweeps=320)
    with cg.Sim(p) as sim:
        sim.init_plasma()
        sim.poisson_solver(1e-9, 1, 320, 32)
        field = sim.efield()
        phi = two_columns(p)
        sim.set_phi(phi)
        np.testing.assert_array_equal(sim.phi64(), phi)
        np.testing.assert_array_equal(sim.phi(), phi.astype(np.float32))
        for g, o in zip(sim.efield(), field):
            np.testing.assert_array_equal(g, o)
        assert faults(fake) == []


@pytest.mark.parametrize("back", ("set_phi", "init_plasma", "init_mesh"))
@pytest.mark.parametrize("ctas", (None, "5"))
def test_equal_seam_columns_bring_the_tiles_back(fake, monkeypatch, back, ctas):
    """Once the columns at the seam are equal again the solves are tiles again, in
    the layout of before and without a trial."""
    if ctas:
        monkeypatch.setenv("CUPIC_JACOBI_CTAS", ctas)
    p = params(64, 90, refine_every=32, max_sweeps=320)
    with cg.Sim(p) as sim:
        sim.init_plasma()
        sim.step(1)
        plan = sim.solver_plan()
        sim.set_phi(two_columns(p))
        sim.step(1)
        for _ in range(2):  # and out again, to the same layout
            monkeypatch.delenv("CUPIC_JACOBI_CTAS", raising=False)
            if back == "set_phi":
                sim.set_phi(two_columns(p, 0.0))
            fake.fake_reset()
            if back != "set_phi":
                getattr(sim, back)()
            sim.poisson_solver(1e-9, 1, 320, 32)
            assert fake.fake_launches(b"k_jacobi") == 0
            assert fake.fake_launches(b"k_tile") == (1 if back == "set_phi" else 2)
            assert sim.solver_plan() == plan
            sim.step(1)
            sim.set_phi(two_columns(p))
            fake.fake_reset()
            sim.poisson_solver(1e-9, 1, 320, 32)
            assert fake.fake_launches(b"k_tile") == 0 and fake.fake_launches(b"k_jacobi") == 11
        assert faults(fake) == []


@pytest.mark.parametrize("ncy,tail", [(4035, 1), (4036, 1), (4085, 1), (4086, 1), (4096, 1), (4097, 0)])
def test_end_of_step_at_its_most_rows(fake, ncy, tail):
    """The end of a step in one launch holds three counts of every row in shared
    memory, up to 4096 rows; beyond, four launches."""
    p = params(2, ncy, max_sweeps=10)
    with cg.Sim(p) as sim:
        sim.init_plasma()
        fake.fake_reset()
        sim.step(1)
        assert fake.fake_launches(b"k_tail") == tail and fake.fake_launches(b"k_finalize") == 1 - tail
        assert faults(fake) == []


@pytest.mark.parametrize("ncx,ncy,form", [(64, 90, "tiles"), (256, 1024, "tiles"), (64, 90, "sweeps"), (256, 1024, "sweeps")])
def test_trial_that_gives_up_is_left_out(fake, monkeypatch, ncx, ncy, form):
    """A trial whose bounded wait expired ran only a part of its sweeps: it is no
    candidate however fast it was, and the trials after it start without its
    flags, as does the context."""
    if form == "sweeps":
        monkeypatch.setenv("CUPIC_JACOBI_NOSTRIP", "1")  # no register tiles
    p = params(ncx, ncy, max_sweeps=100, init_max_sweeps=100)
    with cg.Sim(p) as sim:  # the pick without a fault, kept for the shape
        first = sim.solver_plan()
    p = params(ncx, ncy, max_sweeps=101, init_max_sweeps=101)  # another solve to the tuner
    fake.fake_give_up(first[0], first[2])
    with cg.Sim(p) as sim:
        sim.init_plasma()
        assert sim.flags() == 0
        assert (sim.solver_plan()[0], sim.solver_plan()[2]) != (first[0], first[2])
    assert faults(fake) == []


def test_batched_trial_that_gives_up_tunes_nothing(fake):
    """The batched solve's trials run on the members: once one has given up, those
    after it stop early, so the knobs stay the default ones and are not kept."""
    p = params(16, 40)
    sims = [cg.Sim(p) for _ in range(16)]
    for s in sims:
        s.init_plasma()
    plans = []
    for n in (4, None):  # the second candidate's second launch; no trial
        if n is not None:
            fake.fake_batch_give_up(n)
        with cg.Batch(sims) as b:
            plans.append((b.plan(), fake.fake_launches(b"k_jacobi_batch")))
        assert all(s.flags() == 0 for s in sims)
    assert plans[0][0][:2] == (4, 1)
    assert plans[1][1] > plans[0][1]  # tuned again
    for s in sims:
        s.close()
    assert faults(fake) == []


def test_static_scratch_keeps_words_and_counters_apart(fake, monkeypatch):
    """Calls of the solve on device buffers share one static array, and a halo word
    is told by the number in its upper half: no call's words lie where another
    leaves counters or residuals."""
    fake.fake_watch()
    fake.fake_alloc.restype = ctypes.c_void_p
    fake.fake_alloc.argtypes = [ctypes.c_uint64]
    for ncx, ncy in ((256, 1024), (40, 3000), (1024, 300), (64, 90), (300, 700)):
        p = params(ncx, ncy)
        nodes = p.nnx * p.nny
        rho, phi = fake.fake_alloc(8 * nodes), fake.fake_alloc(4 * nodes)
        for ctas in (None, "2", "5", "7", "151"):
            if ctas:
                monkeypatch.setenv("CUPIC_JACOBI_CTAS", ctas)
            else:
                monkeypatch.delenv("CUPIC_JACOBI_CTAS", raising=False)
            for sweeps in (0, 50):  # no sweeps: the launches of jacobi.cu
                rc = fake.cupic_poisson_solver_static(ctypes.byref(p), rho, phi, None, 1e-3, 1, sweeps, 1, None, None,
                                                      None)
                assert rc in (0, 5), (ncx, ncy, ctas)
    assert fake.fake_launches(b"k_jacobi") > 0 and fake.fake_launches(b"k_tile") > 0
    assert faults(fake) == []


def test_static_solve_without_host_memory_returns_a_status(fake):
    """The layout's search allocates host memory: where that fails, the C entry returns
    a status, and no exception leaves it (in a child: one would end it)."""
    run = """
import ctypes, sys
import cupic_gb300 as cg
cg.library_path = lambda: sys.argv[1]
L = cg.load_library()
L.fake_alloc.restype = ctypes.c_void_p
L.fake_alloc.argtypes = [ctypes.c_uint64]
L.fake_new_left.argtypes = [ctypes.c_longlong]
p = cg.workload_params("tiny")
rho, phi = L.fake_alloc(8 * p.nnx * p.nny), L.fake_alloc(4 * p.nnx * p.nny)
codes = set()
for left in list(range(40)) + [-1]:
    L.fake_new_left(left)
    rc = L.cupic_poisson_solver_static(ctypes.byref(p), rho, phi, None, 1e-3, 1, 50, 1, None, None, None)
    L.fake_new_left(-1)
    codes.add(rc)
assert codes == {0, 3}, codes  # CUPIC_ERR_NOMEM
"""
    subprocess.run([sys.executable, "-c", run, cg.library_path()], check=True, cwd=os.path.dirname(HERE))


def test_draws_beside_the_solve_take_memory_only_where_they_are_made(fake):
    """The scratch of few draws made beside the solve (24 bytes each) is for contexts
    that draw few; one that draws many holds no more than the draws themselves."""
    sizes = {}
    for kte in (1.0, 1e10):  # electrons of mass 1
        p = params(64, 4, kte=kte)
        fake.fake_reset()
        with cg.Sim(p):
            sizes[kte] = fake.fake_allocated()
    caps = [4 * np.ceil(p.dt * p.n * p.ncx * p.ds ** 2 * (kte / (2 * np.pi)) ** 0.5) + 1024 for kte in sizes]
    assert caps[0] < 1100 and caps[1] > 2e4
    # a draw's time, particle and row: 8 + 16 + 4 bytes
    assert sizes[1e10] - sizes[1.0] <= 28 * (caps[1] - caps[0])


def test_steps_of_many_launches_go_one_to_a_graph(fake, monkeypatch):
    """A graph of several steps saves the time between graph launches, 2.5 us a step;
    a precision-form step off the tiles is a launch per correction, and eight of
    them would take longer to capture than that earns."""
    monkeypatch.setenv("CUPIC_JACOBI_NOSTRIP", "1")  # no tiles
    p = params(48, 40, refine_every=4, max_sweeps=400)
    with cg.Sim(p) as sim:
        sim.init_plasma()
        fake.fake_reset()
        sim.step(64)
        assert fake.fake_launches(b"k_jacobi") == 101  # one step's, captured once
    monkeypatch.delenv("CUPIC_JACOBI_NOSTRIP")
    with cg.Sim(p) as sim:
        sim.init_plasma()
        fake.fake_reset()
        sim.step(64)
        assert fake.fake_launches(b"k_tile") == 1 + 8
