"""Where the epochs of the halo words start over (after 0xc0000000 exchanges) the
maxima of checked sweeps, which carry epochs too, are cleared with them: after a
wrap inside a batched solve, and after one on a single CTA of the solve on device
buffers, the next solve reads its own maxima.  The base is moved near the end
by hand (epoch/set_epoch.cu: the library with two functions more)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import cupic_gb300 as cg
from cupic_gb300 import build
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
END = 0xc0000000


@pytest.fixture
def lib(gpu_lib, tmp_path_factory, monkeypatch):
    out = str(tmp_path_factory.mktemp("epoch") / "libcupic_epoch.so")
    objs = [os.path.join(build.OUT, os.path.splitext(s)[0] + ".o") for s in build.SOURCES if s != "noalloc.cu"]
    subprocess.run([build.nvcc()] + build.common_flags() + ["-I", build.CSRC, "-shared", "-Xlinker", "-Bsymbolic",
                   "-cudart", "static", "-o", out, os.path.join(HERE, "epoch", "set_epoch.cu")] + objs, check=True)
    for name in ("CTAS", "DEPTH", "TUNE"):
        monkeypatch.delenv("CUPIC_JACOBI_" + name, raising=False)
    monkeypatch.setattr(cg, "_LIB", None)
    monkeypatch.setattr(cg, "library_path", lambda: out)
    L = cg.load_library()
    L.set_epoch.argtypes = [ctypes.c_void_p, ctypes.c_uint]
    L.get_epoch.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint)]
    return L


def test_wrap_inside_a_batched_solve(lib):
    # columns in blocks: the maxima go by way of L2
    p = cg.workload_params("tiny", ncx=220, ncy=70, n=4.0, tol=2e-2, min_sweeps=1, max_sweeps=200)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    rng = np.random.default_rng(5)
    with cg.Sim(p) as sim:
        sim.init_plasma()
        assert lib.set_epoch(sim.h, END - 500) == 0
        # maxima and all halo words with epochs just below the end
        sim.poisson_solver(1e-30, 1, 200, 1)
        ora.solve(1e-30, 1, 200, 1)
        with cg.Batch([sim]) as b:
            assert lib.set_epoch(sim.h, END - 1) == 0
            b.step(1)
            ora.step(1)
        epoch = ctypes.c_uint()
        assert lib.get_epoch(sim.h, ctypes.byref(epoch)) == 0 and epoch.value < 1000
        for _ in range(3):
            phi = rng.standard_normal((p.nny, p.nnx)).astype(np.float32).astype(np.float64)
            sim.set_phi(phi)
            ora.set_phi(phi)
            sim.poisson_solver(2e-2, 1, 200, 1)
            ora.solve(2e-2, 1, 200, 1)
            np.testing.assert_array_equal(sim.phi().astype(np.float64), ora.phi())
        sim.step(1)
        ora.step(1)
        g, o = sim.stats(1)[0], ora.stats()
        assert g["sweeps"] == o["sweeps"] and g["residual"] == o["residual"]
    ora.close()


def test_wrap_on_one_cta_of_the_solve_on_device_buffers(lib, monkeypatch):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(6)

    def solve(ncx, ncy, phi, tol=2e-2):
        p = cg.workload_params("tiny", ncx=ncx, ncy=ncy)
        d_rho = torch.zeros(p.nnx * p.nny, dtype=torch.int64, device="cuda")
        d_phi = torch.from_numpy(phi.copy()).to("cuda")
        sweeps, res = ctypes.c_int32(), ctypes.c_float()
        torch.cuda.synchronize()
        rc = lib.cupic_poisson_solver_static(ctypes.byref(p), d_rho.data_ptr(), d_phi.data_ptr(), None, tol, 1, 150, 1,
                                             None, ctypes.byref(sweeps), ctypes.byref(res))
        assert rc == 0
        return d_phi.cpu().numpy(), sweeps.value, res.value

    big = rng.standard_normal((71, 201)).astype(np.float32)
    small = rng.standard_normal((34, 101)).astype(np.float32)
    first = solve(200, 70, big)  # epochs from the start: the answer
    assert lib.set_static_epoch(END - 500) == 0
    solve(200, 70, 0.1 * big, 1e-30)
    assert lib.set_static_epoch(END - 1) == 0
    monkeypatch.setenv("CUPIC_JACOBI_CTAS", "1")
    solve(100, 33, small)
    monkeypatch.delenv("CUPIC_JACOBI_CTAS")
    epoch = ctypes.c_uint()
    assert lib.get_static_epoch(ctypes.byref(epoch)) == 0 and epoch.value < 1000
    again = solve(200, 70, big)
    np.testing.assert_array_equal(again[0], first[0])
    assert again[1:] == first[1:]
