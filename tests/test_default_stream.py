"""No call leaves work behind on the default stream: the solvers' streams are non-blocking, so a late clearing of a buffer
would erase what has been written since (CPU, on a runtime that counts default-stream work which nothing waited for)."""
import ctypes as C

import numpy as np
import pytest

import fake_gpu
from lcdrsimulator_b200 import EnsembleSolver, KZMSolver, QSRSolver

STEP = dict(T=302.0, S_shell=0.6, dt=1.6e-10)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_gpu.build(tmp_path_factory.mktemp("fake_gpu"))


@pytest.mark.parametrize("radius", [0.0, 10.0])
@pytest.mark.parametrize("compensated", [0, 1])
def test_confined_solver(fake, radius, compensated):
    with fake_gpu.use(fake) as g:
        with QSRSolver(Nx=30, Ny=28, Nz=33, droplet_radius_cells=radius, L1=6e-12, compensated=compensated) as s:
            assert g.pending() == 0
            s.upload(np.zeros(5 * s.n))
            s.step(2, **STEP)
            s.step(1, **STEP, semi_implicit=True, L_stab=6e-12, jacobi_iters=2)
            s.autotune(trial_steps=1, **STEP)
            s.observe(302.0, 0.6)
            s.download()
            assert g.pending() == 0


def test_ensemble(fake):
    with fake_gpu.use(fake) as g, EnsembleSolver([dict(N=30, droplet_radius_cells=9.0), dict(N=24)], L1=6e-12) as s:
        assert g.pending() == 0
        s.initial_fields()
        s.step(40)
        s.autotune(trial_steps=1)
        s.observe_all()
        assert g.pending() == 0


def test_periodic_solver(fake):
    with fake_gpu.use(fake) as g:
        s = KZMSolver(20, 18, 22, 1e-8, 1e-8, 1e-8, 6.5e-12, 0.1)
        assert g.pending() == 0
        s.upload(np.zeros(5 * s.n))
        s.download()
        assert g.pending() == 0
        s.close()


def test_convolution(fake):
    class Shape(C.Structure):
        _fields_ = [(n, C.c_int) for n in ("N", "D", "H", "W", "Ci", "Co")]

    with fake_gpu.use(fake) as g:
        stream = C.c_void_p(0x1000)
        p = [C.c_void_p(256 * (i + 1)) for i in range(3)]  # device addresses that nothing reads here
        s = Shape(1, 8, 8, 8, 32, 32)
        assert g.lib.sg_conv3d_fwd(C.byref(s), *p[:2], None, p[2], 0, 0, stream) == 0
        assert g.lib.sg_check(stream) == 0
        assert g.pending() == 0
