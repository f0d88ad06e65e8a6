"""Work-item lengths: what autotuning returns is the length in use, a length is timed once, and LDG_QSR_CHUNK is that
length on lists of any size (CPU, on a runtime that records launches)."""
import ctypes as C

import numpy as np
import pytest

import fake_gpu
from lcdrsimulator_b200 import EnsembleSolver, QSRSolver

STEP = dict(T=302.0, S_shell=0.6, dt=1.6e-10)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_gpu.build(tmp_path_factory.mktemp("fake_gpu"))


def longest(address, n):
    t = np.ctypeslib.as_array((C.c_int * (8 * n)).from_address(address)).reshape(n, 8)
    return int((t[:, 3] - t[:, 2]).max())


def solver(N, R):
    s = QSRSolver(Nx=N, Ny=N, Nz=N, droplet_radius_cells=R, L1=6e-12)
    s.upload(np.zeros(5 * s.n))
    return s


def step_list(g, s):
    start = g.count()
    s.step(1, **STEP)
    (x,) = g.launches("k_step_tiled", start)
    return longest(x.arg[4], x.grid)


# lists of one and of several lengths
@pytest.mark.parametrize("N,R", [(40, 14.0), (128, 58.0), (200, 98.0)])
def test_autotune_returns_the_length_in_use(fake, N, R):
    with fake_gpu.use(fake) as g, solver(N, R) as s:
        g.elapsed([5.0, 4.0, 3.0, 3.5, 6.0, 6.0, 6.0])
        start = g.count()
        got = s.autotune(trial_steps=1, **STEP)
        trials = g.launches("k_step_tiled", start)
        assert got == step_list(g, s)
        assert len(trials) % 3 == 0 and len(trials) // 3 == len({x.grid for x in trials})  # one trial per list


def test_ensemble_autotune_returns_the_length_in_use(fake):
    with fake_gpu.use(fake) as g, EnsembleSolver([dict(N=40, droplet_radius_cells=13.0), dict(N=33)], L1=6e-12) as s:
        s.initial_fields()
        got = s.autotune(trial_steps=1)
        s.step(1)
        x = g.launches("k_step_ensemble")[-1]
        assert got == longest(x.arg[2], x.arg[4])


@pytest.mark.parametrize("planes", [1, 5, 8, 16, 20])
def test_the_variable_sets_the_length(fake, monkeypatch, planes):
    monkeypatch.setenv("LDG_QSR_CHUNK", str(planes))
    with fake_gpu.use(fake) as g, solver(40, 14.0) as s:
        assert step_list(g, s) == planes
