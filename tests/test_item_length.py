"""Work-item lengths: autotuning keeps the list of its fastest trial, times a list once and returns the longest item that it
allowed, and LDG_QSR_CHUNK is the length on lists of any size (CPU, on a runtime that records launches)."""
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


CANDIDATES = (8, 12, 16, 24, 32, 48, 64)


# lists of one and of several lengths
@pytest.mark.parametrize("N,R", [(40, 14.0), (128, 58.0), (200, 98.0)])
@pytest.mark.parametrize("ms", [[5.0, 4.0, 3.0, 3.5, 6.0, 6.0, 6.0], [1.0, 4.0, 4.0, 4.0, 4.0, 4.0, 4.0]])
def test_autotune_keeps_the_fastest_list(fake, N, R, ms):
    with fake_gpu.use(fake) as g, solver(N, R) as s:
        g.elapsed(ms)
        start = g.count()
        got = s.autotune(trial_steps=1, **STEP)
        lists = [x.grid for x in g.launches("k_step_tiled", start)][::3]  # two steps before each timed one
        assert len(lists) == len(set(lists))  # one trial per list
        start = g.count()
        longest_item = step_list(g, s)
        (step,) = g.launches("k_step_tiled", start)
        assert step.grid == lists[int(np.argmin(ms[:len(lists)]))]
        assert got in CANDIDATES and longest_item <= got


def test_ensemble_autotune_times_a_list_once(fake):
    with fake_gpu.use(fake) as g, EnsembleSolver([dict(N=40, droplet_radius_cells=13.0), dict(N=33)], L1=6e-12) as s:
        s.initial_fields()
        start = g.count()
        got = s.autotune(trial_steps=1)
        lists = [x.arg[4] for x in g.launches("k_step_ensemble", start)]
        trials = lists[:len(lists) - 32:3]  # the captured graph of 32 steps comes last
        assert len(trials) == len(set(trials))
        s.step(1)
        x = g.launches("k_step_ensemble")[-1]
        assert got in CANDIDATES and longest(x.arg[2], x.arg[4]) <= got


@pytest.mark.parametrize("planes", [1, 5, 8, 16, 20])
def test_the_variable_sets_the_length(fake, monkeypatch, planes):
    monkeypatch.setenv("LDG_QSR_CHUNK", str(planes))
    with fake_gpu.use(fake) as g, solver(40, 14.0) as s:
        assert step_list(g, s) == planes
