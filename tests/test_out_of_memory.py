"""Calls after one that ran out of device memory, on a runtime whose n-th allocation fails: the failing call returns an
error, a later one starts again, and no launch gets memory that is not there."""
import ctypes as C

import numpy as np
import pytest

import fake_gpu
from lcdrsimulator_b200 import EnsembleSolver, LdgError, QSRSolver

STEP = dict(T=302.0, S_shell=0.6, dt=1.6e-10)
IMEX = dict(semi_implicit=True, L_stab=6e-12, jacobi_iters=3)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_gpu.build(tmp_path_factory.mktemp("fake_gpu"))


def solver(**kw):
    s = QSRSolver(Nx=40, Ny=40, Nz=40, droplet_radius_cells=14.0, L1=6e-12, **kw)
    s.upload(np.zeros(5 * s.n))
    return s


def test_a_call_after_a_failed_allocation(fake):
    with fake_gpu.use(fake) as g, QSRSolver(Nx=24, Ny=24, Nz=24, droplet_radius_cells=8.0) as s:
        q = np.zeros(5 * s.n)
        g.fail_malloc(1)
        with pytest.raises(LdgError):
            s.upload(q)  # the staging buffer
        s.upload(q)  # its own launch passed: the failed allocation is not reported again
        s.step(1, **STEP)


@pytest.mark.parametrize("L2", [0.0, 3e-12])
def test_imex_after_a_failed_set_up(fake, L2):
    with fake_gpu.use(fake) as g:
        failed = 0
        for n in range(1, 10):
            before = g.live()
            with solver(L2=L2) as s:
                held = g.live()
                g.fail_malloc(n)
                try:
                    s.step(1, **STEP, **IMEX)
                except LdgError:
                    failed += 1
                    assert g.live() == held  # nothing of the failed set-up stays
                    assert not g.launches("k_sweep_tiled", g.count())
                g.fail_malloc(0)
                start = g.count()
                s.step(1, **STEP, **IMEX)
                sweeps = g.launches("k_sweep_tiled", start)
                assert len(sweeps) == 3
                for x in sweeps:
                    assert g.is_live(x.arg[3]) and g.is_live(x.arg[4])
            assert g.live() == before
        assert failed == 3  # right-hand side, items, masks


def test_steps_after_a_failed_autotune(fake):
    with fake_gpu.use(fake) as g, solver() as s:
        failed = 0
        for n in range(1, 40):
            g.fail_malloc(n)
            try:
                s.autotune(trial_steps=1, **STEP)
            except LdgError:
                failed += 1
            g.fail_malloc(0)
            start = g.count()
            s.step(1, **STEP)
            (step,) = g.launches("k_step_tiled", start)
            assert g.is_live(step.arg[3]) and g.is_live(step.arg[4])
        assert failed >= 5  # the field's copy and at least two lists


def test_ensemble_steps_after_a_failed_autotune(fake):
    instances = [dict(N=40, droplet_radius_cells=13.0, T_high=310.0, T_low=300.0), dict(N=33)]
    with fake_gpu.use(fake) as g, EnsembleSolver(instances, L1=6e-12) as s:
        s.initial_fields()
        s.step(3)
        ctl = g.launches("k_step_ensemble")[-1].arg[5]
        device_step = C.c_longlong.from_address(ctl + 8)  # EnsCtl: next, done, step
        failed = 0
        for n in range(1, 40):
            device_step.value = -1  # as trials that ran would leave it: another step than the host's
            g.fail_malloc(n)
            try:
                s.autotune(trial_steps=1)
            except LdgError:
                failed += 1
            g.fail_malloc(0)
            assert device_step.value == s.step_index
            start = g.count()
            s.step(33)  # one replayed graph and one launch
            assert s.step_index == 3 + 33 * n
            launched = g.launches("k_step_ensemble", start)
            for x in launched:
                assert g.is_live(x.arg[2]) and g.is_live(x.arg[3]) and g.is_live(x.arg[5])
            assert launched
        assert failed >= 6
