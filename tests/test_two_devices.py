"""Solvers on two GPUs of one process (CPU, on a runtime that refuses a launch whose shared-memory limit was not raised on
the current device)."""
import numpy as np
import pytest

import fake_gpu
from lcdrsimulator_b200 import EnsembleSolver, QSRSolver

STEP = dict(T=302.0, S_shell=0.6, dt=1.6e-10)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_gpu.build(tmp_path_factory.mktemp("fake_gpu"))


def solver(L2=0.0, **kw):
    s = QSRSolver(Nx=30, Ny=28, Nz=33, L1=6e-12, L2=L2, **kw)
    s.upload(np.zeros(5 * s.n))
    return s


@pytest.mark.parametrize("kw", [dict(), dict(L2=3e-12), dict(L2=3e-12, L3=1e-12, compensated=1), dict(L3=1e-12)])
def test_steps_and_sweeps_on_both(fake, kw):
    with fake_gpu.use(fake) as g:
        solvers = []
        for d in (0, 1):
            g.set_device(d)
            solvers.append(solver(**kw))
        g.set_device(0)
        for d, s in enumerate(solvers):
            start = g.count()
            s.step(1, **STEP)
            s.step(1, **STEP, semi_implicit=True, L_stab=6e-12, jacobi_iters=2)
            assert {x.device for x in g.launches("_tiled", start)} == {d}
        for s in solvers:
            s.close()


def test_ensembles_on_both(fake):
    with fake_gpu.use(fake) as g:
        for d in (1, 0):
            g.set_device(d)
            with EnsembleSolver([dict(N=30, L2=3e-12, own_material=1)], L1=6e-12) as s:
                s.initial_fields()
                s.step(1)
                assert g.launches("k_step_ensemble")[-1].device == d
