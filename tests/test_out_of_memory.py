"""Calls after one that ran out of device memory, on a runtime whose n-th allocation fails: the failing call returns an
error, a later one starts again, and no launch gets memory that is not there."""
import numpy as np
import pytest

import fake_gpu
from lcdrsimulator_b200 import LdgError, QSRSolver

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
