"""Calls after one that ran out of device memory, on a runtime whose n-th allocation fails: the failing call returns an
error, a later one starts again, and no launch gets memory that is not there."""
import numpy as np
import pytest

import fake_gpu
from lcdrsimulator_b200 import LdgError, QSRSolver

STEP = dict(T=302.0, S_shell=0.6, dt=1.6e-10)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_gpu.build(tmp_path_factory.mktemp("fake_gpu"))


def test_a_call_after_a_failed_allocation(fake):
    with fake_gpu.use(fake) as g, QSRSolver(Nx=24, Ny=24, Nz=24, droplet_radius_cells=8.0) as s:
        q = np.zeros(5 * s.n)
        g.fail_malloc(1)
        with pytest.raises(LdgError):
            s.upload(q)  # the staging buffer
        s.upload(q)  # its own launch passed: the failed allocation is not reported again
        s.step(1, **STEP)
