"""Periodic FP64 observables where the sums, the eigen-solver and the plaquette winding are at their edges (GPU): fields that are
zero, uniform along the axes (director components exactly zero, doubled angles exactly on the branch), in planes of exact
+-45 and 90 degree turns (parallel, perpendicular and antiparallel neighbours), tiny boxes, and cuts at 0 and 1/2.

Against the FP64 oracle; counts equal, values to 1e-10 (FP64 sums in another order).
"""
import math

import numpy as np
import pytest

from gpu_helpers import fp32
from lcdrsimulator_b200 import KZMSolver

pytestmark = pytest.mark.gpu


def _uniaxial(n, S=0.6):
    n = n / np.linalg.norm(n, axis=-1, keepdims=True)
    x, y, z = n[..., 0], n[..., 1], n[..., 2]
    return S * np.stack([x * x - 1 / 3, x * y, x * z, y * y - 1 / 3, y * z], -1)


def _fields(shape):
    a, b, c = np.meshgrid(*[np.arange(k) for k in shape], indexing="ij")
    rng = np.random.default_rng(1)
    turn = (a + 2 * b + c) % 4 * (math.pi / 4)
    return {
        "zero": np.zeros(shape + (5,)),
        "x": _uniaxial(np.broadcast_to([1.0, 0.0, 0.0], shape + (3,))),
        "z": _uniaxial(np.broadcast_to([0.0, 0.0, 1.0], shape + (3,))),
        "turns": _uniaxial(np.stack([np.round(np.cos(turn), 12), np.round(np.sin(turn), 12), 0 * turn], -1)),
        "checker": _uniaxial(np.where(((a + b + c) % 2 == 0)[..., None], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0])),
        "random": _uniaxial(rng.standard_normal(shape + (3,))),
        "negative order": _uniaxial(rng.standard_normal(shape + (3,)), S=-0.4),
        "large": 1e3 * rng.standard_normal(shape + (5,)),
        "small": 1e-8 * rng.standard_normal(shape + (5,)),
    }


NAMES = list(_fields((2, 2, 2)))


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 3, 34)])
@pytest.mark.parametrize("cut", [0.25, 0.5])
def test_periodic_observables(oracle, name, shape, cut):
    from oracle.oracle import OrcBulkParams
    q = fp32(_fields(shape)[name].ravel())
    Nz, Ny, Nx = shape
    s = KZMSolver(Nx, Ny, Nz, 1e-8, 1.1e-8, 0.9e-8, 6e-12, 0.1, defects_charge_cutoff=cut)
    s.upload(q)
    got = s.observe(-9e5, 6e6, 5e6)
    bp = OrcBulkParams()
    for k, v in dict(Nx=Nx, Ny=Ny, Nz=Nz, dx=1e-8, dy=1.1e-8, dz=0.9e-8, kappa=6e-12, gamma=0.1,
                     defects_S_threshold=0.1, defects_charge_cutoff=cut).items():
        setattr(bp, k, v)
    want = oracle.bulk_observe(bp, q, -9e5, 6e6, 5e6)
    assert got["defect_plaquettes_used"] == want["defect_plaquettes_used"]
    if name != "turns" and cut < 0.5:  # exact half turns: which way one rounds is the host's and the GPU's own
        assert got["nonzero_defect_plaquettes"] == want["nonzero_defect_plaquettes"]
    for k in ("bulk", "elastic", "avg_S", "max_S"):
        assert got[k] == pytest.approx(want[k], rel=1e-10, abs=1e-25)
    s.close()
