"""An ensemble whose droplets have materials of their own (with and without the L2 and L3 terms) against each droplet in a
solver of its own. The ensemble's kernel evaluates every droplet with the terms that any of them has, at zero
coefficients where a droplet has not, so the two agree to the rounding of the FP32 updates."""
import numpy as np
import pytest

from lcdrsimulator_b200 import EnsembleSolver, QSRSolver

pytestmark = pytest.mark.gpu

SHARED = dict(dx=1e-8, dy=1e-8, dz=1e-8, a=0.044e6, b=1.413e6, c=1.153e6, T_star=307.0, bulk_modechoice=1, kappa=0.0,
              L1=6e-12, gamma=0.1)
STEPS, DT, T = 6, 1.6e-10, 302.0


@pytest.mark.parametrize("L2,instances", [
    (0.0, [dict(N=40, droplet_radius_cells=13.0), dict(N=33, own_material=1, L2=3e-12),
           dict(N=41, Ny=36, Nz=61, droplet_radius_cells=15.0),
           dict(N=36, own_material=1, L2=3e-12, L3=1e-12, W=1e-5)]),
    (3e-12, [dict(N=40, droplet_radius_cells=13.0), dict(N=33, own_material=1), dict(N=45, own_material=1, L3=1e-12)]),
])
def test_each_droplet_as_in_its_own_solver(L2, instances):
    instances = [dict(d, T_high=T, T_low=T, seed=5 + n) for n, d in enumerate(instances)]
    with EnsembleSolver(instances, L2=L2, L3=0.0, W=0.0, dt=DT, boundary_custom=1, boundary_S=0.6, **SHARED) as e:
        e.initial_fields(S0=0.5)
        start = [e.download(n) for n in range(len(instances))]
        e.step(STEPS)
        got = [e.download(n) for n in range(len(instances))]
    for n, d in enumerate(instances):
        own = {k: d.get(k, 0.0) for k in ("L2", "L3", "W")} if d.get("own_material") else dict(L2=L2, L3=0.0, W=0.0)
        with QSRSolver(Nx=d["N"], Ny=d.get("Ny", d["N"]), Nz=d.get("Nz", d["N"]),
                       droplet_radius_cells=d.get("droplet_radius_cells", 0.0), **own, **SHARED) as s:
            s.upload(start[n])
            s.step(STEPS, T, 0.6, DT)
            want = s.download()
        assert not np.array_equal(start[n], want)
        # one FP32 rounding of the field per step and side, and the update's own (dt mu of order 0.1 of the field)
        assert np.abs(got[n] - want).max() <= STEPS * 2.0 ** -23 * np.abs(want).max(), n
