"""Work lists of ensembles whose droplets do not share one material: the kernel has the L2 term when any droplet has, and
its tiles must start where that kernel's loads may (a TMA box starts on 16 bytes: column k0 - 2 with the L2 term, k0 - 4
without, a multiple of 4 floats)."""
import ctypes as C

import numpy as np
import pytest

import fake_gpu
from lcdrsimulator_b200 import EnsembleSolver


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_gpu.build(tmp_path_factory.mktemp("fake_gpu"))


def items(launch):
    n = launch.arg[4]
    return np.ctypeslib.as_array((C.c_int * (8 * n)).from_address(launch.arg[2])).reshape(n, 8).copy()


MIXED = [dict(N=40, droplet_radius_cells=13.0), dict(N=33, own_material=1, L2=3e-12), dict(N=50, Ny=36, Nz=61),
         dict(N=36, droplet_radius_cells=10.0, own_material=1, L2=3e-12, L3=1e-12, W=1e-5)]


@pytest.mark.parametrize("L2,instances", [
    (0.0, MIXED),
    (3e-12, [dict(N=40, droplet_radius_cells=13.0), dict(N=33, own_material=1), dict(N=50, own_material=1, L3=1e-12)]),
    (0.0, [dict(N=40, droplet_radius_cells=13.0), dict(N=33, own_material=1, L3=1e-12)]),
])
def test_tiles_start_where_the_kernel_may_load(fake, L2, instances):
    with fake_gpu.use(fake) as g, EnsembleSolver(instances, L1=6e-12, L2=L2) as s:
        s.initial_fields()
        s.step(1)
        step = g.launches("k_step_ensemble")[-1]
        l2_kernel = "k_step_ensembleILb1E" in step.name
        assert l2_kernel == (L2 != 0 or any(d.get("L2") for d in instances))
        t = items(step)
        assert set(t[:, 4]) == set(range(len(instances)))
        for j0, k0, ib, ie, inst, *_ in t:
            assert (k0 - (2 if l2_kernel else 4)) % 4 == 0, (j0, k0, ib, ie, inst)
            assert l2_kernel or k0 % 8 == 0


def test_every_changing_cell_lies_in_one_item(fake):
    with fake_gpu.use(fake) as g, EnsembleSolver(MIXED, L1=6e-12) as s:
        s.initial_fields()
        s.step(1)
        t = items(g.launches("k_step_ensemble")[-1])
        for n, masks in enumerate(g.launches("k_tile_masks")[-len(MIXED):]):
            flags, nx, ny, nz, sj, si = masks.arg[1:7]
            f = np.ctypeslib.as_array((C.c_uint8 * (nx * si)).from_address(flags)).reshape(nx, si // sj, sj)
            seen = np.zeros((nx, ny + 8, nz + 64), dtype=int)
            for j0, k0, ib, ie, *_ in t[t[:, 4] == n]:
                seen[ib:ie, j0:j0 + 8, max(k0, 0):k0 + 32] += 1
            change = (f[:, :ny, :nz] & 3) != 0
            assert change.any() and (seen[:, :ny, :nz][change] == 1).all()
