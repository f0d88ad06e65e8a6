"""The confined step at grid sizes where the work list is cut into items of different lengths (1 to 12 planes,
chosen from the size and the elastic terms), against the FP64 oracle (GPU).

Tolerance: five explicit steps from an identical FP32-representable field, <= 2e-6 of max |Q| (a handful of FP32
roundings of 6e-8 per step).
"""
import pytest

from gpu_helpers import make_pair, fp32, rel_err

pytestmark = pytest.mark.gpu

ALL = dict(L1=6e-12, L2=3e-12, L3=1e-12, W=1e-5)
CASES = {
    "L1_40": dict(Nx=40, Ny=40, Nz=40, L1=6e-12),
    "L1_ragged_61_50_67": dict(Nx=61, Ny=50, Nz=67, L1=6e-12, W=1e-5),
    "L1_112": dict(Nx=112, Ny=112, Nz=112, L1=6e-12, droplet_radius_cells=50.0),
    "all_48": dict(Nx=48, Ny=48, Nz=48, droplet_radius_cells=20.0, **ALL),
    "all_ragged_75_90_66": dict(Nx=75, Ny=90, Nz=66, **ALL),
    "all_112": dict(Nx=112, Ny=112, Nz=112, droplet_radius_cells=52.0, **ALL),
    # radius beyond the box: cells on the faces move, L1 only (stencils two cells in from the face) and L3 only
    "L1_faces_move": dict(Nx=18, Ny=15, Nz=41, L1=6e-12, W=1e-5, droplet_radius_cells=40.0),
    "L3_faces_move": dict(Nx=18, Ny=15, Nz=41, L1=6e-12, L3=1e-12, W=1e-5, droplet_radius_cells=40.0),
    "all_faces_move": dict(Nx=18, Ny=15, Nz=41, droplet_radius_cells=40.0, **ALL),
}


@pytest.mark.parametrize("name", list(CASES))
def test_step_matches_oracle_at_every_item_length(oracle, name):
    op, solver, d = make_pair(**CASES[name])
    g, fl = oracle.geometry(op)
    q0 = fp32(oracle.init(op, g, 0, 17, 0.5))
    solver.upload(q0)
    solver.step(5, 302.0, 0.6, 1.4e-10)
    want = oracle.step_explicit(op, g, fl, q0, 302.0, 0.6, 1.4e-10, n=5)
    assert rel_err(solver.download(), want) <= 2e-6
    solver.close()
