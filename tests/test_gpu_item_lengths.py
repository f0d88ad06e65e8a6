"""The confined step and the IMEX sweeps with work items of forced lengths (LDG_QSR_CHUNK) and at a size where the step's and
the sweeps' own lengths differ: ring slots that are refilled once, often, or never (GPU).

Against the FP64 oracle, <= 2e-6 of max |Q| (a handful of FP32 roundings of 6e-8 a step); with noise against the
one-thread-per-cell kernel (the same draws), the same bound; compensated storage keeps only the rounding of the
increments (at most 0.3 of max |Q| a step, some 8 roundings of 6e-8): <= 7e-7 after five steps.
"""
import pytest

from gpu_helpers import fp32, make_pair, rel_err

pytestmark = pytest.mark.gpu

ALL = dict(L1=6e-12, L2=3e-12, L3=1e-12, W=1e-5)
GRIDS = {
    "L1": dict(Nx=61, Ny=50, Nz=67, L1=6e-12, W=1e-5),
    "all": dict(Nx=48, Ny=43, Nz=52, droplet_radius_cells=20.0, **ALL),
    "all_faces": dict(Nx=33, Ny=15, Nz=41, droplet_radius_cells=40.0, **ALL),
}
T, S_SHELL, DT = 302.0, 0.6, 1.4e-10


def _problem(oracle, kw):
    op, solver, d = make_pair(**kw)
    g, fl = oracle.geometry(op)
    q0 = fp32(oracle.init(op, g, 0, 17, 0.5))
    solver.upload(q0)
    return op, solver, g, fl, q0


@pytest.mark.parametrize("planes", [1, 2, 5, 9, 16, 64])
@pytest.mark.parametrize("name", list(GRIDS))
def test_forced_lengths(oracle, monkeypatch, name, planes):
    monkeypatch.setenv("LDG_QSR_CHUNK", str(planes))
    op, solver, g, fl, q0 = _problem(oracle, GRIDS[name])
    solver.step(5, T, S_SHELL, DT)
    assert rel_err(solver.download(), oracle.step_explicit(op, g, fl, q0, T, S_SHELL, DT, n=5)) <= 2e-6
    solver.upload(q0)
    solver.step(2, T, S_SHELL, 4 * DT, semi_implicit=True, L_stab=6e-12, jacobi_iters=7)
    assert rel_err(solver.download(), oracle.step_imex(op, g, fl, q0, T, S_SHELL, 4 * DT, 6e-12, 7, n=2)) <= 2e-6
    solver.upload(q0)
    solver.step(3, T, S_SHELL, DT, noise_sigma=1e-3, seed=9, step_index=4)
    got = solver.download()
    solver.upload(q0)
    monkeypatch.setenv("LDG_QSR_KERNEL", "direct")
    solver.step(3, T, S_SHELL, DT, noise_sigma=1e-3, seed=9, step_index=4)
    assert rel_err(got, solver.download()) <= 2e-6
    solver.close()


@pytest.mark.parametrize("planes", [1, 5, 16])
@pytest.mark.parametrize("name", list(GRIDS))
def test_compensated_storage(oracle, monkeypatch, name, planes):
    monkeypatch.setenv("LDG_QSR_CHUNK", str(planes))
    op, solver, g, fl, q0 = _problem(oracle, dict(GRIDS[name], compensated=1))
    solver.step(5, T, S_SHELL, DT)
    assert rel_err(solver.download(), oracle.step_explicit(op, g, fl, q0, T, S_SHELL, DT, n=5)) <= 7e-7
    solver.close()


@pytest.mark.parametrize("kw", [dict(Nx=112, Ny=112, Nz=112, L1=6e-12, droplet_radius_cells=50.0),
                                dict(Nx=90, Ny=96, Nz=101, droplet_radius_cells=44.0, **ALL)], ids=["L1", "all"])
def test_imex_at_the_lengths_that_the_size_picks(oracle, kw):
    op, solver, g, fl, q0 = _problem(oracle, kw)
    solver.step(2, T, S_SHELL, 4 * DT, semi_implicit=True, L_stab=6e-12, jacobi_iters=5)
    assert rel_err(solver.download(), oracle.step_imex(op, g, fl, q0, T, S_SHELL, 4 * DT, 6e-12, 5, n=2)) <= 2e-6
    solver.close()
