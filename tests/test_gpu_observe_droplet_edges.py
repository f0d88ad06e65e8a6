"""The droplet's log point where its sums and the eigen-solver are at their edges (GPU): zero and uniform fields, orders whose
row sums are the smallest eigenvector (negative uniaxial along the diagonals, one negative off-diagonal entry), fields that
do not vanish outside the droplet, the smallest grids, large and small values, infinities and NaN.

Against the FP64 oracle: counts equal, values to 1e-10 (FP64 sums in another order; the elastic and anchoring sums of a field
that has no gradient or fits the shell are rounding noise against the squares that they are formed from).
"""
import math

import numpy as np
import pytest

from gpu_helpers import fp32, make_pair
from lcdrsimulator_b200 import KZMSolver

pytestmark = pytest.mark.gpu

GRIDS = {
    "droplet": dict(Nx=20, Ny=24, Nz=37, L1=6e-12, L2=3e-12, L3=1e-12, W=1e-5, droplet_radius_cells=8.0),
    "whole_box": dict(Nx=9, Ny=12, Nz=33, L1=6e-12, W=0.0, droplet_radius_cells=40.0),
    "smallest": dict(Nx=3, Ny=3, Nz=3, L1=6e-12, W=1e-5, droplet_radius_cells=2.0),
    "kappa": dict(Nx=16, Ny=16, Nz=16, L1=0.0, kappa=6.5e-12),
}


def _uniaxial(n, S):
    n = np.asarray(n, dtype=float)
    n = n / np.linalg.norm(n, axis=-1, keepdims=True)
    x, y, z = n[..., 0], n[..., 1], n[..., 2]
    return S * np.stack([x * x - 1 / 3, x * y, x * z, y * y - 1 / 3, y * z], -1)


def _fields(n):
    rng = np.random.default_rng(2)
    one = np.ones((n, 1))
    return {
        "zero": np.zeros((n, 5)),
        "z": one * _uniaxial([0, 0, 1], 0.6),
        "negative along (1, 1, 1)": one * _uniaxial([1, 1, 1], -0.5),
        "negative along (1, -1, 1)": one * _uniaxial([1, -1, 1], -0.3),
        "negative xy": one * np.array([0, -0.3, 0, 0, 0]),
        "negative yz": one * np.array([0, 0, 0, 0, -0.1]),
        "random": _uniaxial(rng.standard_normal((n, 3)), 0.6),
        "random negative": _uniaxial(rng.standard_normal((n, 3)), -0.4),
        "large": 1e3 * rng.standard_normal((n, 5)),
        "small": 1e-8 * rng.standard_normal((n, 5)),
    }


NAMES = list(_fields(1))


def _same(got, want, key, floor=0.0):
    if math.isnan(want):
        assert math.isnan(got), key
    else:
        assert got == pytest.approx(want, rel=1e-10, abs=max(floor, 1e-300)), key


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("grid", list(GRIDS))
def test_droplet_observables(oracle, grid, name):
    op, solver, d = make_pair(**GRIDS[grid])
    g, fl = oracle.geometry(op)
    q = fp32(_fields(solver.n)[name].ravel())
    solver.upload(q)
    got = solver.observe(300.0, 0.6)
    want = oracle.observe(op, g, fl, q, 300.0, 0.6)
    for k in ("radiality_count", "core_count", "defect_count", "defect_plaquettes", "xi_edges"):
        assert got[k] == want[k], k
    # squares of the field that the elastic and anchoring terms are differences of, summed over the box: 1e-16 of them
    square = (q ** 2).max() * solver.n * d["dx"] * d["dy"] * d["dz"]
    elastic = 1e-14 * max(d["L1"], d["kappa"]) / d["dx"] ** 2 * square
    anchoring = 1e-14 * abs(d["W"]) / d["dx"] * (square + solver.n * d["dx"] ** 3)
    _same(got["bulk"], want["bulk"], "bulk")
    _same(got["elastic"], want["elastic"], "elastic", elastic)
    _same(got["anchoring"], want["anchoring"], "anchoring", anchoring)
    _same(got["total"], want["total"], "total", elastic + anchoring)
    for k in ("radiality", "avg_S", "max_S", "checker_rel", "defect_density", "xi_grad_proxy"):
        _same(got[k], want[k], k, 1e-12)
    assert got["nonfinite_cells"] == 0
    assert got["max_q_norm"] == pytest.approx(
        math.sqrt(max((q.reshape(-1, 5) ** 2 @ [1, 2, 2, 1, 2] + (q[0::5] + q[3::5]) ** 2).max(), 0.0)), rel=1e-12)
    solver.close()


@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf])
@pytest.mark.parametrize("component", [0, 4])
def test_infinities_and_nan(oracle, bad, component):
    """One bad cell in the middle of a radial droplet: it is counted, the energies that it enters are not finite, and the counts
    are those of the other cells."""
    op, solver, d = make_pair(**GRIDS["droplet"])
    g, fl = oracle.geometry(op)
    q = fp32(oracle.init(op, g, 1, 1, 0.6))
    cell = 18 + 37 * (12 + 24 * 9)
    q.reshape(-1, 5)[cell, component] = bad
    solver.upload(q)
    got = solver.observe(300.0, 0.6)
    want = oracle.observe(op, g, fl, q, 300.0, 0.6)
    assert got["nonfinite_cells"] == 1
    for k in ("bulk", "elastic", "total", "avg_S", "radiality"):
        assert math.isfinite(got[k]) == math.isfinite(want[k]), (k, got[k], want[k])
    for k in ("radiality_count", "core_count", "defect_plaquettes", "xi_edges", "defect_count"):
        assert got[k] == want[k], k
    assert got["max_S"] == pytest.approx(want["max_S"], rel=1e-10)
    solver.close()


@pytest.mark.parametrize("entry", [1, 2, 4])
def test_periodic_order_of_one_negative_entry(oracle, entry):
    from oracle.oracle import OrcBulkParams
    q = np.zeros((6, 5, 7, 5))
    q[..., entry] = -0.3
    q = fp32(q.ravel())
    s = KZMSolver(7, 5, 6, 1e-8, 1.1e-8, 0.9e-8, 6e-12, 0.1)
    s.upload(q)
    got = s.observe(-9e5, 6e6, 5e6)
    bp = OrcBulkParams()
    for k, v in dict(Nx=7, Ny=5, Nz=6, dx=1e-8, dy=1.1e-8, dz=0.9e-8, kappa=6e-12, gamma=0.1, defects_S_threshold=0.1,
                     defects_charge_cutoff=0.25).items():
        setattr(bp, k, v)
    want = oracle.bulk_observe(bp, q, -9e5, 6e6, 5e6)
    for k in ("bulk", "elastic", "avg_S", "max_S"):
        assert got[k] == pytest.approx(want[k], rel=1e-10, abs=1e-25), k
    assert got["defect_plaquettes_used"] == want["defect_plaquettes_used"]
    s.close()


@pytest.mark.parametrize("name", ["z", "random", "random negative"])
@pytest.mark.parametrize("cut", [1e-6, 0.4999, 0.5001, 0.9999])
def test_periodic_winding_next_to_the_cuts(oracle, name, cut):
    """The winding is a whole number of half turns up to rounding, so cuts of exactly 0, 1/2 and 1 are decided by that rounding;
    next to them every count is determined."""
    from oracle.oracle import OrcBulkParams
    q = fp32(_fields(9 * 8 * 34)[name].ravel())
    s = KZMSolver(34, 8, 9, 1e-8, 1.1e-8, 0.9e-8, 6e-12, 0.1, defects_charge_cutoff=cut)
    s.upload(q)
    got = s.observe(-9e5, 6e6, 5e6)
    bp = OrcBulkParams()
    for k, v in dict(Nx=34, Ny=8, Nz=9, dx=1e-8, dy=1.1e-8, dz=0.9e-8, kappa=6e-12, gamma=0.1, defects_S_threshold=0.1,
                     defects_charge_cutoff=cut).items():
        setattr(bp, k, v)
    want = oracle.bulk_observe(bp, q, -9e5, 6e6, 5e6)
    for k in ("defect_plaquettes_used", "nonzero_defect_plaquettes"):
        assert got[k] == want[k], k
    s.close()
