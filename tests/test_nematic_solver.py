"""The log points' eigen-solver (matrix powers) against the reference's own 15 normalised power steps
(QSR.cu:191-243), on the tensors where a start vector has no share of the largest eigenvector."""
import itertools

import numpy as np
import pytest

from device_math import build, nematic


@pytest.fixture(scope="module")
def math(tmp_path_factory):
    return build(tmp_path_factory.mktemp("device_math"))


def steps15(q, iso_cut):
    xx, xy, xz, yy, yz = (float(v) for v in q)
    if all(abs(v) < iso_cut for v in (xx, xy, xz, yy, yz)):
        return np.array([0.0, 0.0, 0.0, 1.0])
    Q = np.array([[xx, xy, xz], [xy, yy, yz], [xz, yz, -xx - yy]])
    n = np.array([xx + xy + xz, xy + yy + yz, xz + yz - xx - yy])
    r = np.sqrt(n @ n)
    n = n / r if r > 1e-12 else np.array([0.0, 0.0, 1.0])
    alpha = np.abs(Q).sum(axis=1).max() + 1e-12
    for _ in range(15):
        a = np.array([Q[i, 0] * n[0] + Q[i, 1] * n[1] + Q[i, 2] * n[2] + alpha * n[i] for i in range(3)])
        r = np.sqrt(a @ a)
        if r < 1e-13:
            break
        n = a / r
    if n[2] < 0:
        n = -n
    return np.array([1.5 * (n @ Q @ n), *n])


def compare(math, q, iso_cut, tol):
    got = nematic(math, q, iso_cut)
    want = np.array([steps15(t, iso_cut) for t in q])
    assert np.isfinite(got).all()
    scale = np.abs(q).max(axis=1)
    assert (np.abs(got[:, 0] - want[:, 0]) <= tol * scale).all()
    # the director up to its sign (a sign that rounding gives where nz is 0 is no difference)
    assert (1.0 - np.abs((got[:, 1:] * want[:, 1:]).sum(axis=1)) <= tol).all()


@pytest.mark.parametrize("S", [-0.5, -0.3, -0.25, -1e-3, 0.5, 0.3])
def test_uniaxial_along_the_diagonals(math, S):
    d = np.array(list(itertools.product((-1.0, 0.0, 1.0), repeat=3)))
    d = d[(d != 0).any(axis=1)]
    d /= np.sqrt((d * d).sum(axis=1))[:, None]
    q = S * np.stack([d[:, 0] ** 2 - 1 / 3, d[:, 0] * d[:, 1], d[:, 0] * d[:, 2], d[:, 1] ** 2 - 1 / 3,
                      d[:, 1] * d[:, 2]], axis=1)
    compare(math, q.astype(np.float32).astype(np.float64), 1e-9, 1e-12)


@pytest.mark.parametrize("a", [0.1, 0.25, 0.3, 1e-6])
def test_single_entries_of_either_sign(math, a):
    q = np.array([[s * a if i == m else 0.0 for i in range(5)] for m in range(5) for s in (-1.0, 1.0)])
    compare(math, q.astype(np.float32).astype(np.float64), 1e-9, 1e-12)


def test_tensors_at_the_early_stop(math):
    rng = np.random.default_rng(5)
    compare(math, rng.uniform(-4e-12, 4e-12, (400, 5)), 1e-12, 1e-9)


def test_general_tensors(math):
    rng = np.random.default_rng(6)
    compare(math, rng.normal(size=(2000, 5)) * 0.3, 1e-9, 1e-9)
