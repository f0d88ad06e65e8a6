"""Rounding of the step kernels' packed chemical potential against FP64: no larger than that of the term-by-term form
(QSR.cu:373-621) which the one-thread-per-cell kernel keeps."""
import numpy as np
import pytest

from device_math import build, chem

DX = 1e-8
N = 18


@pytest.fixture(scope="module")
def math(tmp_path_factory):
    return build(tmp_path_factory.mktemp("device_math"))


def field(seed, S, rough):
    rng = np.random.default_rng(seed)
    x = np.arange(N) * 0.15
    X, Y, Z = np.meshgrid(x, x, x, indexing="ij")
    k = rng.normal(size=4)
    th, ph = k[0] * X + k[1] * Y + k[2] * Z + 3 * k[3], k[1] * X - k[0] * Y + 0.5 * Z + 1
    d = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)])
    s = S * (1 + 0.1 * np.sin(X + Y))
    q = np.stack([s * (d[0] ** 2 - 1 / 3), s * d[0] * d[1], s * d[0] * d[2], s * (d[1] ** 2 - 1 / 3), s * d[1] * d[2]])
    return np.ascontiguousarray((q + rough * S * rng.normal(size=q.shape)).astype(np.float32))


def exact(q, e):
    """The chemical potential in FP64 on cells 2 .. N - 3."""
    L1, L2, L3, A, B, Cc = e
    q = q.astype(np.float64)
    full = np.array([[q[0], q[1], q[2]], [q[1], q[3], q[4]], [q[2], q[4], -q[0] - q[3]]])
    c = slice(2, N - 2)

    def at(f, *steps):
        o = [0, 0, 0]
        for ax, by in steps:
            o[ax] += by
        return f[..., 2 + o[0]:N - 2 + o[0], 2 + o[1]:N - 2 + o[1], 2 + o[2]:N - 2 + o[2]]

    Q = at(full)

    def d1(a):
        return (at(full, (a, 1)) - at(full, (a, -1))) / (2 * DX)

    def d2(a, b):
        if a == b:
            return (at(full, (a, 1)) + at(full, (a, -1)) - 2 * Q) / DX ** 2
        return (at(full, (a, 1), (b, 1)) - at(full, (a, 1), (b, -1)) - at(full, (a, -1), (b, 1)) +
                at(full, (a, -1), (b, -1))) / (4 * DX ** 2)

    def wide(a, b):
        return (at(full, (a, 2)) + at(full, (a, -2)) - 2 * Q) / (4 * DX ** 2) if a == b else d2(a, b)

    eye = np.eye(3)[:, :, None, None, None]
    Q2 = np.einsum("ac...,cb...->ab...", Q, Q)
    tr = np.einsum("aa...->...", Q2)
    h = A * Q - B * (Q2 - eye * tr / 3) + Cc * tr * Q - L1 * (d2(0, 0) + d2(1, 1) + d2(2, 2))
    if L2:
        g = np.array([[sum(wide(k, a)[k, b] for k in range(3)) for b in range(3)] for a in range(3)])  # d_a D_b
        for a in range(3):
            for b in range(3):
                h[a, b] -= L2 * (g[a, a] if a == b else g[a, b] + g[b, a])
    h = h - eye * np.einsum("aa...->...", h) / 3
    if L3:
        g = [d1(a) for a in range(3)]
        D = [sum(g[k][k, b] for k in range(3)) for b in range(3)]
        Bq = sum(D[a] * g[a] for a in range(3)) + sum(Q[a, b] * d2(a, b) for a in range(3) for b in range(3))
        M = np.array([[(g[a] * g[b]).sum(axis=(0, 1)) for b in range(3)] for a in range(3)])
        h = h + 0.5 * L3 * M - L3 * Bq
        h = h - eye * np.einsum("aa...->...", h) / 3
    return np.stack([h[0, 0], h[0, 1], h[0, 2], h[1, 1], h[1, 2]]), c


@pytest.mark.parametrize("S,rough", [(0.5, 0.0), (0.5, 0.05), (0.2, 0.01)])
@pytest.mark.parametrize("L", [(0.0, 0.0, 0.0), (6e-12, 0.0, 0.0), (6e-12, 3e-12, 0.0), (6e-12, 0.0, 1e-12),
                               (6e-12, 3e-12, 1e-12)])
def test_packed_form_rounds_no_more_than_the_terms(math, L, S, rough):
    T, a, b, cc = 302.0, 0.044e6, 1.413e6, 1.153e6
    packed = terms = 0.0
    for seed in range(6):
        k = (1.0, 1.0, 1.0) if seed % 2 else (3.0, 4.5, 4.5)  # the two conventions of the bulk energy
        e = (*L, k[0] * a * (T - 307.0), k[1] * b, k[2] * cc)
        q = field(seed, S, rough)
        want, c = exact(q, e)
        for form in (True, False):
            got = chem(math, q, DX, e, form)[:, c, c, c].astype(np.float64)
            assert np.isfinite(got).all()
            assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()  # the same quantity
            sq = float(((got - want) ** 2).sum())
            packed, terms = (packed + sq, terms) if form else (packed, terms + sq)
    assert np.sqrt(packed) <= np.sqrt(terms), (np.sqrt(packed), np.sqrt(terms), np.sqrt(packed / terms))
