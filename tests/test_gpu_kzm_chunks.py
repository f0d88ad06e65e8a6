"""The periodic step with every length of its plane chunks from one plane to the whole box: slots of the plane ring that are
never refilled, refilled once, and refilled with either parity, and last chunks that are shorter (GPU).

Four steps without noise from an FP32-representable field against FP64, three steps with noise against the
one-thread-per-site kernel (the same draws): <= 2e-6 of max |Q| each, a handful of FP32 roundings of 6e-8 per step.
"""
import numpy as np
import pytest

from gpu_helpers import fp32, rel_err
from lcdrsimulator_b200 import KZMSolver
from lcdrsimulator_b200.physics import bulk_ABC

pytestmark = pytest.mark.gpu

H, KAPPA, GAMMA, DT = (1e-8, 1.1e-8, 0.9e-8), 6e-12, 0.1, 1e-9
ABC = bulk_ABC(0.044e6, 1.413e6, 1.153e6, 300.0, 307.0)


def _update64(q, n, steps):
    A, B, C = ABC
    q = q.reshape(n[2], n[1], n[0], 5).copy()
    for _ in range(steps):
        lap = sum((np.roll(q, 1, a) + np.roll(q, -1, a) - 2 * q) / h ** 2 for a, h in zip((2, 1, 0), H))
        xx, xy, xz, yy, yz = (q[..., m] for m in range(5))
        Q = [[xx, xy, xz], [xy, yy, yz], [xz, yz, -xx - yy]]
        tr = sum(Q[a][b] * Q[b][a] for a in range(3) for b in range(3))
        sq = [[sum(Q[a][c] * Q[c][b] for c in range(3)) - (tr / 3 if a == b else 0) for b in range(3)] for a in range(3)]
        h = [(A + C * tr) * Q[a][b] - B * sq[a][b] for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2))]
        q = q - DT / GAMMA * (np.stack(h, -1) - KAPPA * lap)
    return q.ravel()


def _check(n, monkeypatch):
    q0 = fp32(0.2 * np.random.default_rng(3).standard_normal(5 * n[0] * n[1] * n[2]))
    s = KZMSolver(*n, *H, KAPPA, GAMMA)
    s.upload(q0)
    s.step(4, *ABC, DT)
    assert rel_err(s.download(), _update64(q0, n, 4)) <= 2e-6
    s.upload(q0)
    s.step(3, *ABC, DT, noise_sigma=1e-3, seed=5, step_index=7)
    got = s.download()
    s.upload(q0)
    monkeypatch.setenv("LDG_KZM_KERNEL", "direct")
    s.step(3, *ABC, DT, noise_sigma=1e-3, seed=5, step_index=7)
    assert rel_err(got, s.download()) <= 2e-6
    s.close()


@pytest.mark.parametrize("planes", [1, 2, 3, 4, 5, 7, 8, 12, 32, 70])
@pytest.mark.parametrize("n", [(33, 17, 70), (65, 24, 33)])
def test_chunk_lengths(n, planes, monkeypatch):
    monkeypatch.setenv("LDG_KZM_PLANES", str(planes))
    _check(n, monkeypatch)


def test_the_length_that_a_large_box_picks(monkeypatch):
    monkeypatch.delenv("LDG_KZM_PLANES", raising=False)
    _check((128, 120, 130), monkeypatch)
