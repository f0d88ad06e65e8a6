"""The periodic step at box sizes around its tile (32 x 8 columns), with row lengths that are and are not a multiple
of the 16-byte copy, and with every chunk length the size picks, against the FP64 oracle and the one-thread-per-site
kernel (GPU).

Tolerances: four steps without noise from an FP32-representable field against FP64, <= 2e-6 of max |Q|; with noise
against the one-thread-per-site kernel (the same draws, other rounding order), <= 2e-6.
"""
import os

import numpy as np
import pytest

from gpu_helpers import fp32, rel_err
from lcdrsimulator_b200 import KZMSolver
from lcdrsimulator_b200.physics import bulk_ABC

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 2), (3, 2, 5), (5, 9, 4), (31, 7, 6), (32, 8, 8), (33, 17, 3), (36, 10, 70), (65, 24, 33), (130, 9, 12)]


def _solver(n):
    return KZMSolver(*n, 1e-8, 1.1e-8, 0.9e-8, 6e-12, 0.1)


@pytest.mark.parametrize("n", SIZES)
def test_periodic_step_sizes(n):
    A, B, C = bulk_ABC(0.044e6, 1.413e6, 1.153e6, 300.0, 307.0)
    rng = np.random.default_rng(3)
    q0 = fp32(0.2 * rng.standard_normal(5 * n[0] * n[1] * n[2]))
    dt = 1e-9
    s = _solver(n)
    s.upload(q0)
    s.step(4, A, B, C, dt)
    got = s.download()
    # FP64 on the host: the reference's periodic update
    q = q0.reshape(n[2], n[1], n[0], 5).copy()
    for _ in range(4):
        lap = sum((np.roll(q, 1, a) + np.roll(q, -1, a) - 2 * q) / h ** 2 for a, h in ((2, 1e-8), (1, 1.1e-8), (0, 0.9e-8)))
        xx, xy, xz, yy, yz = (q[..., m] for m in range(5))
        zz = -xx - yy
        tr = xx ** 2 + yy ** 2 + zz ** 2 + 2 * (xy ** 2 + xz ** 2 + yz ** 2)
        g = A + C * tr
        h = np.stack([g * xx - B * (xx * xx + xy * xy + xz * xz - tr / 3), g * xy - B * (xx * xy + xy * yy + xz * yz),
                      g * xz - B * (xx * xz + xy * yz + xz * zz), g * yy - B * (xy * xy + yy * yy + yz * yz - tr / 3),
                      g * yz - B * (xy * xz + yy * yz + yz * zz)], -1) - 6e-12 * lap
        q = q - dt / 0.1 * h
    assert rel_err(got, q.ravel()) <= 2e-6
    # noise: the same draws as the one-thread-per-site kernel
    s.upload(q0)
    s.step(3, A, B, C, dt, noise_sigma=1e-3, seed=5, step_index=7)
    a = s.download()
    s.upload(q0)
    os.environ["LDG_KZM_KERNEL"] = "direct"
    try:
        s.step(3, A, B, C, dt, noise_sigma=1e-3, seed=5, step_index=7)
    finally:
        del os.environ["LDG_KZM_KERNEL"]
    assert rel_err(a, s.download()) <= 2e-6
    s.close()
