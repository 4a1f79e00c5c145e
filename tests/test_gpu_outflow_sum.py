"""The outflow sum (cmass2d) for each of its block sizes, one class and more
than a group of loads, terms of both signs over twelve decades: the exact sum
of the rounded terms, rounded once.  A sum of N terms kept in twice the working
precision is off by at most (N*2^-53)^2 of the sum of their magnitudes."""
import math

import numpy as np
import pytest

import fall3d_gb300 as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,nc", [(3, 3, 3, 1), (30, 20, 9, 9), (150, 120, 10, 1), (150, 120, 10, 10),
                                         (200, 150, 20, 3)])
def test_outflow_is_the_exact_sum(nx, ny, nz, nc):
    r = np.random.default_rng(nx + nc)
    c = r.random((nc, nz + 2, ny + 2, nx + 2)) * 10.0 ** r.uniform(-9, 3, (nc, nz + 2, ny + 2, nx + 2))
    c[r.random(c.shape) < 0.3] = 0.0
    vx, vy, vz = (r.uniform(-30.0, 30.0, (nz, ny, nx)) for _ in range(3))
    vset = -r.uniform(0.0, 3.0, (nc, nz, ny, nx))
    dz = r.uniform(100.0, 700.0, nz + 1)
    dx, dy, dt = 2000.0, 1800.0, 13.0
    fx, fy = np.ones(nx), np.ones(ny)
    fx[[0, -1]] = fy[[0, -1]] = 0.5
    k = np.arange(1, nz + 1)
    terms = []
    for side in (0, 1):
        w = dt * (fy[None, :] * dy * 0.5 * (dz[k] + dz[k - 1])[:, None]) * vx[:, :, -side]
        terms.append((w if side else -w)[None] * c[:, 1:-1, 1:-1, (nx + 1) * side])
        w = dt * (fx[None, :] * dx * 0.5 * (dz[k] + dz[k - 1])[:, None]) * vy[:, -side, :]
        terms.append((w if side else -w)[None] * c[:, 1:-1, (ny + 1) * side, 1:-1])
    area = dt * (fx[None, :] * fy[:, None] * dx * dy)
    terms.append(area[None] * (vz[-1][None] + vset[:, -1]) * c[:, -1, 1:-1, 1:-1])
    t = np.concatenate([v.ravel() for v in terms])
    want = math.fsum(t)
    got = F.cmass2d(np.ascontiguousarray(c), *(np.ascontiguousarray(v) for v in (vx, vy, vz, vset)), nx, ny, nz, nc, 1,
                    nc, 1, nz, dx, dy, dz, dt, 0.0)
    assert abs(got - want) <= 2.0 ** -52 * abs(want) + (t.size * 2.0 ** -53) ** 2 * math.fsum(np.abs(t))
