"""Kernels that work on tiles, at the sizes where a tile's edges can go wrong: one cell
past, at and short of a tile, the smallest grids, and axes of uneven spacing.

Reference: the CPU oracle.  FP64 without LES is bit for bit; LES differs by the last ulps
of pow / log / cosh (and of the square roots that replace pow), held to 1e-11 of the
residual's maximum as in test_gpu_parity.py; the mixed form is held to FP32 rounding
of its fields (2^-24 relative, amplified by at most a few tens in the face
differences of these smooth fields): 2e-6 of the residual's maximum.
"""
import math

import numpy as np
import pytest

from helpers import rhs_interior
from oracle import oracle
from ouxsbli_b200.grid import cyclic_axis, fill_periodic, jacobian, to_qj
from ouxsbli_b200.solver import SolverConfig

pytestmark = pytest.mark.gpu


def box(n, order=6, seed=0, stretch=False, mach=0.8, **kw):
    """Smooth seeded field on n = (x, y, z) interior cells of a periodic box; stretch:
    spacings that vary by 10 % along every axis."""
    rng = np.random.default_rng(seed)
    g = order // 2
    L, T0, R, gam = 1.0e-3, 300.0, 287.03, 1.4
    c0 = math.sqrt(gam * R * T0)
    ax = [cyclic_axis(m + order, L, order) for m in n]
    d = [a[1].copy() for a in ax]
    if stretch:
        d = [x * (1.0 + 0.1 * np.sin(2.0 * math.pi * np.arange(x.size) / m)) for x, m in zip(d, n)]
    X, Y, Z = np.meshgrid(*[2.0 * math.pi * a[0] / L for a in ax], indexing="ij")
    f = [np.zeros_like(X) for _ in range(5)]
    for _ in range(5):
        k = rng.integers(-2, 3, 3)
        ph = k[0] * X + k[1] * Y + k[2] * Z + rng.uniform(0, 6.0)
        for q in range(5):
            f[q] = f[q] + rng.uniform(-0.3, 0.3) * np.sin(ph + q)
    rho = 0.05 * (1.0 + 0.1 * f[0])
    p = 0.05 * R * T0 * (1.0 + 0.1 * f[1])
    vel = [0.3 * mach * c0 * f[2 + a] for a in range(3)]
    Q = np.zeros((X.shape[0], 5) + X.shape[1:], order="F")
    Q[:, 0] = rho
    for a in range(3):
        Q[:, 1 + a] = rho * vel[a]
    Q[:, 4] = p / (gam - 1.0) + 0.5 * rho * sum(v * v for v in vel)
    fill_periodic(Q, g)
    dt = 0.2 * min(x.min() for x in d) / (2.0 * c0)
    cfg = SolverConfig(dim=3, nx=X.shape[0], ny=X.shape[1], nz=X.shape[2], order=order, dt=dt, gamma=gam, R=R, Pr=0.71,
                       Prt=0.9, dx=d[0], dy=d[1], dz=d[2], **kw)
    return cfg, to_qj(Q, jacobian(*d))


def residuals(cfg, qj):
    """Interior residuals of the GPU and of the oracle."""
    from ouxsbli_b200.solver import Solver
    s = Solver(cfg)
    s.set_state(qj)
    return tuple(rhs_interior(r, cfg.g, 3) for r in (s.rhs(), oracle.rhs(cfg, qj)))


# interior extents: x around one and two 32-wide tiles, y around 8, z around 4, and the smallest grid
POINTWISE = [(26, 2, 1), (27, 3, 2), (28, 10, 6), (59, 11, 7), (1, 1, 1)]


@pytest.mark.parametrize("n", POINTWISE)
def test_primitive_and_sensor_tiles(n):
    """k_prim_fused (FP64: the 3D Euler sensor schemes)."""
    cfg, qj = box(n, scheme="Hybrid", visc="Euler")
    a, b = residuals(cfg, qj)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [m for m in POINTWISE if m != (1, 1, 1)])
def test_primitive_and_sensor_tiles_mixed(n):
    cfg, qj = box(n, scheme="Hybrid", visc="NS", precision="mixed")
    a, b = residuals(cfg, qj)
    for l in range(5):
        assert np.abs(a[:, l] - b[:, l]).max() <= 2e-6 * np.abs(qj[:, l]).max()


@pytest.mark.parametrize("stretch", [False, True])
@pytest.mark.parametrize("n", [(26, 2, 1), (27, 3, 2), (28, 5, 3), (1, 1, 1), (59, 9, 5)])
def test_sgs_viscosity_tiles(n, stretch):
    """k_mut with its edge cells; delta from the host (uniform) or per cell (stretched)."""
    cfg, qj = box(n, scheme="SLAU", visc="LES", stretch=stretch)
    a, b = residuals(cfg, qj)
    assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()
