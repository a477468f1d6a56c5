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


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [(2, 1, 3), (3, 3, 1), (2, 1, 1), (33, 1, 5)])
def test_sgs_edges_of_axes_of_one_cell(n, precision):
    """Order 2: the only interior cell of a periodic axis of three is the source of both
    its edges.  The fields hold NaN beforehand, so that a cell nobody writes shows."""
    from ouxsbli_b200.solver import Solver
    cfg, qj = box(n, order=2, scheme="SLAU", visc="LES", precision=precision)
    s = Solver(cfg)
    s.set_state(qj)
    s.scratch[:10 * s.layout.var_stride // (1 if precision == "fp64" else 2)] = float("nan")
    a, b = (rhs_interior(r, cfg.g, 3) for r in (s.rhs(), oracle.rhs(cfg, qj)))
    if precision == "fp64":
        assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()
    else:
        for l in range(5):
            assert np.abs(a[:, l] - b[:, l]).max() <= 2e-6 * np.abs(qj[:, l]).max()


def box2d(n, order, bc_x=0, bc_y=0, seed=0, boundary=None, **kw):
    """Smooth seeded 2D field on n = (x, y) interior cells."""
    rng = np.random.default_rng(seed)
    g = order // 2
    L = 1.0
    ax, d = [], []
    for m, b in zip(n, (bc_x, bc_y)):
        if b:
            d.append(np.full(m + 1, L / (m + 1)))
            ax.append(np.concatenate([[0.0], np.cumsum(d[-1])]))
        else:
            x, dd = cyclic_axis(m + order, L, order)
            ax.append(x)
            d.append(dd)
    X, Y = np.meshgrid(*[2.0 * math.pi * a / L for a in ax], indexing="ij")
    f = [sum(rng.uniform(-0.2, 0.2) * np.sin(rng.integers(1, 3) * X + rng.integers(-2, 3) * Y + rng.uniform(0, 6))
             for _ in range(4)) for _ in range(4)]
    rho, p = 1.0 + 0.3 * f[0], 1.0 + 0.3 * f[1]
    Q = np.zeros((X.shape[0], 4, X.shape[1]), order="F")
    Q[:, 0], Q[:, 1], Q[:, 2] = rho, rho * f[2], rho * f[3]
    Q[:, 3] = p / 0.4 + 0.5 * rho * (f[2] ** 2 + f[3] ** 2)
    # periodic images along the periodic axes
    for a, (m, b) in enumerate(zip(n, (bc_x, bc_y))):
        if not b:
            i = (np.arange(m + order) - g) % m + g
            Q = np.asfortranarray(np.take(Q, i, axis=0 if a == 0 else 2))
    cfg = SolverConfig(dim=2, nx=X.shape[0], ny=X.shape[1], nz=1, order=order, dt=0.1 * min(x.min() for x in d),
                       gamma=1.4, R=1.0, bc_x=bc_x, bc_y=bc_y, boundary=boundary, dx=d[0], dy=d[1], dz=None, **kw)
    return cfg, to_qj(Q, jacobian(d[0], d[1], None))


@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("scheme,rk", [("KEEP", 4), ("KEEP", 3), ("Hybrid", 3), ("SLAU", 4)])
@pytest.mark.parametrize("n", [(31, 7), (32, 8), (33, 9), (3, 3), (40, 1), (1, 17), (64, 2)])
def test_fused_2d_steps(n, order, scheme, rk):
    """k_stage2d over whole steps, ghost cells included (axes of 2 cells at order 6 keep the
    separate passes, whose outer images are ghost cells themselves)."""
    from ouxsbli_b200.solver import Solver
    if (order == 6 and 2 in n) or n[0] + order < 4:
        pytest.skip("no defined image for the outer ghost cells, or below the smallest grid")
    cfg, qj = box2d(n, order, scheme=scheme, visc="Euler", rk=rk)
    s = Solver(cfg)
    s.set_state(qj)
    s.step(2)
    assert np.array_equal(s.get_state(), oracle.step(cfg, qj, 2))


@pytest.mark.parametrize("y_last", [False, True])
@pytest.mark.parametrize("n,bc", [((31, 8), (1, 0)), ((33, 9), (0, 1)), ((2, 2), (1, 1)), ((40, 17), (1, 1))])
def test_fused_2d_boundaries(n, bc, y_last):
    from ouxsbli_b200.solver import Solver
    rules = {}
    if bc[0]:
        rules.update(x_lo="slip_wall", x_hi="neumann")
    if bc[1]:
        rules.update(y_lo="noslip_wall", y_hi="zero_gradient")
    cfg, qj = box2d(n, 6, *bc, boundary=rules, scheme="Hybrid", visc="Euler", rk=3,
                    boundary_order="y_last" if y_last else "x_last")
    qj = oracle.fill_ghosts(cfg, qj)
    s = Solver(cfg)
    s.set_state(qj)
    s.step(3)
    assert np.array_equal(s.get_state(), oracle.step(cfg, qj, 3))


@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("scheme,rk", [("KEEP", 4), ("Hybrid", 3)])
@pytest.mark.parametrize("n,bc", [((33, 9), (0, 0)), ((40, 1), (0, 0)), ((31, 17), (1, 1))])
def test_fused_2d_mixed(n, bc, scheme, rk, order):
    """The mixed form: three steps round the increments of 3 rk stages to FP32 (6e-8 of an
    increment that is at most 10 % of the state), and the fluxes to a few FP32 ulps."""
    from ouxsbli_b200.solver import Solver
    rules = {"x_lo": "slip_wall", "y_lo": "noslip_wall"} if bc[0] else None
    cfg, qj = box2d(n, order, *bc, boundary=rules, scheme=scheme, visc="Euler", rk=rk, precision="mixed")
    qj = oracle.fill_ghosts(cfg, qj)
    s = Solver(cfg)
    s.set_state(qj)
    s.step(3)
    a, b = s.get_state(), oracle.step(cfg, qj, 3)
    for l in range(4):
        assert np.abs(a[:, l] - b[:, l]).max() <= 2e-6 * np.abs(b).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scheme,rk", [("KEEP", 4), ("SLAU", 3)])
@pytest.mark.parametrize("n", [(60011, 1), (1, 14501), (3, 15001), (17, 58001)])
def test_long_narrow_2d_steps(n, scheme, rk, precision):
    """Both routes of a long grid a few cells wide (1876 to 7251 tiles): fused stages for
    FP64 KEEP, separate passes for the others from the padding on where those are faster."""
    from ouxsbli_b200.solver import Solver
    cfg, qj = box2d(n, 6, scheme=scheme, visc="Euler", rk=rk, precision=precision)
    s = Solver(cfg)
    s.set_state(qj)
    before = s.launches()
    s.step(1)
    fused = (scheme == "KEEP" and (precision == "fp64" or n == (17, 58001))) or (precision == "fp64" and n == (17, 58001))
    assert (s.launches() - before == rk) == fused
    a, b = s.get_state(), oracle.step(cfg, qj, 1)
    if precision == "fp64":
        assert np.array_equal(a, b)
    else:
        for l in range(4):
            assert np.abs(a[:, l] - b[:, l]).max() <= 2e-6 * np.abs(b).max()


# ---- marching sweeps (oux_march.cuh): from 370 000 interior cells (FP64; x and y), 6 000 000 (z, ME4), mixed 100 000 and 11 000 000 ----
# extents one past, at and short of 32 columns (x, z) and of 8 (y), segments of one row and of
# odd lengths, axes of 1 to 3 cells, rows longer than a warp's ring
# few long rows (x on tiles), one plane of many rows, one line of columns split along y
XY_SIZES = [(33, 109, 107), (31, 113, 110), (512, 28, 27), (95, 3, 1340), (3, 350, 366), (620, 613, 1),
            (2048, 14, 14), (330, 1301, 1), (10, 38001, 1)]
Z_SIZES = [(97, 251, 249), (33, 430, 426), (1, 2457, 2443), (70, 301, 287), (24, 509, 493)]


@pytest.mark.parametrize("n", XY_SIZES + Z_SIZES)
def test_marching_sweeps_me4(n):
    cfg, qj = box(n, scheme="Hybrid", visc="NS", visc_stencil="ME4Base")
    a, b = residuals(cfg, qj)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("kw", [
    dict(scheme="SLAU", visc="NS"), dict(scheme="KEEP", visc="NS", rk=4), dict(scheme="Roe", visc="NS", visc_order=4),
    dict(scheme="Hybrid", visc="NS", visc_stencil="ME4Base", stretch=True),
    dict(order=4, scheme="Hybrid", visc="NS", visc_order=4)])
@pytest.mark.parametrize("n", [(65, 77, 79), (97, 113, 111)])
def test_marching_sweeps_stencils(n, kw):
    cfg, qj = box(n, **kw)
    a, b = residuals(cfg, qj)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("rk", [3, 4])
@pytest.mark.parametrize("n", [(65, 77, 79), (182, 184, 183)])
def test_marching_sweeps_stage_combinations(n, rk):
    """Whole steps: the z sweep's combinations of RK3 and RK4 with their operands."""
    from ouxsbli_b200.solver import Solver
    cfg, qj = box(n, scheme="Hybrid", visc="NS", visc_stencil="ME4Base", rk=rk)
    s = Solver(cfg)
    s.set_state(qj)
    s.step(1)
    assert np.array_equal(s.get_state(), oracle.step(cfg, qj, 1))


@pytest.mark.parametrize("n,stencil", [((65, 77, 79), "Central"), ((97, 113, 111), "Central"), ((65, 77, 79), "ME4Base"),
                                       ((97, 113, 111), "ME4Base"), ((182, 184, 183), "ME4Base")])
def test_marching_sweeps_les(n, stencil):
    cfg, qj = box(n, scheme="SLAU", visc="LES", visc_stencil=stencil)
    a, b = residuals(cfg, qj)
    assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()


@pytest.mark.parametrize("n,rk", [((65, 77, 79), 3), ((65, 77, 79), 4), ((225, 223, 221), 3)])
def test_marching_sweeps_mixed(n, rk):
    """One mixed step: increments rounded to FP32 and FP32 fluxes of smooth fields, as above."""
    from ouxsbli_b200.solver import Solver
    cfg, qj = box(n, scheme="KEEP", visc="NS", visc_stencil="ME4Base", rk=rk, precision="mixed")
    s = Solver(cfg)
    s.set_state(qj)
    s.step(1)
    a, b = s.get_state(), oracle.step(cfg, qj, 1)
    for l in range(5):
        assert np.abs(a[:, l] - b[:, l]).max() <= 2e-6 * np.abs(b[:, 1:4] if 1 <= l <= 3 else b[:, l]).max()


@pytest.mark.parametrize("n,kw", [
    ((65, 77, 79), dict(scheme="Hybrid", visc="NS")), ((65, 77, 79), dict(scheme="Hybrid", visc="NS", visc_stencil="ME4Base")),
    ((65, 77, 79), dict(scheme="SLAU", visc="LES")), ((65, 77, 79), dict(scheme="SLAU", visc="LES", visc_stencil="ME4Base")),
    ((225, 223, 221), dict(scheme="Hybrid", visc="NS")), ((225, 223, 221), dict(scheme="SLAU", visc="LES")),
    ((225, 223, 221), dict(scheme="SLAU", visc="LES", visc_stencil="ME4Base"))])
def test_marching_sweeps_mixed_switches(n, kw):
    """Mixed residuals of the schemes that switch (sensor threshold, limiters, the HRSLAU2
    and SMS switches): a face whose switch argument lies within FP32 rounding of its
    threshold may take the other side.  An argument spread over a range of order one falls
    that close with probability about 1e-6 a switch; with some ten switches on the 6 faces
    of a cell fewer than 1e-4 of the cells may differ by more than rounding."""
    cfg, qj = box(n, precision="mixed", **kw)
    a, b = residuals(cfg, qj)
    far = np.zeros(a[:, 0].shape, bool)
    for l in range(5):
        far |= ~(np.abs(a[:, l] - b[:, l]) <= 2e-6 * np.abs(qj[:, l]).max())
    assert far.mean() <= 1e-4


def test_marching_and_tile_parts_of_a_z_slab():
    """Two z slabs of 48 planes: a stage's interior part marches (387 072 cells), the parts
    next to its ends take tiles; the undivided solve marches throughout.  Same bits."""
    from ouxsbli_b200.slabs import LocalSlabs
    from ouxsbli_b200.solver import Solver
    cfg, qj = box((96, 96, 96), scheme="Hybrid", visc="NS", visc_stencil="ME4Base")
    s = Solver(cfg)
    s.set_state(qj)
    s.step(2)
    slabs = LocalSlabs(cfg, 2, "cuda:0")
    slabs.set_state(qj)
    slabs.step(2)
    g = cfg.g
    assert np.array_equal(slabs.get_state()[:, :, :, g:-g], s.get_state()[:, :, :, g:-g])
    slabs.close()


@pytest.mark.parametrize("n,stencil", [((97, 115, 111), "Central"), ((97, 115, 111), "ME4Base"), ((225, 225, 223), "Central"),
                                       ((225, 225, 223), "ME4Base")])
def test_marching_sweeps_mixed_walls(n, stencil):
    """Mixed marches between walls (KEEP: no switches), held as the periodic ones."""
    from helpers import wall_box
    from ouxsbli_b200.solver import Solver
    cfg, qj, _ = wall_box(*n, 6, {"y_lo": "noslip_wall", "y_hi": "noslip_wall", "z_lo": "slip_wall", "z_hi": "noslip_wall"},
                          bc_z=1, scheme="KEEP", visc="NS", visc_stencil=stencil, precision="mixed")
    qj = oracle.fill_ghosts(cfg, qj)
    s = Solver(cfg)
    s.set_state(qj)
    x = slice(cfg.g - 1, 1 - cfg.g)  # the interior of the periodic axis
    a, b = s.rhs()[x], oracle.rhs(cfg, qj)[x]
    for l in range(5):
        assert np.abs(a[:, l] - b[:, l]).max() <= 2e-6 * np.abs(qj[:, 1:4] if 1 <= l <= 3 else qj[:, l]).max()


@pytest.mark.parametrize("stencil,visc", [("Central", "NS"), ("ME4Base", "NS"), ("Central", "LES")])
def test_marching_sweeps_walls(stencil, visc):
    """Walls on every axis: the order fallback and the 2nd-order viscous faces."""
    from helpers import wall_box
    rules = {"x_lo": "slip_wall", "x_hi": "slip_wall", "y_lo": "noslip_wall", "y_hi": "noslip_wall",
             "z_lo": "slip_wall", "z_hi": "noslip_wall"}
    cfg, qj, _ = wall_box(97, 115, 111, 6, rules, bc_x=1, bc_z=1, scheme="Hybrid", visc=visc, visc_stencil=stencil)
    from ouxsbli_b200.solver import Solver
    qj = oracle.fill_ghosts(cfg, qj)
    s = Solver(cfg)
    s.set_state(qj)
    a, b = s.rhs(), oracle.rhs(cfg, qj)
    if visc == "LES":
        assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()
    else:
        assert np.array_equal(a, b)
