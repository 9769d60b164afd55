"""The limiter's two launch forms (a quad per element, and a block scan that lists the elements
to rewrite) at the sizes where they change over, and the positivity bisection against a plain one."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAMMA = 1.4
STEPS = 60


def _pressure(q):
    return (GAMMA - 1.0) * (q[..., 3] - 0.5 * (q[..., 1] * (q[..., 1] / q[..., 0]) + q[..., 2] * (q[..., 2] / q[..., 0])))


def _average(q, weights):
    s = weights[0] * q[0]
    for i in range(1, len(weights)):
        s = s + weights[i] * q[i]
    return s


def _positivity(q, avg):
    """limiting.py:166-200 of CFD-demo, every operation rounded to double."""
    eps = np.minimum(1e-13, np.minimum(avg[:, 0], _pressure(avg)))
    rmin = q[..., 0].min(axis=0)
    thin = rmin < eps
    theta = np.clip((avg[:, 0] - eps) / np.where(thin, avg[:, 0] - rmin, 1.0), 0.0, 1.0)
    q = np.where(thin[None, :, None], avg + theta[None, :, None] * (q - avg), q)
    need = _pressure(q) < eps
    dev = q - avg
    lo, hi = np.zeros(q.shape[:2]), np.ones(q.shape[:2])
    for _ in range(STEPS):
        mid = 0.5 * (lo + hi)
        ok = _pressure(avg + mid[..., None] * dev) >= eps
        lo, hi = np.where(ok, mid, lo), np.where(ok, hi, mid)
    theta = np.where(need, lo, 1.0).min(axis=0)
    return np.where((theta < 1.0)[None, :, None], avg + theta[None, :, None] * dev, q), int(need.any(axis=0).sum())


# 14,000 elements is the largest mesh of the quad form; 1 x 1 the smallest, 7 x 5 and 7001 x 1 ragged
@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 5), (140, 50), (7001, 1)])
@pytest.mark.parametrize("scale", [1.0, 1e-4, 30.0])
def test_positivity_bisection_is_the_plain_one_bit_for_bit(nx, ny, scale):
    """The pressure scaling skips the halvings whose outcome is certain; the state it leaves is that of
    sixty plain halvings in the same operation order, to the last bit (no tolerance: the operations are
    the same ones). Nodes far below the floor, slightly below it, and dense and thin averages."""
    from cfd_demo_b200 import EulerSolver, SlipWall, SolverConfig, rectangle_mesh

    mesh = rectangle_mesh(nx, ny)
    s = EulerSolver(mesh, {t: SlipWall() for t in ("left", "right", "bottom", "top")},
                    SolverConfig(flux="rusanov", limiter="unlimited", gamma=GAMMA))
    rng = np.random.default_rng(nx + ny)
    k = mesh.num_elements
    rho = 10.0 ** rng.uniform(-3, 1, size=(1, k)) * (1.0 + 0.5 * rng.uniform(-1, 1, size=(15, k)))
    u, v = scale * rng.normal(size=(2, 15, k)) * rng.choice([0.0, 0.01, 1.0], size=(2, 1, k))
    p = 10.0 ** rng.uniform(-4, 1, size=(1, k)) * (1.0 + rng.uniform(0.0, 4.0, size=(1, k)) * rng.uniform(-1, 1, size=(15, k)))
    q = np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], axis=-1)
    w = s.reference.cell_weights / s.reference.cell_weights.sum()
    avg = _average(q, w)
    keep = (avg[:, 0] > 0) & (_pressure(avg) > 0)
    q[:, ~keep] = (1.0, 0.1, 0.2, 2.5)
    want, scaled = _positivity(q, _average(q, w))
    assert np.array_equal(s.limit(q), want)
    if k > 60:
        assert scaled > k // 20


@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
@pytest.mark.parametrize("nx,ny", [(7000, 1), (7001, 1), (350, 20), (351, 20)])
def test_limiter_forms_match_the_oracle_across_their_boundary(nx, ny, precision):
    """limit() on both sides of the form's size rule against the oracle (1e-12 of each variable in
    FP64; in FP32-mixed 2e-5, a hundred single roundings, on the elements whose troubled decision the
    wider detection threshold leaves alike), the same troubled count in FP64."""
    import oracle
    from cfd_demo_b200 import EulerSolver, SlipWall, SolverConfig, rectangle_mesh

    mesh = rectangle_mesh(nx, ny)
    wall = {t: SlipWall() for t in ("left", "right", "bottom", "top")}
    s = EulerSolver(mesh, wall, SolverConfig(flux="rusanov", limiter="mc", gamma=GAMMA, precision=precision))
    om = oracle.mesh.TriangleMesh(np.array(mesh.vertices), np.array(mesh.elements),
                                  {t: np.array(e) for t, e in mesh.boundary_edges.items()})
    o = oracle.OracleSolver(om, {t: oracle.physics.SlipWall() for t in wall}, flux="rusanov", limiter="mc", gamma=GAMMA)
    x, y = s.node_coordinates()
    rng = np.random.default_rng(5)
    rho = 1.0 + 0.3 * np.sin(9 * x + 5 * y) + np.where(x > 0.5, 0.4, 0.0) + 0.02 * rng.normal(size=x.shape)
    p = 1.0 + 0.3 * np.cos(7 * x) + np.where(x > 0.5, 0.5, 0.0)
    q = np.stack([rho, 0.2 * rho, -0.1 * rho, p / (GAMMA - 1.0) + 0.025 * rho], axis=-1)
    q = q.astype(np.float32).astype(np.float64)
    got, flags = s.limit_with_flags(q)
    avg = np.einsum("i,ikc->kc", s.reference.cell_weights / s.reference.cell_weights.sum(), q)
    want, troubled = o.troubled_cell_limit(q, avg)
    want = o.positivity_limit(want, avg)
    scale = np.abs(want).reshape(-1, 4).max(axis=0)
    if precision == "fp64":
        assert np.array_equal(flags, troubled)
        assert np.max(np.abs(got - want) / scale) <= 1e-12
    else:
        same = flags == troubled
        assert same.mean() > 0.9
        assert np.max(np.abs(got - want)[:, same] / scale) <= 2e-5
