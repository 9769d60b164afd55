"""The limiter on both sides of every size at which its form changes: a half warp per element up to
8,288 elements, blocks that scan 32 up to 70,000, above them blocks that scan 128 (FP64, or without the
list scratch) and a launch of its own for the listed elements (FP32-mixed with it)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAMMA = 1.4
# 8,288 / 8,296, 70,000 / 70,002 and 90,000 elements
SIZES = [(74, 56), (68, 61), (350, 100), (3889, 9), (300, 150)]


def _solver(nx, ny, limiter, precision):
    from cfd_demo_b200 import EulerSolver, SlipWall, SolverConfig, rectangle_mesh

    mesh = rectangle_mesh(nx, ny)
    return EulerSolver(mesh, {t: SlipWall() for t in ("left", "right", "bottom", "top")},
                       SolverConfig(flux="rusanov", limiter=limiter, gamma=GAMMA, precision=precision))


def _state(s, rough):
    """Waves with noise in the part of the domain x < rough: troubled elements side by side there."""
    x, y = s.node_coordinates()
    rng = np.random.default_rng(5)
    noise = np.where(x < rough, 0.1, 0.0) * rng.normal(size=x.shape)
    rho = 1.0 + 0.3 * np.sin(9 * x + 5 * y) + noise
    p = 1.0 + 0.3 * np.cos(7 * x) + noise * noise
    q = np.stack([rho, 0.2 * rho, -0.1 * rho, p / (GAMMA - 1.0) + 0.025 * rho], axis=-1)
    return q.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("rough", [0.05, 1.0])  # few and nearly all elements rewritten
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_limit_matches_the_oracle_on_both_sides_of_each_size(nx, ny, rough, precision):
    """FP64: the same troubled flags, 1e-12 of each variable's scale. FP32-mixed: 2e-5 (a hundred single
    roundings) on the elements whose troubled decision the wider detection threshold leaves alike."""
    import oracle

    s = _solver(nx, ny, "mc", precision)
    m = s.mesh
    om = oracle.mesh.TriangleMesh(np.array(m.vertices), np.array(m.elements),
                                  {t: np.array(e) for t, e in m.boundary_edges.items()})
    o = oracle.OracleSolver(om, {t: oracle.physics.SlipWall() for t in m.boundary_edges}, flux="rusanov", limiter="mc",
                            gamma=GAMMA)
    q = _state(s, rough)
    got, flags = s.limit_with_flags(q)
    again, count = s.limit_with_count(q)
    assert np.array_equal(got, again) and count == flags.sum()
    avg = np.einsum("i,ikc->kc", s.reference.cell_weights / s.reference.cell_weights.sum(), q)
    want, troubled = o.troubled_cell_limit(q, avg)
    want = o.positivity_limit(want, avg)
    assert troubled.mean() > 0.9 if rough == 1.0 else 0.0 < troubled.mean() < 0.5
    scale = np.abs(want).reshape(-1, 4).max(axis=0)
    if precision == "fp64":
        assert np.array_equal(flags, troubled)
        assert np.max(np.abs(got - want) / scale) <= 1e-12
    else:
        same = flags == troubled
        assert same.mean() > 0.9
        assert np.max(np.abs(got - want)[:, same] / scale) <= 2e-5


@pytest.mark.parametrize("nx,ny", [(3889, 9), (300, 150)])
@pytest.mark.parametrize("limiter", ["minmod", "unlimited", "van_leer"])
@pytest.mark.parametrize("rough", [0.05, 1.0])
def test_the_launch_for_listed_elements_is_bitwise_the_single_launch(nx, ny, limiter, rough):
    """FP32-mixed above 70,000 elements with and without the list scratch: limited states, flags, counts
    and the reports of repeated steps bit for bit (no tolerance: the same operations; the boundary flux
    sums atomics in any order)."""
    s = _solver(nx, ny, limiter, "fp32_mixed")
    q = _state(s, rough)
    scratch = s.native.limit_list
    out = []
    for use in (scratch, None):
        s.native.limit_list = use
        limited, flags = s.limit_with_flags(q)
        dt, x, reports = s.time_step(q), q, []
        for _ in range(3):
            x, r = s.step(x, 0.2 * dt)
            reports.append((r.admissible, r.min_density, r.min_pressure, r.troubled_cells))
        out.append((limited, flags, x, reports))
    s.native.limit_list = scratch
    for a, b in zip(out[0][:3], out[1][:3]):
        assert np.array_equal(a, b)
    assert out[0][3] == out[1][3]
