"""Right-hand sides of states with non-finite fluxes at inner nodes, in every FP64 form of the stage
kernel: which entries are finite is as in the reference, whose [Dr|Ds] products are dense (a NaN or an
infinity times a round-off zero of the matrix is not finite)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAMMA = 1.4
# node (6, 7 and 10 lie inside the element and take no part in a face flux), variable, value
POISON = [(6, 0, np.nan), (10, 2, np.inf), (7, 3, np.inf), (6, 0, 0.0), (10, 1, np.nan), (7, 3, -np.inf)]


# 70 and 598 elements: one thread per node; 9,150, 19,200 and 40,328: the forms of larger meshes
@pytest.mark.parametrize("nx,ny", [(7, 5), (23, 13), (75, 61), (96, 100), (142, 142)])
@pytest.mark.parametrize("flux", ["rusanov", "roe", "hllc"])
def test_finite_entries_of_the_right_hand_side_are_the_oracles(nx, ny, flux):
    import oracle
    from cfd_demo_b200 import EulerSolver, SlipWall, SolverConfig
    from cfd_demo_b200.mesh import jittered_rectangle_mesh

    mesh = jittered_rectangle_mesh(nx, ny, 0.15, 3)
    wall = {t: SlipWall() for t in ("left", "right", "bottom", "top")}
    s = EulerSolver(mesh, wall, SolverConfig(flux=flux, limiter="minmod", gamma=GAMMA))
    om = oracle.mesh.TriangleMesh(np.array(mesh.vertices), np.array(mesh.elements),
                                  {t: np.array(e) for t, e in mesh.boundary_edges.items()})
    o = oracle.OracleSolver(om, {t: oracle.physics.SlipWall() for t in wall}, flux=flux, limiter="minmod", gamma=GAMMA)
    x, y = s.node_coordinates()
    rho, p = 1.0 + 0.4 * np.sin(7 * x + 3 * y), 1.0 + 0.4 * np.cos(5 * x - 4 * y)
    u, v = 0.6 * np.sin(9 * y), -0.5 * np.cos(8 * x)
    q = np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], axis=-1)
    k = mesh.num_elements
    for i, (node, var, value) in enumerate(POISON):
        q[node, (i * k) // len(POISON) + (i > 0), var] = value
    with np.errstate(all="ignore"):
        want, _ = o.rhs(q)
    got, _ = s.rhs(q)
    assert not np.isfinite(want).all()
    assert np.array_equal(np.isfinite(got), np.isfinite(want))


# 70, 9,150, 19,200, 72,900 and 100,352 elements: every form of the stage kernel and of the limiter
@pytest.mark.parametrize("nx,ny,limiter", [(7, 5, "minmod"), (7, 5, "unlimited"), (75, 61, "minmod"), (75, 61, "unlimited"),
                                           (96, 100, "unlimited"), (270, 135, "minmod"), (224, 224, "unlimited")])
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_steps_of_bad_states_are_those_of_the_pair_kernel(nx, ny, limiter, precision):
    """A step from a state with a NaN, an infinity or an inadmissible node: the same verdict, the same
    NaN minima and the same finite entries as with the register-only pair kernel."""
    from tests.test_gpu_stage_forms import _solver, _state

    a, b = (_solver(nx, ny, "hllc", limiter, precision, v) for v in (0, 2))
    q = _state(a, False)
    k = q.shape[1]
    for node, var, value in POISON + [(0, 3, np.nan), (2, 1, np.nan), (12, 0, -0.5), (6, 3, 1e-3)]:
        bad = q.copy()
        bad[node, [0, k // 3 + 1, k - 1], var] = value
        (qa, ra), (qb, rb) = a.step(bad, 1e-4), b.step(bad, 1e-4)
        assert ra.admissible == rb.admissible
        assert np.isnan(ra.min_density) == np.isnan(rb.min_density)
        assert np.isnan(ra.min_pressure) == np.isnan(rb.min_pressure)
        assert np.array_equal(np.isfinite(qa), np.isfinite(qb))
