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
