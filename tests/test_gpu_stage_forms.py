"""The stage kernel's forms behind variant 0 (one thread per node on small meshes; above, four lanes
per element in FP64 and tiles of 32 in FP32-mixed) against a tiled shape of 64, at the smallest
meshes, ragged ones and the sizes where the form changes. Both evaluate the same values in the same order
up to the multiply-adds the compiler contracts. One stage then differs by a few ulps of the largest
value: 1e-13 of each variable's scale in FP64, 2e-6 (16 ulps) in FP32-mixed for a right-hand side and
an unlimited step. With slope limiting, a decision within rounding of its threshold may differ, which
is 1e-10 (FP64) or 1e-5 (FP32-mixed) of the average: 1e-9 and 1e-4 there."""

from __future__ import annotations

import numpy as np
import pytest

from tests.gpu_helpers import rel_err

pytestmark = pytest.mark.gpu

GAMMA = 1.4
# elements: 2, 70, 598 (ragged), the last size of the node form, the first above (8,008), and 10,206
# (ragged against the blocks of 32 and the warps of 8)
MESHES = [(1, 1), (7, 5), (23, 13), (100, 40), (91, 44), (81, 63)]


def _solver(nx, ny, flux, limiter, precision, variant):
    from cfd_demo_b200 import EulerSolver, FixedState, SlipWall, SolverConfig
    from cfd_demo_b200.mesh import jittered_rectangle_mesh

    mesh = jittered_rectangle_mesh(nx, ny, 0.15, 3)
    far = FixedState.from_primitive(1.0, 0.1, -0.2, 1.0, GAMMA)
    return EulerSolver(mesh, {"left": far, "right": far, "bottom": SlipWall(), "top": SlipWall()},
                       SolverConfig(flux=flux, limiter=limiter, gamma=GAMMA, precision=precision), variant=variant)


def _state(s, thin):
    x, y = s.node_coordinates()
    rho = 1.0 + 0.4 * np.sin(7 * x + 3 * y)
    p = 1.0 + 0.4 * np.cos(5 * x - 4 * y)
    if thin:  # nodes below the pressure floor after a stage: the positivity repair of the unlimited form
        p = p * (0.02 + 0.98 * (np.sin(40 * x) * np.sin(31 * y) > 0.3))
    u, v = 0.6 * np.sin(9 * y), -0.5 * np.cos(8 * x)
    return np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], axis=-1)


@pytest.mark.parametrize("nx,ny", MESHES)
@pytest.mark.parametrize("flux", ["rusanov", "roe", "hllc"])
@pytest.mark.parametrize("limiter,thin", [("minmod", False), ("unlimited", False), ("unlimited", True)])
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_default_form_matches_the_tiled_form(nx, ny, flux, limiter, thin, precision):
    a, b = (_solver(nx, ny, flux, limiter, precision, v) for v in (0, 9))
    q = _state(a, thin)
    (ra, fa), (rb, fb) = a.rhs(q), b.rhs(q)
    dt = a.time_step(q)
    (qa, pa), (qb, pb) = a.step(q, dt), b.step(q, dt)
    assert pa.admissible == pb.admissible
    np.testing.assert_allclose(fa, fb, rtol=1e-12 if precision == "fp64" else 1e-5, atol=1e-6 if precision != "fp64" else 1e-13)
    same = 1e-13 if precision == "fp64" else 2e-6
    step = same if limiter == "unlimited" else (1e-9 if precision == "fp64" else 1e-4)
    assert rel_err(ra, rb) <= same and rel_err(qa, qb) <= step
    assert pa.min_density == pytest.approx(pb.min_density, rel=10 * step)
    assert pa.min_pressure == pytest.approx(pb.min_pressure, rel=10 * step, abs=10 * step)


@pytest.mark.parametrize("nx,ny,same", [(317, 157, False), (500, 100, True)])  # 99,538 and 100,000 elements
def test_default_form_of_large_unlimited_fp32_steps(nx, ny, same):
    """From 100,000 elements on an unlimited FP32-mixed step runs shape 9 itself (the same bits); below
    it agrees to 2e-6 of each variable's scale."""
    a, b = (_solver(nx, ny, "roe", "unlimited", "fp32_mixed", v) for v in (0, 9))
    q = _state(a, False)
    dt = a.time_step(q)
    (qa, _), (qb, _) = a.step(q, dt), b.step(q, dt)
    assert np.array_equal(qa, qb) if same else rel_err(qa, qb) <= 2e-6
