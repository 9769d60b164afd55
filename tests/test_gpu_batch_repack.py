"""Repacking a batch into smaller ones as its instances finish, across the sizes where a kernel that
goes by the number of elements changes its form: the stage kernel at 8,000 elements, the limiter at
5,900 and 70,000."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (instances, nx range, last final time): some 12,000 and 80,000 elements at the start
@pytest.mark.parametrize("count,nx_range,last", [(14, (60, 80), 0.03), (10, (190, 210), 0.006)])
@pytest.mark.parametrize("flux,limiter", [("hllc", "superbee"), ("rusanov", "minmod"), ("roe", "unlimited")])
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_repacking_across_the_size_rules_changes_no_result(precision, flux, limiter, count, nx_range, last):
    """With the default stage kernel and separate launches: steps, times, minima and states bit for bit
    those of the batch that keeps sweeping every instance (no tolerance: the same kernels)."""
    from cfd_demo_b200 import SolverConfig, _native
    from cfd_demo_b200.batch import BatchCase, BatchedEulerSolver, riemann_batch
    from cfd_demo_b200.mesh import node_coordinates
    from cfd_demo_b200.reference_element import build_reference_triangle

    cases = riemann_batch(count=count, seed=9, nx_range=nx_range)
    if limiter == "unlimited":  # a smooth flow, which marches without a slope limiter
        ref = build_reference_triangle()
        for i, c in enumerate(cases):
            x, y = node_coordinates(c.mesh, ref.r, ref.s)
            rho, p = 1.0 + 0.1 * np.sin(6 * x + 9 * y), 1.0 + 0.1 * np.cos(7 * x)
            q = np.stack([rho, 0.2 * rho, 0.0 * rho, p / 0.4 + 0.02 * rho], axis=-1)
            cases[i] = BatchCase(c.mesh, c.boundary_conditions, q)
    cfg = SolverConfig(flux=flux, limiter=limiter, gamma=1.4, precision=precision)
    times = np.linspace(0.0015, last, count)[::-1].copy()
    packed = BatchedEulerSolver(cases, cfg, persistent=False, compact=True)
    full = BatchedEulerSolver(cases, cfg, persistent=False, compact=False)
    q = [c.initial_state for c in cases]
    a, b = (s._march(q, times, 16, 400, True) for s in (packed, full))
    sizes = {w[0].native.mesh.num_elements for w in a}
    assert packed.native.mesh.num_elements > _native.NODE_MAX_ELEMENTS
    assert min(sizes) <= (_native.NODE_MAX_ELEMENTS if count == 14 else 16000) and len(sizes) > 1
    for (sa, ia, ca), (sb, ib, cb) in zip(a, b):
        assert (ca.steps, ca.rejected, ca.max_troubled, ca.status) == (cb.steps, cb.rejected, cb.max_troubled, cb.status)
        assert (ca.time, ca.dt, ca.min_density, ca.min_pressure) == (cb.time, cb.dt, cb.min_density, cb.min_pressure)
        xa, xb = (s._ws.x1 if c.parity else s._ws.x0 for s, c in ((sa, ca), (sb, cb)))
        assert np.array_equal(sa.download(xa, ia), sb.download(xb, ib))
