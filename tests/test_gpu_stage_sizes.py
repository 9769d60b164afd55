"""The FP64 stage kernel behind variant 0 at the sizes where waves of resident blocks decide its form:
one thread per node up to 7,104 elements (8,000 for a right-hand side), then four lanes per element or
tiles of 32, up to the 18,944 and 23,680 elements that one wave of each holds. Against the register-only
pair kernel, whose values are the same in the same order up to the multiply-adds the compiler contracts:
1e-13 of each variable's scale for a right-hand side (a few ulps of the largest value), 1e-9 for a limited
step, where a slope-limiter decision within rounding of its 1e-10 threshold may differ."""

from __future__ import annotations

import numpy as np
import pytest

from tests.gpu_helpers import rel_err
from tests.test_gpu_stage_forms import _solver, _state

pytestmark = pytest.mark.gpu

# 7,104 / 7,106, 8,000 / 8,008, 18,944 / 18,952, 23,680 / 23,688 elements, and 20,000
MESHES = [(74, 48), (187, 19), (100, 40), (91, 44), (148, 64), (103, 92), (148, 80), (126, 94), (100, 100)]


@pytest.mark.parametrize("nx,ny", MESHES)
@pytest.mark.parametrize("flux", ["rusanov", "roe", "hllc"])
def test_default_fp64_form_on_both_sides_of_each_size(nx, ny, flux):
    a, b = (_solver(nx, ny, flux, "minmod", "fp64", v) for v in (0, 2))
    q = _state(a, False)
    (ra, fa), (rb, fb) = a.rhs(q), b.rhs(q)
    dt = a.time_step(q)
    (qa, pa), (qb, pb) = a.step(q, dt), b.step(q, dt)
    assert rel_err(ra, rb) <= 1e-13 and rel_err(qa, qb) <= 1e-9
    np.testing.assert_allclose(fa, fb, rtol=1e-12, atol=1e-13)
    assert pa.admissible == pb.admissible
    assert pa.min_density == pytest.approx(pb.min_density, rel=1e-8)
    assert pa.min_pressure == pytest.approx(pb.min_pressure, rel=1e-8, abs=1e-8)
