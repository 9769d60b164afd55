"""cfd_time_step and the initial-state check on finite, non-finite and inadmissible states, at the sizes
where the pass by node takes one element group a block and where its blocks sweep (from 9,472 elements),
where FP32-mixed turns to a thread per element (300,000, and 20,000 with several instances), and with
instances aligned to blocks and not."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAMMA = 1.4
# 2, 70, 9,472 and 9,498, 200,000, 300,000 and 300,600 elements
MESHES = [(1, 1), (7, 5), (74, 64), (1583, 3), (400, 250), (500, 300), (501, 300)]
# node, variable and value put into one element
POISON = {"nan density": (6, 0, np.nan), "nan momentum": (0, 1, np.nan), "nan energy": (14, 3, np.nan),
          "infinite energy": (3, 3, np.inf), "minus infinite energy": (3, 3, -np.inf), "infinite density": (9, 0, np.inf),
          "infinite momentum": (9, 2, np.inf), "negative density": (1, 0, -0.5), "negative pressure": (2, 3, -1.0)}


def _solver(nx, ny, precision):
    from cfd_demo_b200 import EulerSolver, SlipWall, SolverConfig
    from cfd_demo_b200.mesh import jittered_rectangle_mesh

    mesh = jittered_rectangle_mesh(nx, ny, 0.15, 5)
    return EulerSolver(mesh, {t: SlipWall() for t in ("left", "right", "bottom", "top")},
                       SolverConfig(flux="rusanov", limiter="minmod", gamma=GAMMA, precision=precision))


def _state(s):
    x, y = s.node_coordinates()
    rho, p = 1.0 + 0.4 * np.sin(7 * x + 3 * y), 1.0 + 0.4 * np.cos(5 * x - 4 * y)
    u, v = 0.6 * np.sin(9 * y), -0.5 * np.cos(8 * x)
    q = np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], axis=-1)
    return q.astype(np.float32).astype(np.float64)


def _expected(s, q):
    """Per element dt_geo / max(|u| + c), NaN where a node's speed is NaN (time_integration.py:37-41)."""
    with np.errstate(invalid="ignore", divide="ignore"):
        u, v = q[..., 1] / q[..., 0], q[..., 2] / q[..., 0]
        p = (GAMMA - 1.0) * (q[..., 3] - 0.5 * (q[..., 1] * u + q[..., 2] * v))
        speed = np.sqrt(u * u + v * v) + np.sqrt(GAMMA * p / q[..., 0])
        return s.operators.dt_geo[: q.shape[1]].cpu().numpy() / np.max(speed, axis=0)


def _assert_dt(got, want, precision):
    """FP64: the same operations in the same order. FP32-mixed: a dozen single roundings of the speed,
    and up to 1e-4 of it where the pressure cancels."""
    if np.isnan(want):
        assert np.isnan(got)
    else:
        assert got == pytest.approx(want, rel=1e-15 if precision == "fp64" else 1e-5)


@pytest.mark.parametrize("nx,ny", MESHES)
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_time_step_of_any_state(nx, ny, precision):
    from cfd_demo_b200 import SolverError

    s = _solver(nx, ny, precision)
    q = _state(s)
    cfl = s.config.cfl
    _assert_dt(s.time_step(q), cfl * np.min(_expected(s, q)), precision)
    s.begin_run(q, 1.0)
    k = q.shape[1]
    for node, var, value in POISON.values():
        bad = q.copy()
        bad[node, (2 * k) // 3, var] = value
        _assert_dt(s.time_step(bad), cfl * np.min(_expected(s, bad)), precision)
        with pytest.raises(SolverError):
            s.begin_run(bad, 1.0)


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("nx,ny,starts", [(23, 13, (192, 448)), (150, 100, (64, 19968)), (150, 100, (9984, 29952))])
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_time_step_of_each_instance(precision, aligned, nx, ny, starts):
    """Three instances in one launch, their elements starting at multiples of 64 (a block's elements
    belong to one) or anywhere: each instance's step is its own, and a NaN poisons only its own. With
    30,000 elements a block of the FP64 pass takes several groups and meets the next instance among them."""
    import torch

    from cfd_demo_b200 import _native

    s = _solver(nx, ny, precision)
    q = _state(s)
    first = np.array([0, *starts]) + (np.array([0, 9, 11]) if not aligned else 0)
    owner = np.searchsorted(first, np.arange(q.shape[1]), side="right") - 1
    table = torch.full((s.operators.ld,), -1, dtype=torch.int32, device="cuda")
    table[: q.shape[1]] = torch.from_numpy(owner.astype(np.int32)).cuda()
    native = _native.CfdSolver.from_buffer_copy(bytes(s.native))
    native.mesh.instance, native.mesh.num_instances = table.data_ptr(), 3
    native.mesh.flags, native.variant = (1, 0) if aligned else (0, 2)
    acc = torch.zeros(9 * _native.SIZES["CfdStageAcc"], dtype=torch.uint8, device="cuda")
    native.acc = acc.data_ptr()
    for poisoned in (None, 0, 1, 2):
        bad = q.copy()
        if poisoned is not None:
            bad[4, first[poisoned] + 30, 3] = np.nan
        dt = torch.zeros(3, dtype=torch.float64, device="cuda")
        check = torch.zeros(9, dtype=torch.float64, device="cuda")
        x, stream = s.upload(bad), torch.cuda.current_stream().cuda_stream
        _native.check(s._lib.cfd_time_step(C.byref(native), x.data_ptr(), dt.data_ptr(), stream))
        _native.check(s._lib.cfd_check_state(C.byref(native), x.data_ptr(), check.data_ptr(), stream))
        e, finite = _expected(s, bad), check.cpu().numpy().reshape(3, 3)[:, 2]
        for i in range(3):
            _assert_dt(float(dt[i]), s.config.cfl * np.min(e[owner == i]), precision)
            assert finite[i] == (0.0 if i == poisoned else 1.0)
