"""Any leading dimension >= num_elements, and any element alignment, is served: the stage forms that
copy whole blocks of elements by 16 bytes run only where those copies are aligned and end inside the
buffers; elsewhere the pair kernel (explicit shapes) or the node kernel (variant 0) takes the call, and
the persistent batch launch refuses it on the host."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

GAMMA = 1.4
TABLES = ("metric", "face_geo", "face_hlen", "dt_geo", "jacobian", "cs_coef", "neighbor", "face_info")


def _fake_solver(k, ld, shift=0, precision=0):
    """A CfdSolver whose pointers are never followed: the checks run before any launch."""
    from cfd_demo_b200 import _native

    s = _native.CfdSolver()
    s.mesh.num_elements, s.mesh.ld, s.mesh.num_instances = k, ld, 1
    for i, name in enumerate(TABLES + ("metric32", "face_geo32", "cs_coef32")):
        setattr(s.mesh, name, 4096 * (i + 1))
    for i, name in enumerate(("averages", "element_aux", "acc", "report", "control", "limit_list")):
        setattr(s, name, 4096 * (i + 20))
    s.gamma, s.cfl, s.precision = GAMMA, 0.5, precision
    return s, [4096 * 30 + shift, 4096 * 31, 4096 * 32]


@pytest.mark.parametrize("k,ld,shift", [(598, 599, 0), (598, 598, 0), (598, 600, 0), (598, 639, 0), (598, 640, 8)])
def test_persistent_batch_refuses_buffers_its_tiles_do_not_fit(k, ld, shift):
    """Before any launch (attempts = 0 launches nothing): odd ld, an ld that ends inside the last tile
    of 64, and a state off the 16-byte grid."""
    from cfd_demo_b200 import _native

    lib = _native.load()
    for precision in (_native.CFD_FP64, _native.CFD_FP32_MIXED):
        s, x = _fake_solver(k, ld, shift, precision)
        assert lib.cfd_batch_advance(C.byref(s), *x, 0, None) == -1
        assert b"whole tiles of 64 elements" in lib.cfd_last_error()


def _setup(nx, ny, limiter, precision, ld=None, shift=0, variant=0):
    """(solver struct, states) of one mesh with its tables and buffers laid out with leading dimension
    ld, every row table and state `shift` entries off its allocation's start."""
    import torch

    from cfd_demo_b200 import EulerSolver, FixedState, SlipWall, SolverConfig, _native
    from cfd_demo_b200.mesh import jittered_rectangle_mesh

    mesh = jittered_rectangle_mesh(nx, ny, 0.15, 3)
    far = FixedState.from_primitive(1.0, 0.1, -0.2, 1.0, GAMMA)
    solver = EulerSolver(mesh, {"left": far, "right": far, "bottom": SlipWall(), "top": SlipWall()},
                         SolverConfig(flux="hllc", limiter=limiter, gamma=GAMMA, precision=precision), variant=variant)
    ops, ws, k = solver.operators, solver._ws, mesh.num_elements
    ld = ops.ld if ld is None else ld
    keep = []

    def lay(src, rows):
        flat = torch.zeros(rows * ld + 16, dtype=src.dtype, device=src.device)
        view = flat[shift:shift + rows * ld].view(rows, ld)
        view[:, :k] = src.reshape(rows, -1)[:, :k]
        keep.append(flat)
        return view

    s = _native.CfdSolver.from_buffer_copy(bytes(solver.native))
    s.mesh.ld = ld
    names = TABLES + (("metric32", "face_geo32", "cs_coef32") if precision != "fp64" else ())
    for name in names:
        src = getattr(ops, name)
        setattr(s.mesh, name, lay(src, 1 if src.dim() == 1 else src.shape[0]).data_ptr())
    s.averages, s.element_aux = lay(ws.averages, 4).data_ptr(), lay(ws.aux, 3).data_ptr()
    x, y = solver.node_coordinates()
    rho, p = 1.0 + 0.4 * np.sin(7 * x + 3 * y), 1.0 + 0.4 * np.cos(5 * x - 4 * y)
    u, v = 0.6 * np.sin(9 * y), -0.5 * np.cos(8 * x)
    q = np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], axis=-1)
    q0 = lay(solver.upload(q), 60)
    states = [q0] + [lay(torch.zeros_like(ws.x0), 60) for _ in range(2)]
    return solver, s, states, keep


def _attempt(solver, s, states, dt):
    import torch

    from cfd_demo_b200 import _native

    k = s.mesh.num_elements
    solver._write_control(dt=dt, final_time=np.inf, status=_native.RUN_ACTIVE, parity=0)
    _native.check(solver._lib.cfd_rk3_attempt(C.byref(s), *(x.data_ptr() for x in states),
                                              torch.cuda.current_stream().cuda_stream))
    return states[1][:, :k].double().cpu().numpy()


# 598 elements: odd ld; ld that ends inside the last block of 32; one that holds blocks of 32 but not
# of 64; whole blocks, but rows off the 16-byte grid
ROWS = [(599, 0), (600, 0), (608, 0), (640, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("ld,shift", ROWS)
@pytest.mark.parametrize("variant", [0, 1, 2, 3, 9, 10, 14])
@pytest.mark.parametrize("limiter", ["minmod", "unlimited"])
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_attempt_with_any_leading_dimension(ld, shift, variant, limiter, precision):
    """The step of buffers that no tile fits is, bit for bit, that of the form that takes it over (the
    node kernel for variant 0, else the pair kernel) on aligned buffers; where blocks of 32 fit, a shape
    of 32 elements runs itself."""
    fits = (ld, shift) == (608, 0) and variant == 1
    same = variant if variant in (0, 2) or fits else 2
    a = _setup(23, 13, limiter, precision, ld, shift, variant)
    b = _setup(23, 13, limiter, precision, None, 0, same)
    dt = 1e-3
    assert np.array_equal(_attempt(*a[:3], dt), _attempt(*b[:3], dt))


@pytest.mark.gpu
@pytest.mark.parametrize("ld", [10207, 10208, 10240])
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_large_default_attempt_with_any_leading_dimension(ld, precision):
    """10,206 elements, past the node kernel's range: it serves them all the same where blocks of 32 do
    not fit (odd ld; 10,208 holds them exactly). Unlimited, so the forms differ by a few ulps of each
    variable's largest value: 1e-13 in FP64, 2e-6 (16 ulps) in FP32-mixed."""
    a = _setup(81, 63, "unlimited", precision, ld)
    b = _setup(81, 63, "unlimited", precision)
    qa, qb = _attempt(*a[:3], 1e-4), _attempt(*b[:3], 1e-4)
    scale = np.abs(qb).reshape(4, 15, -1).max(axis=(1, 2))
    err = (np.abs(qa - qb).reshape(4, 15, -1).max(axis=(1, 2)) / scale).max()
    assert err <= (1e-13 if precision == "fp64" else 2e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("ld,shift", ROWS)
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_taped_step_with_any_leading_dimension(ld, shift, precision):
    """cfd_rk3_step_fixed: the result with a tape is that without (the default shape in both), the tape
    holds the stage states, and a step whose buffers fit agrees to round-off (the unlimited step, a few
    ulps of each variable's largest value)."""
    import torch

    from cfd_demo_b200 import _native

    out, tapes = [], []
    prec = _native.CFD_FP64 if precision == "fp64" else _native.CFD_FP32_MIXED
    for setup in (_setup(23, 13, "unlimited", precision, ld, shift), _setup(23, 13, "unlimited", precision)):
        solver, s, (x0, x1, stage), _ = setup
        k, width = s.mesh.num_elements, s.mesh.ld
        stream = torch.cuda.current_stream().cuda_stream
        dt = torch.tensor([1e-3], dtype=torch.float64, device="cuda")
        tape = torch.zeros(solver._lib.cfd_tape_bytes(width, prec), dtype=torch.uint8, device="cuda")
        args = (C.byref(s), x0.data_ptr(), x1.data_ptr(), stage.data_ptr(), dt.data_ptr())
        _native.check(solver._lib.cfd_rk3_step_fixed(*args, tape.data_ptr(), stream))
        taped = x1[:, :k].clone()
        _native.check(solver._lib.cfd_rk3_step_fixed(*args, None, stream))
        assert torch.equal(taped, x1[:, :k])
        size = 60 * width * x0.element_size()
        slots = [tape[i * size:(i + 1) * size].view(x0.dtype).view(60, width)[:, :k].double() for i in range(5)]
        for i in (1, 3):  # an admissible unlimited step: the limited stage states are the stage states
            assert torch.equal(slots[i], slots[i - 1])
        assert torch.equal(slots[4], taped.double())
        out.append(taped.double()), tapes.append(torch.stack(slots))
    scale = out[1].view(4, -1).abs().amax(1)
    tol = 1e-13 if precision == "fp64" else 2e-6
    for a, b in ((out[0], out[1]), *zip(*tapes)):
        assert float(((a - b).view(4, -1).abs().amax(1) / scale).max()) <= tol
