"""The pointwise pass on pixel models and the three (P)MINRES passes of Stokes models, at odd sizes.

Oracles: an extruded image of one layer solved by the 3D passes for any matrix has the tensor of its
2D image (the solution does not depend on z); a Stokes solution's residual through the operator
gathered by DOF number (cudapcgB200ApplyOperator), which the (P)MINRES passes do not use, for voxels
and pixels; a Stokes block (voxels only) against its directions one by one.
"""
import ctypes
import zlib

import numpy as np
import pytest

from tests import helpers as H
from tests.test_gpu_parity import host_arrays, setup_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multirhs", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,nmat", [((1, 2), 2), ((5, 7), 2), ((33, 31), 4), ((8, 34), 3), ((64, 128), 2)])
@pytest.mark.parametrize("analysis", ["conductivity", "elasticity"])
def test_pixels_equal_one_layer_of_voxels(monkeypatch, analysis, shape, nmat, precision, multirhs):
    from chfem_b200 import compute_property
    monkeypatch.setenv("CHFEM_B200_THERMAL_OP", "generic")
    monkeypatch.setenv("CHFEM_B200_BLOCK_OP", "element")
    img = H.small_image(shape, nmat, seed=zlib.crc32(repr(shape).encode()) % 1000)
    vals = [(1.0, 0.3), (10.0, 0.2), (4.0, 0.25), (0.5, 0.35)]
    props = {int(c): (vals[i] if analysis == "elasticity" else vals[i][0]) for i, c in enumerate(np.unique(img))}
    kw = dict(mat_props=props, solver_tolerance=1e-9 if precision == "fp64" else 1e-7, solver_maxiter=20000, precision=precision)
    C2 = np.array(compute_property(analysis, img, multirhs=multirhs, **kw))
    C3 = np.array(compute_property(analysis, img[None], **kw))
    ax = [0, 1, 5] if analysis == "elasticity" else [0, 1]  # plane strain: xx, yy, xy
    # both stop at tol: the tensor's error is of the order tol; FP32 fields add theirs
    assert H.rel_to_max(C2, C3[np.ix_(ax, ax)]) < (1e-6 if precision == "fp64" else 1e-4)


def stokes_case(tmp_path, shape, porosity):
    rng = np.random.default_rng(zlib.crc32(repr((shape, porosity)).encode()) % 10000)
    img = np.where(rng.random(shape) < porosity, 0, 255).astype(np.uint8)
    if porosity < 0:  # a duct: more than four nodes per fluid node, the records by DOF number
        img[:] = 255
        img[..., 4:10, 5:11] = 0
    elif len(shape) == 3 and min(shape) > 8:  # connected pores: a smooth field
        from chfem_b200.synthetic import pore_grf
        img = pore_grf(shape, corr=2.0, porosity=porosity, seed=5)
    return img, H.write_small_case(str(tmp_path), "fl", img, 2, tol=1e-8, maxit=20000)


@pytest.mark.parametrize("precondition", [0, 1])
@pytest.mark.parametrize("shape,porosity", [((3, 3, 3), 1.0), ((5, 6, 7), 0.9), ((9, 33, 10), 0.6), ((17, 12, 35), 0.45),
                                            ((24, 20, 28), -1), ((3, 4), 1.0), ((25, 21), 0.75), ((40, 33), 0.7), ((31, 28), -1)])
def test_stokes_solution_meets_its_tolerance(tmp_path, shape, porosity, precondition):
    from chfem_b200 import _native
    img, (nf, raw) = stokes_case(tmp_path, shape, porosity)
    a = dict(host_arrays(nf, raw), dim2=len(shape) == 2)
    lib = _native.cudapcg()
    p = lambda v: v.ctypes.data_as(ctypes.c_void_p)
    lib.cudapcgGetResidual.restype = ctypes.c_double
    lib.cudapcgSetNumTol.argtypes = [ctypes.c_double]
    setup_model(lib, a)
    # a consistent right-hand side: the image of a random vector
    y = np.random.default_rng(1).standard_normal(a["ndof"])
    b, r, z0, z = (np.zeros(a["ndof"]) for _ in range(4))
    assert lib.cudapcgB200ApplyOperator(p(y), p(b)), lib.cudapcgB200LastError()
    tol = 1e-7
    assert lib.cudapcgSetSolver(1) and lib.cudapcgSetPreconditioner(precondition) and lib.cudapcgSetNumTol(tol)
    assert lib.cudapcgSetMaxIterations(20000) and lib.cudapcgAllocateArrays() and lib.cudapcgSetRHS(p(b))
    x = np.zeros(a["ndof"])
    assert lib.cudapcgSolve(p(x)), lib.cudapcgB200LastError()
    lib.cudapcgEnd()
    setup_model(lib, a)
    assert lib.cudapcgB200ApplyOperator(p(x), p(r))
    r -= b
    if precondition:
        assert lib.cudapcgB200ApplyPreconditioner(p(b), p(z0)) and lib.cudapcgB200ApplyPreconditioner(p(r), p(z))
        rel = np.sqrt(abs(r @ z) / abs(b @ z0))
    else:
        rel = np.linalg.norm(r) / np.linalg.norm(b)
    lib.cudapcgEnd()
    # the recurrence's residual stops the solve at tol; the true one drifts from it by FP64 round-off,
    # far below tol (at most 0.998 tol over these cases with three right-hand sides each)
    assert rel < 1.01 * tol, rel


@pytest.mark.parametrize("shape,porosity", [((6, 7, 9), 0.9), ((12, 33, 10), 0.6), ((24, 20, 28), -1)])
def test_stokes_block_equals_single_cases(tmp_path, shape, porosity):
    from chfem_b200 import compute_property
    img, _ = stokes_case(tmp_path, shape, porosity)
    kw = dict(solver_tolerance=1e-8, solver_maxiter=20000, solver="minres")
    C1 = np.array(compute_property("permeability", img, **kw))
    C3 = np.array(compute_property("permeability", img, multirhs=True, **kw))
    assert H.rel_to_max(C3, C1) < 1e-5
