"""The passes in voxel modes (stencil_modal.cuh, modal_point.cuh) against the passes that take any
element matrix (CHFEM_B200_THERMAL_OP=generic, CHFEM_B200_BLOCK_OP=element), at the edges of their
tiles: thin and ragged images, 1 to 4 materials, every operator mode, with a density field.

Bars: the operator sums the same products in another order -- 64 (voxel, node) pairs per node
and at most 24 terms each, so 1e-13 of the largest entry in FP64 and 1e-5 in FP32; solutions of
the same iteration to the same tolerance agree to 10 tol, iteration counts to one.
"""
import ctypes

import numpy as np
import pytest

from tests import helpers as H
from tests.test_gpu_parity import build_small, host_arrays, setup_model

pytestmark = pytest.mark.gpu
ENV = {0: ("CHFEM_B200_THERMAL_OP", "generic"), 1: ("CHFEM_B200_BLOCK_OP", "element")}


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def both(monkeypatch, analysis, fn):
    out = []
    for value in ("", ENV[analysis][1]):
        monkeypatch.setenv(ENV[analysis][0], value)
        out.append(fn())
    return out


SPECS = [((1, 1, 1), 1), ((1, 2, 3), 2), ((9, 33, 31), 2), ((3, 32, 8), 3), ((33, 7, 65), 2), ((4, 64, 10), 4), ((3, 70, 700), 2)]  # the last: more tiles than SMs


@pytest.mark.parametrize("shape,nmat", SPECS)
@pytest.mark.parametrize("analysis", [0, 1])
@pytest.mark.parametrize("precision", [0, 1])
def test_apply_equals_general_pass(tmp_path, monkeypatch, analysis, shape, nmat, precision):
    from chfem_b200 import _native
    nf, raw = build_small(tmp_path, "modal", analysis, ("img", shape, nmat))
    a = host_arrays(nf, raw)
    x = np.random.default_rng(3).standard_normal(a["ndof"])
    lib = _native.cudapcg()

    def run():
        setup_model(lib, a)
        assert lib.cudapcgB200SetPrecision(precision)
        y = np.zeros(a["ndof"])
        assert lib.cudapcgB200ApplyOperator(ptr(x), ptr(y)), lib.cudapcgB200LastError()
        lib.cudapcgEnd()
        return y
    y, yref = both(monkeypatch, analysis, run)
    # a single voxel's operator is zero: compare with the size of the products that cancel
    scale = max(np.abs(yref).max(), np.abs(a["lcl"]).max() * np.abs(x).max())
    assert np.abs(y - yref).max() < (1e-13 if precision == 0 else 1e-5) * scale


@pytest.mark.parametrize("density", [False, True])
@pytest.mark.parametrize("solver,norm", [(0, 0), (0, 1), (0, 2), (1, 0), (1, 2), (2, 0), (2, 2)])
@pytest.mark.parametrize("analysis,shape,nmat", [(0, (9, 33, 12), 2), (0, (4, 10, 35), 4), (1, (5, 33, 9), 2), (1, (7, 8, 34), 3),
                                                 (0, (2, 40, 650), 2)])
def test_solve_equals_general_pass(tmp_path, monkeypatch, analysis, shape, nmat, solver, norm, density):
    """Every operator mode and both pointwise forms (x in every pass or in every second one), with
    iteration counts of either parity."""
    from chfem_b200 import _native
    nf, raw = build_small(tmp_path, "modal", analysis, ("img", shape, nmat))
    a = host_arrays(nf, raw)
    lib = _native.cudapcg()
    rng = np.random.default_rng(11)
    b = rng.standard_normal(a["ndof"])
    dof = 3 if analysis == 1 else 1
    b -= np.tile(b.reshape(-1, dof).mean(axis=0), a["ndof"] // dof)
    sdf = rng.integers(0, 65536, size=a["N"]).astype(np.uint16)
    lib.cudapcgSetParametricDensityField.argtypes = [ctypes.c_void_p, ctypes.c_double, ctypes.c_double]
    tol = 1e-8

    def run():
        setup_model(lib, a)
        if density:
            assert lib.cudapcgSetParametricDensityField(ptr(sdf), 0.5, 1.5)
            assert lib.cudapcgSetImage(ptr(np.ascontiguousarray(a["keys"])))
        assert lib.cudapcgSetSolver(solver) and lib.cudapcgSetPreconditioner(1) and lib.cudapcgSetResNorm(norm)
        assert lib.cudapcgSetNumTol(tol) and lib.cudapcgSetMaxIterations(20000) and lib.cudapcgAllocateArrays()
        assert lib.cudapcgSetRHS(ptr(b))
        x = np.zeros(a["ndof"])
        # under the error norm CG may stop on the residual first, which reports "not found"
        found = lib.cudapcgSolve(ptr(x))
        assert (found or norm == 2) and not lib.cudapcgB200LastError(), lib.cudapcgB200LastError()
        its = lib.cudapcgGetNumIterations()
        lib.cudapcgEnd()
        x -= np.tile(x.reshape(-1, dof).mean(axis=0), a["ndof"] // dof)
        return x, its
    (x, its), (xref, itsref) = both(monkeypatch, analysis, run)
    assert abs(its - itsref) <= 1 and its < 20000
    # the error norm bounds the last step instead of the residual: the iterates of one count
    assert H.rel_to_max(x, xref) < (10 * tol if its == itsref else 1e-4)


def test_maxit_of_either_parity(tmp_path, monkeypatch):
    """A solve stopped by the iteration limit returns the iterate of that count, also when the last
    pass is one that leaves x to the next."""
    from chfem_b200 import _native
    nf, raw = build_small(tmp_path, "modal", 1, ("img", (6, 9, 10), 2))
    a = host_arrays(nf, raw)
    lib = _native.cudapcg()
    b = np.random.default_rng(2).standard_normal(a["ndof"])
    b -= np.tile(b.reshape(-1, 3).mean(axis=0), a["N"])
    for maxit in (1, 2, 5, 16, 17):
        def run():
            setup_model(lib, a)
            assert lib.cudapcgSetNumTol(1e-14) and lib.cudapcgSetMaxIterations(maxit) and lib.cudapcgAllocateArrays()
            assert lib.cudapcgSetRHS(ptr(b))
            x = np.zeros(a["ndof"])
            lib.cudapcgSolve(ptr(x))
            assert lib.cudapcgGetNumIterations() == maxit
            lib.cudapcgEnd()
            return x
        x, xref = both(monkeypatch, 1, run)
        assert H.rel_to_max(x, xref) < 1e-11


def test_other_matrices_keep_the_general_pass(tmp_path, monkeypatch):
    """Element matrices that are not those of an isotropic material (C ABI): both settings give the
    same operator, which is not the isotropic one."""
    from chfem_b200 import _native
    nf, raw = build_small(tmp_path, "modal", 1, ("img", (5, 9, 8), 2))
    a = host_arrays(nf, raw)
    x = np.random.default_rng(3).standard_normal(a["ndof"])
    lib = _native.cudapcg()
    ys = []
    for factor in (1.0, 1.2):
        m = dict(a, lcl=a["lcl"].copy())
        K = m["lcl"].reshape(-1, 24, 24)
        K[:, 0::3, 0::3] *= factor  # stiffer along x only
        def run():
            setup_model(lib, m)
            y = np.zeros(a["ndof"])
            assert lib.cudapcgB200ApplyOperator(ptr(x), ptr(y)), lib.cudapcgB200LastError()
            lib.cudapcgEnd()
            return y
        y, yref = both(monkeypatch, 1, run)
        assert H.rel_to_max(y, yref) < 1e-13
        ys.append(y)
    assert H.rel_to_max(ys[1], ys[0]) > 1e-3
