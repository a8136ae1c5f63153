"""The passes that take any element matrices: assembled by neighbour for at most two materials
(stencil_asm.cuh, asm_apply.cu), element by element otherwise (CHFEM_B200_BLOCK_OP=element), in
every operator mode and as blocks.  Models of isotropic materials run in voxel modes, so these are
reached with other matrices: an elastic material that is stiffer along one axis (C ABI), and
thermal models under CHFEM_B200_THERMAL_OP=generic.

Bars: the operators sum the same products in another order, 1e-13 of the largest product in FP64
and 1e-5 in FP32; solutions to the same tolerance agree to 10 tol, iteration counts to one (mixed
precision: both meet the tolerance on the true residual, and agree to 10 times that).
"""
import ctypes
import zlib

import numpy as np
import pytest

from tests import helpers as H
from tests.test_gpu_parity import build_small, host_arrays, setup_model

pytestmark = pytest.mark.gpu


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def arr(vs):
    return (ctypes.c_void_p * len(vs))(*[v.ctypes.data for v in vs])


def laplace_element():
    """Stiffness matrix of a unit voxel's trilinear Laplacian: symmetric, constants in its null space."""
    at = np.array([(0, 0, 1), (0, 1, 1), (0, 1, 0), (0, 0, 0), (1, 0, 1), (1, 1, 1), (1, 1, 0), (1, 0, 0)])
    same = at[:, None, :] == at[None, :, :]
    S, M = np.where(same, 1.0, -1.0), np.where(same, 1 / 3, 1 / 6)
    return sum(S[..., i] * M[..., (i + 1) % 3] * M[..., (i + 2) % 3] for i in range(3))


def model(tmp_path, analysis, shape, nmat):
    a = host_arrays(*build_small(tmp_path, "asm", analysis, ("img", shape, nmat)))
    if analysis == 1:
        a["lcl"] = a["lcl"].copy()
        a["lcl"].reshape(-1, 24, 24)[:, 0::3, 0::3] += 0.4 * laplace_element()
    return a


def select(monkeypatch, analysis, element):
    """Passes that take any matrices; element: not the assembled ones."""
    monkeypatch.setenv("CHFEM_B200_THERMAL_OP", "generic")
    monkeypatch.setenv("CHFEM_B200_BLOCK_OP", "element" if element else "")


def loads(a, n, seed=11):
    dof = 3 if a["analysis"] == 1 else 1
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        b = rng.standard_normal(a["ndof"])
        out.append(b - np.tile(b.reshape(-1, dof).mean(axis=0), a["N"]))
    return out


def centred(a, x):
    dof = 3 if a["analysis"] == 1 else 1
    return x - np.tile(x.reshape(-1, dof).mean(axis=0), a["N"])


def solve(lib, a, b, solver, norm, precision, tol, x0=None):
    setup_model(lib, a)
    lib.cudapcgSetNumTol.argtypes = [ctypes.c_double]
    assert lib.cudapcgB200SetPrecision(precision) and lib.cudapcgSetSolver(solver) and lib.cudapcgSetPreconditioner(1)
    assert lib.cudapcgSetResNorm(norm) and lib.cudapcgSetNumTol(tol) and lib.cudapcgSetMaxIterations(20000) and lib.cudapcgAllocateArrays()
    assert lib.cudapcgSetRHS(ptr(b))
    x = np.zeros(a["ndof"])
    lib.cudapcgSolve(ptr(x))
    assert not lib.cudapcgB200LastError(), lib.cudapcgB200LastError()
    its = lib.cudapcgGetNumIterations()
    lib.cudapcgEnd()
    return centred(a, x), its


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("solver,norm", [(0, 0), (0, 1), (1, 0), (1, 1), (2, 0), (2, 1)])
@pytest.mark.parametrize("shape,nmat", [((9, 33, 12), 2), ((5, 8, 35), 1)])
def test_single_solves(tmp_path, monkeypatch, shape, nmat, solver, norm, precision):
    from chfem_b200 import _native
    lib = _native.cudapcg()
    a = model(tmp_path, 1, shape, nmat)
    b = loads(a, 1)[0]
    tol = 1e-8 if precision == 0 else 1e-5
    out = []
    for element in (False, True):
        select(monkeypatch, 1, element)
        out.append(solve(lib, a, b, solver, norm, precision, tol))
    (x, its), (xref, itsref) = out
    assert its < 20000 and itsref < 20000
    if precision == 0:
        assert abs(its - itsref) <= 1
    assert H.rel_to_max(x, xref) < 10 * tol * (1 if its == itsref else 10)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("element", [False, True])
@pytest.mark.parametrize("analysis,shape,nmat,nr", [(1, (9, 33, 12), 2, 6), (1, (9, 33, 11), 2, 6), (1, (5, 8, 34), 1, 3), (1, (1, 3, 5), 2, 6),
                                                    (1, (3, 7, 9), 2, 3), (0, (9, 33, 12), 2, 3), (0, (7, 9, 11), 1, 3), (0, (7, 9, 11), 3, 3)])
def test_block_operator_equals_single(tmp_path, monkeypatch, analysis, shape, nmat, nr, element, precision):
    from chfem_b200 import _native
    lib = _native.cudapcg()
    a = model(tmp_path, analysis, shape, nmat)
    rng = np.random.default_rng(zlib.crc32(repr((shape, nr)).encode()))
    xs = [rng.standard_normal(a["ndof"]) for _ in range(nr)]
    select(monkeypatch, analysis, True)  # the reference: one field at a time, element by element, FP64
    setup_model(lib, a)
    ref = [np.zeros(a["ndof"]) for _ in xs]
    for x, y in zip(xs, ref):
        assert lib.cudapcgB200ApplyOperator(ptr(x), ptr(y)), lib.cudapcgB200LastError()
    lib.cudapcgEnd()
    select(monkeypatch, analysis, element)
    setup_model(lib, a)
    assert lib.cudapcgB200SetPrecision(precision)
    ys = [np.zeros(a["ndof"]) for _ in xs]
    assert lib.cudapcgB200ApplyBlockOperator(nr, arr(xs), arr(ys)), lib.cudapcgB200LastError()
    lib.cudapcgEnd()
    scale = max(np.abs(ref).max(), np.abs(a["lcl"]).max() * np.abs(xs).max())
    assert np.abs(np.array(ys) - np.array(ref)).max() < (1e-13 if precision == 0 else 1e-5) * scale


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("norm", [0, 1])
@pytest.mark.parametrize("analysis,shape,nmat,nr,element", [
    (1, (6, 9, 10), 2, 6, False), (1, (5, 9, 11), 2, 6, False), (1, (6, 9, 10), 2, 6, True), (1, (5, 7, 9), 3, 6, False),
    (1, (4, 33, 10), 1, 3, False), (0, (9, 33, 12), 2, 3, False), (0, (7, 9, 11), 2, 3, True), (0, (7, 9, 11), 4, 3, False)])
def test_block_solve_equals_single(tmp_path, monkeypatch, analysis, shape, nmat, nr, element, norm, precision):
    """Vectors that start aligned (n divisible by 4) and not.  The first three of six cases begin at
    their solutions and finish at once, which leaves the passes to the last three."""
    from chfem_b200 import _native
    lib = _native.cudapcg()
    a = model(tmp_path, analysis, shape, nmat)
    bs = loads(a, nr)
    tol = 1e-8 if precision == 0 else 1e-5
    select(monkeypatch, analysis, True)
    ref = [solve(lib, a, b, 0, norm, 0, tol) for b in bs]
    head = [solve(lib, a, b, 0, 0, 0, 1e-12)[0] for b in bs[:3]] if nr == 6 else []
    select(monkeypatch, analysis, element)
    for guess in ([], head) if head else ([],):
        setup_model(lib, a)
        assert lib.cudapcgB200SetPrecision(precision) and lib.cudapcgSetSolver(0) and lib.cudapcgSetPreconditioner(1)
        assert lib.cudapcgSetResNorm(norm) and lib.cudapcgSetNumTol(tol) and lib.cudapcgSetMaxIterations(20000)
        xs = [np.zeros(a["ndof"]) for _ in bs]
        its, res = (ctypes.c_uint * nr)(), (ctypes.c_double * nr)()
        x0 = (ctypes.c_void_p * nr)(*[g.ctypes.data for g in guess])
        ok = lib.cudapcgB200SolveBlock(nr, arr(bs), x0 if guess else None, 0, arr(xs), its, res)
        assert ok, lib.cudapcgB200LastError()
        lib.cudapcgEnd()
        for k in range(nr):
            x, (xref, itsref) = centred(a, xs[k]), ref[k]
            started = k < len(guess)
            if started:
                assert its[k] == 0
            elif precision == 0:
                assert abs(its[k] - itsref) <= 1, (k, its[k], itsref)
            assert res[k] <= tol, (k, res[k])
            assert H.rel_to_max(x, xref) < 100 * tol, k
