"""Host side of the solver library over a stand-in for the CUDA runtime (fake_cuda.py): launch
settings per device, and the order of uploads with the solver's stream."""
import os
import pickle
import subprocess
import sys

import numpy as np
import pytest

from tests import fake_cuda
from tests import helpers as H

pytestmark = pytest.mark.skipif(not fake_cuda.available(), reason="needs g++ and the built objects")

# run in a child process: the stand-in's names are the CUDA runtime's
PREAMBLE = r'''
import ctypes, pickle, sys
import numpy as np
sys.path.insert(0, sys.argv[3])
from chfem_b200._native import setup_cudapcg_model as setup
lib = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_LOCAL)
lib.fake_report.restype = ctypes.c_char_p
models = pickle.load(open(sys.argv[2], "rb"))
P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
lib.cudapcgB200LastError.restype = ctypes.c_char_p
lib.cudapcgSetParametricDensityField.argtypes = [ctypes.c_void_p, ctypes.c_double, ctypes.c_double]
def apply(a):
    x, y = np.ones(a["ndof"]), np.zeros(a["ndof"])
    assert lib.cudapcgB200ApplyOperator(P(x), P(y)), lib.cudapcgB200LastError()
def block(a):
    n = {0: 3, 1: 6}[a["analysis"]]
    v = [np.ones(a["ndof"]) for _ in range(n)]; y = [np.zeros(a["ndof"]) for _ in range(n)]
    arr = lambda vs: (ctypes.c_void_p * n)(*[w.ctypes.data for w in vs])
    assert lib.cudapcgB200ApplyBlockOperator(n, arr(v), arr(y)), lib.cudapcgB200LastError()
class Scalars(ctypes.Structure):  # DevScalars (common.cuh)
    _fields_ = [(n, ctypes.c_double) for n in "delta delta0 delta_old alpha beta res0 metric".split()] + [
        ("red", ctypes.c_double * 6), ("xa", ctypes.c_double)] + [(n, ctypes.c_int) for n in "iteration done found status".split()]
lib.fake_finish(ctypes.c_size_t(ctypes.sizeof(Scalars)), ctypes.c_size_t(Scalars.done.offset))
lib.cudapcgSetNumTol.argtypes = [ctypes.c_double]
def solve(a):
    x = np.zeros(a["ndof"])
    lib.cudapcgSolve(P(x))
    assert not lib.cudapcgB200LastError(), lib.cudapcgB200LastError()
def rhs(a):
    assert lib.cudapcgSetRHS(P(np.ones(a["ndof"]))), lib.cudapcgB200LastError()
def free_of(fault, what):
    lines = [l for l in lib.fake_report().decode().split("\n") if l and fault in l]
    assert not lines, what + ": " + "; ".join(sorted(set(lines)))
'''


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    """The library and one model of every analysis, in the formats of the C ABI."""
    from tests.test_gpu_parity import host_arrays
    wd = tmp_path_factory.mktemp("fake")
    lib = fake_cuda.build(wd)
    rng = np.random.default_rng(1)
    models = {}
    for name, analysis, nmat in (("thermal", 0, 3), ("elastic", 1, 3), ("elastic2", 1, 2), ("fluid", 2, 2)):
        img = H.small_image((6, 7, 8), nmat, seed=2) if analysis < 2 else np.where(rng.random((6, 7, 8)) < 0.8, 0, 255).astype(np.uint8)
        models[name] = host_arrays(*H.write_small_case(str(wd), name, img, analysis))
    # a matrix that is not isotropic: the passes assembled by neighbour
    models["other"] = dict(models["elastic2"], lcl=models["elastic2"]["lcl"].copy())
    K = models["other"]["lcl"].reshape(-1, 24, 24)
    K[:, 0::3, 0::3] *= 1.2
    pk = os.path.join(str(wd), "models.pkl")
    pickle.dump(models, open(pk, "wb"))

    def run(script):
        p = subprocess.run([sys.executable, "-c", PREAMBLE + script, lib, pk, H.ROOT], capture_output=True, text=True, timeout=300,
                           cwd=str(wd))
        assert p.returncode == 0, p.stdout[-2000:] + p.stderr[-2000:]
    return run


def test_launch_settings_hold_on_every_device(fake):
    """Large dynamic shared memory is granted per device, and a process may solve on one device
    after another: every operator pass opts in on each, once."""
    fake(r'''
asked = []
for turn in range(2):
    for device in (0, 3):
        lib.fake_set_device(device)
        before = lib.fake_asked()
        for name in ("thermal", "elastic", "other"):
            for precision in (0, 1):
                setup(lib, models[name])
                lib.cudapcgB200SetPrecision(precision)
                apply(models[name]); block(models[name])
                free_of("shared memory", f"{name} on device {device}")
                lib.cudapcgEnd()
        asked.append(lib.fake_asked() - before)
assert asked[0] == asked[1] > 0 and asked[2:] == [0, 0], asked
''')


def test_uploads_and_passes_are_ordered(fake):
    """Whatever is uploaded on the legacy stream is in place before a pass on the solver's stream, and
    no upload meets a fill that is still queued there -- for every entry point that takes model data,
    also on a model whose vectors exist already (no allocation in between)."""
    fake(r'''
for name in ("thermal", "elastic", "other", "fluid"):
    a = models[name]
    fluid = name == "fluid"
    for precision in (0, 1):
        setup(lib, a)
        lib.cudapcgB200SetPrecision(precision)
        lib.cudapcgSetSolver(1 if fluid else 0)
        apply(a); rhs(a); solve(a)
        free_of("", name)
        guess = np.ones(a["ndof"])
        keep = [np.ascontiguousarray(a[k]) for k in ("keys", "dof_of_node", "border", "node_of_dof", "lcl")]
        steps = [lambda: lib.cudapcgSetX0(P(guess), 0), lambda: lib.cudapcgB200SetX0Device(P(guess)), lambda: lib.cudapcgSetX0(None, 0),
                 lambda: lib.cudapcgSetX0(P(guess), 0), lambda: lib.cudapcgSetLclMtxs(P(keep[4]))]
        if fluid:
            steps += [lambda: lib.cudapcgSetPeriodic2DOFMap(P(keep[1])), lambda: lib.cudapcgSetPoreMap(P(keep[2])),
                      lambda: lib.cudapcgSetDOF2PeriodicMap(P(keep[3]))]
        else:
            density = np.full(a["N"], 7, np.uint16)
            steps += [lambda: lib.cudapcgSetImage(P(keep[0])), lambda: lib.cudapcgSetParametricDensityField(P(density), 0.5, 1.5),
                      lambda: lib.cudapcgSetImage(P(keep[0]))]
        for i, step in enumerate(steps):
            assert step(), (i, lib.cudapcgB200LastError())
            rhs(a); solve(a)
            free_of("", f"{name}, precision {precision}, step {i}")
        lib.cudapcgEnd()
        n = 6 if name in ("elastic", "other") else 3
        arr = lambda vs: (ctypes.c_void_p * n)(*[v.ctypes.data for v in vs])
        b, x, g = ([np.ones(a["ndof"]) for _ in range(n)] for _ in range(3))
        setup(lib, a)
        lib.cudapcgB200SetPrecision(precision)
        lib.cudapcgSetSolver(1 if fluid else 0)
        for mode in (0, 2, 0, 2):
            lib.cudapcgB200SolveBlock(n, arr(b), arr(g), mode, arr(x), None, None)
            assert not lib.cudapcgB200LastError(), lib.cudapcgB200LastError()
            free_of("", f"{name} block, precision {precision}, guess {mode}")
        lib.cudapcgEnd()
''')


def test_captured_passes_follow_the_settings(fake):
    """A graph of passes captured for one tolerance, iteration limit, norm, preconditioner or solver
    is not replayed under another; the same settings replay it."""
    fake(r'''
lib.cudapcgSetMaxIterations.argtypes = [ctypes.c_uint]
for name in ("thermal", "elastic", "fluid"):
    a = models[name]
    minres = 1 if name == "fluid" else 0
    n = 6 if name == "elastic" else 3
    arr = lambda vs: (ctypes.c_void_p * n)(*[v.ctypes.data for v in vs])
    b, x = [np.ones(a["ndof"]) for _ in range(n)], [np.zeros(a["ndof"]) for _ in range(n)]
    def solve_block(a):
        lib.cudapcgB200SolveBlock(n, arr(b), None, 0, arr(x), None, None)
        assert not lib.cudapcgB200LastError(), lib.cudapcgB200LastError()
    solvers = [(minres, solve), (minres, solve_block)] + ([(5, solve)] if minres else [(2, solve), (1, solve)])
    for solver, run in solvers:
        setup(lib, a)
        lib.cudapcgSetSolver(solver)
        def captures():
            before = lib.fake_graphs()
            if run is solve: rhs(a)
            run(a)
            return lib.fake_graphs() - before
        assert captures() == 1 and captures() == 0
        for change in (lambda: lib.cudapcgSetNumTol(1e-3), lambda: lib.cudapcgSetMaxIterations(77), lambda: lib.cudapcgSetResNorm(1),
                       lambda: lib.cudapcgSetPreconditioner(0), lambda: lib.cudapcgB200SetIterationsPerLaunch(8)):
            assert change()
            assert captures() == 1, (name, solver)
            assert captures() == 0, (name, solver)
        lib.cudapcgEnd()
''')


def test_jacobi_diagonal_follows_the_image(fake):
    """Under a density field the inverse diagonal is computed once per model from keys and density:
    a new image on the same model drops it, and the graphs that hold its address."""
    fake(r'''
import tempfile
for name in ("thermal", "elastic"):
    a = models[name]
    setup(lib, a)
    density = np.full(a["N"], 7, np.uint16)
    assert lib.cudapcgSetParametricDensityField(P(density), 0.5, 1.5)
    keys = np.ascontiguousarray(a["keys"])
    colors = np.zeros(a["N"], np.uint8)
    lut = (ctypes.c_int * 256)(*([0] * 256))
    rhs(a); solve(a)
    for image in (lambda: lib.cudapcgSetImage(P(keys)),
                  lambda: lib.cudapcgB200SetImageColors(P(colors), a["ny"], a["nx"], a["nz"], 1, lut)):
        launched, graphs = lib.fake_launches(), lib.fake_graphs()
        rhs(a); solve(a)
        same = lib.fake_launches() - launched
        assert lib.fake_graphs() == graphs
        assert image(), lib.cudapcgB200LastError()
        launched = lib.fake_launches()
        rhs(a); solve(a)
        assert lib.fake_launches() - launched > same and lib.fake_graphs() == graphs + 1, name
    lib.cudapcgEnd()
''')


def test_device_bytes_of_minres(fake):
    """(P)MINRES keeps one direction buffer: x, b, r, r', d, q, s on thermal and elastic models (56 B
    per unknown in FP64; 44 B mixed, with the FP64 scratch of the residual replacement), x, b, r,
    d, q, s and the records of M^-1 r on Stokes models; the operator can still be applied."""
    fake(r'''
lib.cudapcgB200DeviceBytes.restype = ctypes.c_ulonglong
for name in ("thermal", "elastic", "fluid"):
    a = models[name]
    for precision in (0, 1) if name != "fluid" else (0,):
        setup(lib, a)
        lib.cudapcgB200SetPrecision(precision)
        lib.cudapcgSetSolver(1)
        rhs(a); solve(a)
        held = lib.cudapcgB200DeviceBytes()
        if name == "fluid":
            nodes = a["nV"] + a["nB"]
            records = 32 * (a["N"] if a["N"] <= 4 * nodes else nodes)
            assert held <= 48 * a["ndof"] + records + 4 * a["N"] + 4 * nodes + a["nB"], held / a["ndof"]
        else:
            assert held <= (44 if precision else 56) * a["ndof"] + 2 * a["N"], (name, precision, held / a["ndof"])
        apply(a)
        lib.cudapcgB200TimeOperator.restype = lib.cudapcgB200TimeKernel.restype = ctypes.c_double
        assert lib.cudapcgB200TimeOperator(1) > 0
        assert all(lib.cudapcgB200TimeKernel(which, 1) > 0 for which in range(5)), lib.cudapcgB200LastError()
        free_of("", name)
        lib.cudapcgEnd()
''')


def test_trim_releases_what_is_kept(fake):
    """A solver's and a batch's stream, events and pinned record outlive them, serve the next, and go
    with cudapcgB200TrimMemory, as do those of batches in several threads."""
    fake(r'''
import threading
lib.cudapcgB200BatchLastError.restype = ctypes.c_char_p
a = models["thermal"]
def batch():
    keys, nmat, K, CB = np.ascontiguousarray(a["keys"]), np.array([a["nkeys"]], np.uint32), np.ones(256), np.ones(96)
    one = lambda v: (ctypes.c_void_p * 1)(v.ctypes.data)
    dims = np.array([[a["ny"], a["nx"], a["nz"]]], np.uint32)
    m, its, res = np.zeros(9), np.zeros(3, np.uint32), np.zeros(3)
    assert lib.cudapcgB200SolveThermalBatch(ctypes.c_uint(1), P(dims), one(keys), P(nmat), one(K), one(CB), ctypes.c_double(1e-6),
                                            ctypes.c_uint(10), 0, 1, P(m), P(its), P(res), None), lib.cudapcgB200BatchLastError()
for turn in range(2):
    setup(lib, a); rhs(a); solve(a); lib.cudapcgEnd()
    batch()
    kept = lib.fake_live()
    assert kept > 0
    setup(lib, a); rhs(a); solve(a); lib.cudapcgEnd()
    batch()
    assert lib.fake_live() == kept
    threads = [threading.Thread(target=batch) for _ in range(8)]
    [t.start() for t in threads]; [t.join() for t in threads]
    assert lib.cudapcgB200TrimMemory() and lib.fake_live() == 0, lib.fake_live()
''')


def test_batches_in_threads_keep_their_own_state(fake):
    """Batches of many signatures at once, sound and refused ones: every thread reads its own error,
    and the tile choices they store in common are complete."""
    fake(r'''
import threading
lib.cudapcgB200BatchLastError.restype = ctypes.c_char_p
wrong = []
def batch(shape, nmat):
    n = int(np.prod(shape))
    keys, nmats, K, CB = np.zeros(n, np.uint16), np.array([nmat], np.uint32), np.ones(256), np.ones(96)
    one = lambda v: (ctypes.c_void_p * 1)(v.ctypes.data)
    m, its, res = np.zeros(9), np.zeros(3, np.uint32), np.zeros(3)
    rc = lib.cudapcgB200SolveThermalBatch(ctypes.c_uint(1), P(np.array([shape], np.uint32)), one(keys), P(nmats), one(K), one(CB),
                                          ctypes.c_double(1e-6), ctypes.c_uint(10), 0, 1, P(m), P(its), P(res), None)
    return rc, lib.cudapcgB200BatchLastError()
def work(t):
    for i in range(40):
        rc, err = batch((2 + t, 3 + i, 4), 1)
        if not rc or err: wrong.append((rc, err))
        rc, err = batch((2 + t, 3 + i, 4), 9)
        if rc or b"materials" not in err: wrong.append((rc, err))
threads = [threading.Thread(target=work, args=(t,)) for t in range(8)]
[t.start() for t in threads]; [t.join() for t in threads]
assert not wrong, wrong[:3]
''')


def test_single_passes_are_small_modules():
    """The first launch of a kernel loads its whole module: the passes of one right-hand side are kept
    apart from each other's field types and from the blocks', a megabyte or less each."""
    sizes = {o: os.path.getsize(o) for o in fake_cuda.OBJECTS if o.endswith(("_PASS.o", "_DENSITY.o", "_POINT.o"))}
    assert len(sizes) == 12 and max(sizes.values()) < 1.2e6, sizes
