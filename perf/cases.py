"""The performance cases of chfem_b200: what a user of the framework has it do.

Almost every user hands over a voxel (or pixel) image and the phases' properties and wants an
effective tensor, so most cases are whole calls of compute_property or
compute_conductivity_batch: image in host memory -> tensor, new inputs each time.  The rest are
the drop-in C ABI driven by a host program that keeps the solution vector, and a training step
of the network behind the learned initial guess.

A case's "kind" names the path, and its other entries the sizes and options:
  conductivity / elasticity / permeability   compute_property on an nz x ny x nx image
                                             (nz = 0: an ny x nx pixel image)
  batch                                      compute_conductivity_batch on n images
  abi                                        the cudapcg C ABI: model, right-hand side, solve, x
  unet                                       Net.forward, mse, backward
"""
import ctypes
import itertools
import math
import os
import tempfile

import numpy as np
import torch

TOL = 1e-6  # the default solver tolerance of compute_property
CODES = (0, 255, 100, 50)
CONDUCTIVITY = (1.0, 10.0, 3.0, 0.5)
ELASTICITY = ((1.0, 0.30), (10.0, 0.20), (4.0, 0.25), (0.5, 0.35))


def listed():
    return [
        # the smallest call: a 16 x 14 x 12 image, where launches and host work are what counts
        dict(name="conductivity_tiny", kind="conductivity", nz=12, ny=14, nx=16, phases=2, precision="fp64", block=False, corr=2.0),
        # the 64^3 two-phase conductivity of the framework's first benchmark workload, defaults
        dict(name="conductivity_64", kind="conductivity", nz=64, ny=64, nx=64, phases=2, precision="fp64", block=False, corr=5.0),
        # the large end of plain FP64 conductivity, one direction after the other
        dict(name="conductivity_256", kind="conductivity", nz=256, ny=256, nx=256, phases=2, precision="fp64", block=False, corr=6.0),
        # a ragged scan with four phases, FP32 fields, all directions as one block
        dict(name="conductivity_ragged_mixed_block", kind="conductivity", nz=97, ny=75, nx=130, phases=4, precision="mixed", block=True, corr=5.0),
        # many independent images in one call, edges as in the batch benchmark (32 to 96)
        dict(name="batch_mixed", kind="batch", n=24, lo=32, hi=96, precision="mixed"),
        # the default elasticity call: FP64, six load cases one after the other
        dict(name="elasticity_96", kind="elasticity", nz=96, ny=96, nx=96, phases=2, precision="fp64", block=False, learned=False, corr=6.0),
        # the flagship workload: 128^3, FP32 fields, six load cases as one block, learned guess
        dict(name="elasticity_128_mixed_block_learned", kind="elasticity", nz=128, ny=128, nx=128, phases=2, precision="mixed", block=True,
             learned=True, corr=6.0),
        # pixel images (2D, plane strain), ragged
        dict(name="elasticity_pixels", kind="elasticity", nz=0, ny=217, nx=300, phases=3, precision="fp64", block=False, learned=False, corr=6.0),
        # a host program on the C ABI: a ragged three-phase elastic model, one load case, x back
        dict(name="abi_elastic_ragged", kind="abi", nz=50, ny=61, nx=45, phases=3, corr=4.0),
        # Stokes permeability with the default solver, three flow directions one after the other
        dict(name="permeability_96", kind="permeability", nz=96, ny=96, nx=96, block=False, porosity=0.35, corr=6.0),
        # a ragged, more open pore space, the flow directions as one block
        dict(name="permeability_ragged_block", kind="permeability", nz=40, ny=57, nx=64, block=True, porosity=0.5, corr=4.0),
        # training of the guess network: forward, loss and backward on a batch of 64^3 samples
        dict(name="unet_step", kind="unet", n=2, size=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["conductivity", "conductivity", "elasticity", "elasticity", "permeability", "batch", "abi", "unet"])
    if kind == "unet":
        return dict(kind=kind, n=rng.randint(1, 4), size=8 * rng.randint(3, 8))
    if kind == "batch":
        lo = rng.randint(12, 40)
        return dict(kind=kind, n=rng.randint(4, 32), lo=lo, hi=lo + rng.randint(0, 56), precision=rng.choice(["fp64", "mixed"]))
    # an edge over its whole range, the other two within a factor of two of it
    top = dict(conductivity=200, elasticity=96, permeability=80, abi=80)[kind]
    edge = _log_int(rng, 12 if kind != "permeability" else 24, top)
    nz, ny, nx = (max(8, min(top, int(edge * math.exp(rng.uniform(-0.35, 0.35))))) for _ in range(3))
    corr = round(rng.uniform(2.0, 6.0), 2)
    if kind == "permeability":
        return dict(kind=kind, nz=nz, ny=ny, nx=nx, block=rng.random() < 0.5, porosity=round(rng.uniform(0.4, 0.6), 3), corr=corr)
    phases = rng.randint(2, 4)
    if kind == "abi":
        return dict(kind=kind, nz=nz, ny=ny, nx=nx, phases=phases, corr=corr)
    if rng.random() < 0.2:
        nz, ny, nx = 0, _log_int(rng, 40, 400), _log_int(rng, 40, 400)
    case = dict(kind=kind, nz=nz, ny=ny, nx=nx, phases=phases, precision=rng.choice(["fp64", "mixed"]), block=nz > 0 and rng.random() < 0.5,
                corr=corr)
    if kind == "elasticity":
        case["learned"] = False
    return case


# ---- inputs -----------------------------------------------------------------------------
def _gpu():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _field(shape, corr, seed):
    """A periodic Gaussian random field (white noise smoothed in Fourier space)."""
    g = torch.Generator().manual_seed(int(seed))
    f = torch.fft.fftn(torch.randn(shape, generator=g, dtype=torch.float32).to(_gpu()))
    for ax, n in enumerate(shape):
        k = torch.fft.fftfreq(n, device=f.device)
        f = f * torch.exp(-2.0 * (math.pi * corr * k) ** 2).reshape([-1 if a == ax else 1 for a in range(len(shape))])
    return torch.fft.ifftn(f).real


def _image(shape, phases, corr, seed):
    """uint8 image of 2 to 4 phases: bands of a random field, phase 0 the largest."""
    f = _field(shape, corr, seed)
    order = torch.argsort(torch.argsort(f.flatten())) if phases > 2 else None
    img = torch.zeros(f.numel(), dtype=torch.uint8, device=f.device)
    if phases == 2:  # 40 % of the second phase
        cut = torch.kthvalue(f.flatten(), max(1, int(0.6 * f.numel()))).values
        img[f.flatten() > cut] = CODES[1]
    else:
        share = 0.55 / (phases - 1)
        for p in range(1, phases):
            img[order >= int((0.45 + share * (p - 1)) * f.numel())] = CODES[p]
    return np.ascontiguousarray(img.reshape(f.shape).cpu().numpy())


def _pores(case, seed):
    """Pore space of the given porosity; only what percolates, where anything does."""
    from chfem_b200 import synthetic
    shape = (case["nz"], case["ny"], case["nx"])
    img = synthetic.pore_grf(shape, corr=case["corr"], porosity=case["porosity"], seed=seed)
    if not (img == 0).any():
        img = np.where(synthetic.grf(shape, corr=case["corr"], fraction=1.0 - case["porosity"], seed=seed) == 0, 0, 255).astype(np.uint8)
    return img


def _shape(case):
    return (case["nz"], case["ny"], case["nx"]) if case["nz"] else (case["ny"], case["nx"])


def _props(case, img):
    table = ELASTICITY if case["kind"] in ("elasticity", "abi") else CONDUCTIVITY
    return {c: table[i] for i, c in enumerate(CODES) if (img == c).any()}


def _batch(case, seed):
    rng = np.random.default_rng(seed)
    images, props = [], []
    for s in range(case["n"]):
        edge = case["lo"] + (case["hi"] - case["lo"]) * s // max(1, case["n"] - 1)  # the same sizes for every seed
        images.append(_image((edge, edge, edge), 2, 3.0, seed * 1000 + s))
        props.append({0: 1.0, 255: float(math.exp(rng.uniform(math.log(2.0), math.log(100.0))))})
    return images, props


def _unet_inputs(case, seed):
    """Two-phase images' material features and a smooth target, as the training loop holds them."""
    from chfem_b200 import learned
    n, size = case["n"], case["size"]
    g = torch.Generator().manual_seed(int(seed))
    feat = torch.zeros((n, learned.IN_CH, size, size, size))
    for s in range(n):
        img = torch.from_numpy(_image((size, size, size), 2, 6.0, seed * 100 + s))
        contrast = math.log(2.0 + 48.0 * float(torch.rand(1, generator=g))) / math.log(50.0)
        feat[s, 0] = (img > 0) * contrast
        feat[s, 1] = torch.where(img > 0, -0.2, 0.2)
    target = torch.stack([torch.stack([_field((size, size, size), 4.0, seed * 10007 + 97 * s + c) for c in range(learned.OUT_CH)]) for s in range(n)])
    target = (target / target.std()).float()
    return feat.to(_gpu()).contiguous(), target.to(_gpu()).contiguous()


def _abi_arrays(case, seed):
    """The maps, matrices and right-hand side that a host program hands over the C ABI."""
    from chfem_b200 import _native
    from chfem_b200.io import export_for_chfem
    img = _image(_shape(case), case["phases"], case["corr"], seed)
    h = _native.chfem()
    h.chfemB200SetQuiet(1)
    with tempfile.TemporaryDirectory() as d:
        export_for_chfem(os.path.join(d, "m.raw"), img, 1, mat_props=_props(case, img), solver_tolerance=TOL, export_raw=False)
        flat = np.ascontiguousarray(img.reshape(-1))
        if not h.hmgInit(os.path.join(d, "m.nf").encode(), None, None, flat.ctypes.data_as(ctypes.c_void_p)):
            raise RuntimeError(h.chfemB200LastError().decode())
    info = (ctypes.c_uint * 9)()
    h.chfemB200ModelInfo(info)

    def copied(which, dtype):
        a = np.zeros(h.chfemB200ModelArraySize(which) // np.dtype(dtype).itemsize, dtype=dtype)
        if a.size:
            h.chfemB200CopyModelArray(which, a.ctypes.data_as(ctypes.c_void_p), a.nbytes)
        return a
    a = dict(nx=info[0], ny=info[1], nz=info[2], N=info[3], ndof=info[4], nV=info[5], nB=info[6], nkeys=info[7], analysis=info[8],
             keys=copied(0, np.uint16), dof_of_node=copied(1, np.uint32), node_of_dof=copied(2, np.uint32), border=copied(3, np.uint8),
             lcl=copied(4, np.float64))
    rhs = np.zeros(a["ndof"])
    h.chfemB200AssembleRHS(0, rhs.ctypes.data_as(ctypes.c_void_p))
    h.hmgEnd()
    return dict(arrays=a, rhs=rhs, x=np.zeros(a["ndof"]))


def prepare(case, seed):
    from chfem_b200 import _native
    state = dict(case=case)
    if case["kind"] == "unet":
        from chfem_b200 import learned
        feat, target = _unet_inputs(case, seed)
        state.update(net=learned.Net(seed=seed), feat=feat, target=target, grad=torch.zeros_like(target))
        return state
    _native.chfem().chfemB200SetQuiet(1)
    if case["kind"] == "abi":
        state.update(_abi_arrays(case, seed))
    elif case["kind"] == "batch":
        state["images"], state["props"] = _batch(case, seed)
    elif case["kind"] == "permeability":
        state["image"] = _pores(case, seed)
    else:
        state["image"] = _image(_shape(case), case["phases"], case["corr"], seed)
        state["props"] = _props(case, state["image"])
    return state


# ---- one pass ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "unet":
        net = state["net"]
        out = net.forward(state["feat"])
        loss = net.mse(out, state["target"], state["grad"])
        net.backward(state["grad"])
        return {"out": out, "loss": loss, "grad": net.g}
    if case["kind"] == "abi":
        return _run_abi(state)
    import chfem_b200
    if case["kind"] == "batch":
        return chfem_b200.compute_conductivity_batch(state["images"], state["props"], precision=case["precision"])
    if case["kind"] == "permeability":
        C = chfem_b200.compute_property("permeability", state["image"], voxel_size=1.0, multirhs=case["block"])
    else:
        C = chfem_b200.compute_property(case["kind"], state["image"], mat_props=state["props"], precision=case["precision"],
                                        multirhs=case["block"], initial_guess="learned" if case.get("learned") else None)
    return np.array(C)


def _run_abi(state):
    from chfem_b200 import _native
    lib = _native.cudapcg()
    _native.setup_cudapcg_model(lib, state["arrays"])
    ok = (lib.cudapcgSetSolver(0) and lib.cudapcgSetPreconditioner(1) and lib.cudapcgSetNumTol(TOL) and lib.cudapcgSetMaxIterations(10000) and
          lib.cudapcgAllocateArrays() and lib.cudapcgSetRHS(state["rhs"].ctypes.data_as(ctypes.c_void_p)) and
          lib.cudapcgSolve(state["x"].ctypes.data_as(ctypes.c_void_p)))
    if not ok:
        raise RuntimeError(lib.cudapcgB200LastError().decode())
    lib.cudapcgEnd()
    return state["x"]


# ---- what a pass cannot do without --------------------------------------------------------
def work(case):
    """Bytes and operations of one pass.

    A solve: per iteration of the conjugate-gradient (Stokes: conjugate-residual) recurrence each
    vector of its state is read once and written once -- x, r, d and q = A d (8 bytes each in
    FP64; FP32 except x under mixed precision), for Stokes also A M^-1 r -- and the element matrix
    of every voxel is applied in the cheapest form the repository has, 27 neighbour blocks per
    node.  The iteration count is that of the case's size and contrast at tolerance 1e-6, counted
    once and fitted to the edge of the image.  The network: its tensors once per pass, and two
    operations per multiply-add of the convolutions, forward and both backward products."""
    kind = case["kind"]
    if kind == "unet":
        s, n = case["size"] ** 3, case["n"]
        ch = (16, 32, 48, 64)
        macs = [(s, 16 * 2 * 27), (s // 8, 32 * 16 * 27), (s // 64, 48 * 32 * 27), (s // 512, 64 * 48 * 27),
                (s // 64, 48 * 112 * 27), (s // 8, 32 * 80 * 27), (s, 16 * 48 * 27), (s, 18 * 16)]
        words = s * (2 + ch[0] + ch[0] + 18) + (s // 8) * 2 * ch[1] + (s // 64) * 2 * ch[2] + (s // 512) * ch[3]
        return {"bytes": float(3 * 4 * n * words), "flops": float(3 * 2 * n * sum(a * b for a, b in macs))}
    if kind == "batch":
        nodes = sum((case["lo"] + (case["hi"] - case["lo"]) * s // max(1, case["n"] - 1)) ** 3 for s in range(case["n"]))
        edge, dof, cases, mixed = (case["lo"] + case["hi"]) / 2, 1, 3, case["precision"] == "mixed"
    else:
        sh = _shape(case)
        nodes, edge = float(np.prod(sh)), float(np.prod(sh)) ** (1.0 / len(sh))
        dof = 1 if kind == "conductivity" else len(sh)
        cases = 1 if kind == "abi" else (3 if dof == 1 else 6) if len(sh) == 3 else (2 if dof == 1 else 3)
        mixed = case.get("precision") == "mixed"
    neighbours = 9 if case.get("nz") == 0 else 27
    if kind == "permeability":
        unknowns, its = nodes * case["porosity"] * 4, 8.0 * edge
        return {"bytes": 3 * its * unknowns * 80.0, "flops": 3 * its * nodes * case["porosity"] * 2.0 * neighbours * 16}
    its = (2.0 if dof == 1 else 4.0) * edge + 30.0
    return {"bytes": cases * its * nodes * dof * (40.0 if mixed else 64.0), "flops": cases * its * nodes * 2.0 * neighbours * dof * dof}


def tolerance(case):
    """Largest relative error another correct implementation would show: four times what was seen.

    Tensors come from iterations stopped at a relative residual of 1e-6: up to 7e-6 from the exact
    ones, and Stokes permeabilities up to 5.5e-6 from those of a tolerance of 1e-10.  Solution
    vectors likewise.  The network is FP32 with sums over up to a million terms: its gradients
    are 9e-6 from FP64's."""
    if case["kind"] == "unet":
        return {"rel": 4e-5, "max": 4e-3}
    if case["kind"] == "permeability":
        return {"rel": 4e-5, "max": 4e-4}
    if case["kind"] == "abi":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 3e-5, "max": 3e-4}


# ---- the same in 64 bits, with plain torch ------------------------------------------------
def _element(dim, dof, prop):
    """Q1 element matrix of a unit cube (square) by Gauss quadrature: corners in binary order,
    axes (x, y[, z]); conduction (dof 1) or isotropic elasticity (plane strain in 2D).  Also the
    strain (gradient) matrix integrated over the element and the constitutive matrix."""
    corners = list(itertools.product((0, 1), repeat=dim))
    pts = [0.5 - 0.5 / math.sqrt(3.0), 0.5 + 0.5 / math.sqrt(3.0)]
    if dof == 1:
        D = prop * np.eye(dim)
    else:
        E, nu = prop
        lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
        ns = 6 if dim == 3 else 3
        D = np.zeros((ns, ns))
        D[:dim, :dim] = lam
        D[np.arange(dim), np.arange(dim)] += 2 * mu
        D[np.arange(dim, ns), np.arange(dim, ns)] = mu
    K, Bbar = 0.0, 0.0
    for g in itertools.product(pts, repeat=dim):
        dN = np.zeros((dim, len(corners)))
        for a, c in enumerate(corners):
            for i in range(dim):
                dN[i, a] = np.prod([(1 if c[j] else -1) if j == i else (g[j] if c[j] else 1 - g[j]) for j in range(dim)])
        if dof == 1:
            B = dN
        else:
            B = np.zeros((D.shape[0], dim * len(corners)))
            shear = [(1, 2), (0, 2), (0, 1)] if dim == 3 else [(0, 1)]
            for a in range(len(corners)):
                for i in range(dim):
                    B[i, dim * a + i] = dN[i, a]
                for s, (i, j) in enumerate(shear):
                    B[dim + s, dim * a + i] = dN[j, a]
                    B[dim + s, dim * a + j] = dN[i, a]
        w = 1.0 / 2 ** dim
        K = K + w * B.T @ D @ B
        Bbar = Bbar + w * B
    return K, Bbar, D


def _homogenize(img, props, dof):
    """Effective tensor of a periodic image in FP64: periodic corrector per unit macroscopic
    gradient by conjugate gradients, C_ij = mean of (e_i + grad chi_i) D (e_j + grad chi_j)."""
    dim = img.ndim
    img = img[tuple(slice(None, None, -1) if a != dim - 1 else slice(None) for a in range(dim))].copy()  # y and z run against the image's axes
    dev = _gpu()
    lab = torch.from_numpy(img).to(dev)
    mats = [(c, *(torch.tensor(v, device=dev, dtype=torch.float64) for v in _element(dim, dof, p))) for c, p in props.items()]
    corners = list(itertools.product((0, 1), repeat=dim))
    axes = tuple(dim - 1 - i for i in range(dim))  # array axis of x, y, z
    masks = [(lab == c).reshape(-1).to(torch.float64) for c, *_ in mats]

    def gather(u):  # [dof, *shape] -> [corner * dof, cells]
        return torch.cat([torch.roll(u, [-c for c in cn], [1 + a for a in axes]).reshape(dof, -1) for cn in corners])

    def scatter(f):
        out = torch.zeros((dof,) + tuple(lab.shape), device=dev, dtype=torch.float64)
        for k, cn in enumerate(corners):
            out += torch.roll(f[k * dof:(k + 1) * dof].reshape(out.shape), list(cn), [1 + a for a in axes])
        return out

    def weighted(pick, u):  # sum over phases of matrix @ u on the phase's cells
        out = pick(mats[0]) @ u
        for m, mask in zip(mats[1:], masks[1:]):
            out += ((pick(m) - pick(mats[0])) @ u) * mask
        return out

    diag = scatter(weighted(lambda m: torch.diag(m[1])[:, None], torch.ones((1, lab.numel()), device=dev, dtype=torch.float64)))
    ns = mats[0][3].shape[0]
    chis, flux = [], []
    for s in range(ns):
        e = torch.zeros((ns, 1), device=dev, dtype=torch.float64)
        e[s] = 1.0
        load = weighted(lambda m: m[2].T @ m[3] @ e, torch.ones((1, lab.numel()), device=dev, dtype=torch.float64))
        b = -scatter(load)
        x, r = torch.zeros_like(b), b.clone()
        z = r / diag
        d, rz = z.clone(), torch.sum(r * z)
        rz0 = float(rz)
        for it in range(20000):
            if it % 10 == 0 and not float(rz) > 1e-16 * rz0:
                break
            q = scatter(weighted(lambda m: m[1], gather(d)))
            alpha = rz / torch.sum(d * q)
            x += alpha * d
            r -= alpha * q
            z = r / diag
            new = torch.sum(r * z)
            d = z + (new / rz) * d
            rz = new
        chis.append(x)
        del b, r, z, d
    C = torch.zeros((ns, ns), device=dev, dtype=torch.float64)
    for s in range(ns):
        u = gather(chis[s])
        for (c, K, Bbar, D), mask in zip(mats, masks):
            C[:, s] += D @ (Bbar @ (u @ mask)) + D[:, s] * mask.sum()
        del u
    return (C / lab.numel()).cpu().numpy()


def _unet_exact(case, seed):
    from torch.nn import functional as F
    from chfem_b200 import learned  # the parameters' start values and layout
    feat, target = _unet_inputs(case, seed)
    net = learned.Net(seed=seed, device=_gpu())
    p = net.p.double().requires_grad_(True)

    def conv(name, x, relu=True):
        w0, b0, co, ci, k = net.offsets[name]
        w, b = p[w0:b0].reshape(co, ci, k, k, k), p[b0:b0 + co]
        y = F.conv3d(F.pad(x, [k // 2] * 6, mode="circular") if k > 1 else x, w, b)
        return torch.relu(y) if relu else y

    def up(x):
        return x.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
    x0 = conv("enc0", feat.double())
    x1 = conv("enc1", F.avg_pool3d(x0, 2))
    x2 = conv("enc2", F.avg_pool3d(x1, 2))
    x3 = conv("enc3", F.avg_pool3d(x2, 2))
    d2 = conv("dec2", torch.cat([up(x3), x2], 1))
    d1 = conv("dec1", torch.cat([up(d2), x1], 1))
    d0 = conv("dec0", torch.cat([up(d1), x0], 1))
    out = conv("head", d0, relu=False)
    loss = F.mse_loss(out, target.double())
    loss.backward()
    return {"out": out.detach(), "loss": float(loss), "grad": p.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("permeability", "abi"):
        return None
    if kind == "unet":
        return _unet_exact(case, seed)
    if not torch.cuda.is_available() and work(case)["bytes"] > 2e10:
        return None  # minutes on the host's cores
    if kind == "batch":
        images, props = _batch(case, seed)
        return np.stack([_homogenize(i, p, 1) for i, p in zip(images, props)])
    img = _image(_shape(case), case["phases"], case["corr"], seed)
    return _homogenize(img, _props(case, img), 1 if kind == "conductivity" else img.ndim)
