"""Work that programs have this library do, as cases that can be timed and compared.

A case is one call through the public entry points of the Python binding (the C table's
`gemv` and `assemble_generic`, the device-pointer products, the fused adjoint, the batches):

  product   y = op(H) x on device buffers (hmat_b200_gemv_device); `batch` > 0: the
            block-diagonal matrix of that many members
  host      y = op(H) x on host buffers through the C table's gemv, copies included
  adjoint   dx = H^T r and the gradients of every leaf factor (hmat_b200_gemv_adjoint)
  assemble  the H-matrix computed on a cluster and block tree that the program holds (a new
            kernel parameter on known points, say), then multiplied once: outputs are the leaf
            table (partition and ranks) and the product

Geometries, kernels and accuracies are those of the repository's configurations
(hmat-oss_b200/workloads.py) and tests: points of a regular grid on a cylinder with the
regularised Laplace or Helmholtz kernel, uniform points of the unit cube with the exponential
covariance and a nugget; leaves of 32 to 128 points, epsilon 1e-3 to 1e-6, ACA+ (or partial ACA),
1 to 32 right-hand sides.  A case's points are fixed; the seed draws the vectors and, for an
assembly, the kernel's parameter.
`svd_below` is the library's compressionMinLeafSize (admissible blocks below it are compressed by
dense SVD): 100 is the library's default, the configurations set 0.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_TYPES = {"S": (0, torch.float32), "D": (1, torch.float64), "C": (2, torch.complex64), "Z": (3, torch.complex128)}


def _engine():
    if "hmat_oss_b200" in sys.modules:
        return sys.modules["hmat_oss_b200"]
    folder = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hmat-oss_b200")
    spec = importlib.util.spec_from_file_location("hmat_oss_b200", os.path.join(folder, "__init__.py"),
                                                  submodule_search_locations=[folder])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["hmat_oss_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


def _case(name, op, geo, n, vt, nrhs, trans="N", leaf=64, eta=2.0, eps=1e-4, svd_below=0, partial=False, batch=0):
    c = dict(op=op, geo=geo, n=n, vt=vt, nrhs=nrhs, trans=trans, leaf=leaf, eta=eta, eps=eps, svd_below=svd_below,
             partial=partial, batch=batch)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a small kriging system multiplied from host memory, one vector
        _case("host_cube2k_D_1", "host", "cube", 2000, "D", 1),
        # the product of an iterative solver's step on the plain FP64 cylinder of 8,000 points
        _case("gemv_cyl8k_D_1", "product", "cylinder", 8000, "D", 1),
        # the headline: 100,000-point cylinder, block of 16 vectors (a block solver, many sources)
        _case("gemv_cyl100k_S_16", "product", "cylinder", 100000, "S", 16, eps=1e-6),
        # the same in FP64, with a block width that fills no tile
        _case("gemv_cyl60k_D_11", "product", "cylinder", 60000, "D", 11, eps=1e-6),
        # the transposed product (least squares, two-sided Krylov methods), an odd point count
        _case("gemvT_cyl50k_S_16", "product", "cylinder", 50001, "S", 16, trans="T", eps=1e-6),
        # scattering: complex Helmholtz, leaves of 128, four sources
        _case("gemv_helm50k_C_4", "product", "helmholtz", 50000, "C", 4, leaf=128, eta=3.0),
        # a batch of covariance matrices of uneven sizes, one vector each
        _case("gemv_batch12_S_1", "product", "cube", 60000, "S", 1, eps=1e-5, batch=12),
        # backward of a loss on H x: gradients of x and of every leaf factor
        _case("adjoint_cube20k_S_1", "adjoint", "cube", 20000, "S", 1, eps=1e-6),
        # assembly, small, FP64, with the library's default parameters
        _case("assemble_cyl8k_D", "assemble", "cylinder", 8000, "D", 1, svd_below=100),
        # assembly of the headline matrix
        _case("assemble_cyl100k_S", "assemble", "cylinder", 100000, "S", 16, eps=1e-6),
        # assembly of a complex matrix of long, high-rank blocks
        _case("assemble_helm30k_C", "assemble", "helmholtz", 30000, "C", 4, leaf=128, eta=3.0),
        # assembly of a covariance matrix in FP64, as maximum-likelihood fits repeat it
        _case("assemble_cube20k_D", "assemble", "cube", 20000, "D", 1, eps=1e-5),
    ]


def draw(rng):
    op = rng.choice(["host", "product", "product", "product", "adjoint", "assemble", "assemble"])
    geo = rng.choice(["cylinder", "cylinder", "cube", "helmholtz"] if op != "adjoint" else ["cylinder", "cube"])
    # the largest of each are below the listed ones' cost
    most = {"cylinder": 80000, "cube": 20000, "helmholtz": 25000}[geo]
    svd_below = rng.choice([0, 0, 100])
    if op == "host":
        most //= 4
    elif op == "assemble" and geo == "helmholtz":
        most = 12000
    elif op == "assemble" and svd_below:
        most = 10000
    n = int(round(math.exp(rng.uniform(math.log(1200), math.log(most)))))
    vt = rng.choice("CZ" if geo == "helmholtz" else "SSD")
    # block widths of 1 to 16 and, for a product, some past one tile of 16
    nrhs = rng.choice([1, 1, 2, 3, 4, 5, 7, 8, 11, 13, 16] + ([19, 32] if op == "product" else []))
    trans = rng.choice("NNT" if geo != "helmholtz" else "NTC") if op in ("product", "host") else "N"
    batch = rng.choice([0, 0, 3, 6]) if op == "product" and geo == "cube" and n > 8000 else 0
    return _case(None, op, geo, n, vt, nrhs, trans=trans,
                 leaf=rng.choice([32, 50, 64, 64, 100, 128]), eta=rng.choice([2.0, 3.0]) if geo != "cube" else 2.0,
                 eps=10.0 ** -rng.choice([3, 4, 4, 5, 6 if geo == "cylinder" else 5]),
                 svd_below=svd_below, partial=rng.random() < 0.15, batch=batch)


def _points(case):
    """Points of every member of the case, as a program holds them: host arrays."""
    rng = np.random.default_rng(0)
    n = case["n"]
    if case["geo"] == "cube":
        if not case["batch"]:
            return [rng.random((n, 3))]
        # uneven members, sizes log-uniform over a factor of eight, n points in all
        w = np.exp(rng.uniform(0.0, math.log(8.0), case["batch"]))
        sizes = np.maximum(200, np.round(n * w / w.sum()).astype(int))
        return [rng.random((int(s), 3)) for s in sizes]
    # a grid of n_theta x n_z with n_z / n_theta = 1.6 (height 4, radius 1); the last row may
    # be short
    nt = max(8, int(round(math.sqrt(n / 1.6))))
    nz = -(-n // nt)
    i = np.arange(n)
    th = 2.0 * math.pi * (i % nt) / nt
    return [np.stack([np.cos(th), np.sin(th), 4.0 * (i // nt) / max(nz - 1, 1)], axis=1)]


def _parameters(case, seed):
    """The kernel's parameter for every member: the correlation length, the regularisation, or the
    wavenumber of ten points per wavelength (hmat-oss_b200/workloads.py)."""
    if case["geo"] == "cube":
        ps = [0.3] if not case["batch"] else [float(v) for v in
                                              np.random.default_rng(2).uniform(0.1, 0.5, case["batch"])]
    elif case["geo"] == "cylinder":
        ps = [0.01]
    else:
        ps = [2.0 * math.pi / (10.0 * 1.75 * math.pi / math.sqrt(case["n"]))]
    if case["op"] == "assemble":
        f = np.random.default_rng(seed).uniform(0.95, 1.05)
        ps = [p * float(f) for p in ps]
    return ps


def _matrix(case, seed, assemble):
    hb = _engine()
    hb.set_parameters(compressionMinLeafSize=case["svd_below"])
    pts = _points(case)
    if case["geo"] == "cube":
        kers = [hb.kernel(hb.EXP_COV, ell=v, nugget=1e-6) for v in _parameters(case, seed)]
    elif case["geo"] == "cylinder":
        kers = [hb.kernel(hb.LAPLACE_REG, delta=v) for v in _parameters(case, seed)]
    else:
        kers = [hb.kernel(hb.HELMHOLTZ_REG, delta=0.01, wavenumber=v) for v in _parameters(case, seed)]
    kw = dict(value_type=_TYPES[case["vt"]][0], leaf_size=case["leaf"], eta=case["eta"], epsilon=case["eps"],
              compression="aca_partial" if case["partial"] else "aca_plus", assemble=assemble)
    return hb.HMatrixBatch(pts, kers, **kw) if case["batch"] else hb.HMatrix(pts[0], kers[0], **kw)


def _vectors(case, seed, n, count):
    """`count` blocks of nrhs vectors ~ N(0, 1) (or CN(0, 1)): row q is vector q, contiguous, as
    the library's column-major buffers are."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = _TYPES[case["vt"]][1]
    wide = torch.complex128 if dt.is_complex else torch.float64
    return [torch.randn((case["nrhs"], n), generator=g, dtype=wide, device="cuda").to(dt) for _ in range(count)]


def prepare(case, seed):
    h = _matrix(case, seed, case["op"] != "assemble")
    state = {"case": case, "h": h, "stream": torch.cuda.Stream()}
    if case["op"] == "host":
        state["x"] = np.asfortranarray(_vectors(case, seed, h.n, 1)[0].cpu().numpy().T)
    elif case["op"] == "adjoint":
        state["x"], state["r"] = _vectors(case, seed, h.n, 2)
        state["dx"] = torch.zeros_like(state["x"])
        state["grad"] = torch.zeros(h.payload_layout()[1], dtype=state["x"].dtype, device="cuda")
    else:
        state["x"] = _vectors(case, seed, h.n, 1)[0]
        state["y"] = torch.zeros_like(state["x"])
    torch.cuda.synchronize()
    return state


def run(state):
    case, h, stream = state["case"], state["h"], state["stream"].cuda_stream
    if case["op"] == "host":
        return h.gemv(state["x"], trans=case["trans"])
    if case["op"] == "adjoint":
        h.gemv_adjoint(state["x"].data_ptr(), state["r"].data_ptr(), case["nrhs"], state["dx"].data_ptr(),
                       state["grad"].data_ptr(), stream=stream)
        return {"dx": state["dx"], "grad": state["grad"]}
    if case["op"] == "assemble":
        _engine().set_parameters(compressionMinLeafSize=case["svd_below"])
        h.assemble()
    h.gemv_device(state["x"].data_ptr(), state["y"].data_ptr(), case["nrhs"], trans=case["trans"], stream=stream)
    if case["op"] == "assemble":
        return {"leaves": h.leaf_table(), "y": state["y"]}
    return state["y"]


def work(case):
    """Products: every stored leaf scalar read once, x read and y written once.  The adjoint
    writes a gradient for every stored scalar too.  Assembly writes the stored scalars; its
    operations are the kernel entries that ACA and the full leaves need (about 20 each), the
    rank-k updates of ACA and the QR factorisations of the truncation."""
    h = _matrix(case, 0, True)
    t = h.leaf_table().astype(np.int64)
    s = np.dtype(h.dtype).itemsize
    full = t[t[:, 4] == 0]
    rk = t[(t[:, 4] == 1) & (t[:, 5] > 0)]
    k, mn = rk[:, 5], rk[:, 1] + rk[:, 3]
    entries = int((full[:, 1] * full[:, 3]).sum())
    stored = entries + int((k * mn).sum())
    vec = 2 * h.n * case["nrhs"] * s
    mul = 8 if case["vt"] in "CZ" else 2
    h.close()
    if case["op"] == "assemble":
        flops = 20 * (entries + int((k * mn).sum())) + mul * 3 * int((k * k * mn).sum())
        return {"bytes": 2 * stored * s + vec + 24 * h.n, "flops": flops + mul * stored * case["nrhs"]}
    if case["op"] == "adjoint":
        return {"bytes": 2 * stored * s + 2 * vec, "flops": 2 * mul * stored * case["nrhs"]}
    return {"bytes": stored * s + vec, "flops": mul * stored * case["nrhs"]}


def _dense_product(case, seed, x, trans):
    """op(K) x in 64 bits with the dense kernel matrix, blocks of rows at a time."""
    wide = torch.complex128 if case["vt"] in "CZ" else torch.float64
    x = x.to(wide)
    outs, at = [], 0
    for p, param in zip(_points(case), _parameters(case, seed)):
        p = torch.from_numpy(np.ascontiguousarray(p)).cuda()
        n = p.shape[0]
        xb = x[:, at:at + n].T.contiguous()
        at += n
        rows = max(1, min(n, (1 << 27) // n))
        out = torch.empty((n, x.shape[0]), dtype=wide, device="cuda")
        for i0 in range(0, n, rows):
            q = p[i0:i0 + rows]
            r = torch.zeros((q.shape[0], n), dtype=torch.float64, device="cuda")
            for d in range(3):
                r += (q[:, d, None] - p[None, :, d]).square_()
            r.sqrt_()
            if case["geo"] == "cube":
                k = torch.exp_(r / -param)
                ar = torch.arange(q.shape[0], device="cuda")
                k[ar, i0 + ar] += 1e-6
            elif case["geo"] == "cylinder":
                k = 1.0 / (4.0 * math.pi * (r + param))
            else:
                k = torch.polar(1.0 / (4.0 * math.pi * (r + 0.01)), r * param)
            # the kernels are symmetric: K^T = K, and K^H = conj(K)
            out[i0:i0 + rows] = (k.conj() if trans == "C" else k) @ xb
        outs.append(out)
    return torch.cat(outs, dim=0).T.contiguous()


def exact(case, seed):
    n = sum(len(p) for p in _points(case))
    if case["op"] == "adjoint":
        # the gradients belong to the stored factors, which the dense matrix does not have
        _, r = _vectors(case, seed, n, 2)
        return {"dx": _dense_product(case, seed, r, "T"), "grad": None}
    y = _dense_product(case, seed, _vectors(case, seed, n, 1)[0], case["trans"])
    if case["op"] == "host":
        return np.asfortranarray(y.cpu().numpy().T)
    return {"leaves": None, "y": y} if case["op"] == "assemble" else y
