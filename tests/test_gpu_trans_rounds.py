"""Transposed products whose column pass runs in rounds: matrices of small leaves, nearly all of them
full, whose partial rows would not fit the scratch at once.  Regular and allocation-free products
(the latter take such matrices by their bound of 16 MiB) and the adjoint, against the kernel matrix."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# value type, points, leaf, eta (1e-9: every leaf full; 0.02: points in two clouds far apart, full leaves
# inside them and one Rk leaf over all blocks of a cloud each way), whether the allocation-free products take it
CASES = [(0, 8192, 32, 1e-9, True), (1, 3000, 12, 1e-9, True), (2, 3000, 12, 1e-9, True), (3, 3000, 12, 1e-9, False),
         (0, 4096, 8, 0.02, True), (1, 4096, 8, 0.02, True), (2, 4096, 8, 0.02, True), (3, 3000, 8, 0.02, False)]


def _problem(hb, vt, n, leaf, eta):
    pts = np.random.default_rng(n + leaf).random((n, 3))
    if eta > 1e-3:
        pts[n // 2:, 0] += 100.0
    k = (hb.kernel(hb.HELMHOLTZ_REG, delta=0.05, wavenumber=6.0) if vt >= 2 else
         hb.kernel(hb.LAPLACE_REG, delta=0.05))
    hb.set_parameters(compressionMinLeafSize=0)
    h = hb.HMatrix(pts, k, value_type=vt, leaf_size=leaf, eta=eta, epsilon=1e-6)
    r = np.sqrt(((pts[:, None] - pts[None]) ** 2).sum(-1))
    K = (np.exp(6j * r) if vt >= 2 else 1.0) / (4.0 * np.pi * (r + 0.05))
    return h, K


def _close(got, op, x, vt, full):
    want = op @ x
    if full:  # the bound of test_gpu_transposed.py
        u = 2.0 ** -24 if vt in (0, 2) else 2.0 ** -53
        assert np.all(np.abs(got - want) <= 16.0 * u * np.sqrt(len(x)) * (np.abs(op) @ np.abs(x)) + 1e-300)
    else:  # the far blocks, below a tenth of the near ones, compressed at 1e-6; in FP32 as many roundings as above
        assert np.linalg.norm(got - want) <= (1e-6 if vt in (1, 3) else 1e-4) * np.linalg.norm(want)


@pytest.mark.parametrize("vt,n,leaf,eta,noalloc", CASES)
def test_products(hb, vt, n, leaf, eta, noalloc):
    import torch
    h, K = _problem(hb, vt, n, leaf, eta)
    dt = {0: torch.float32, 1: torch.float64, 2: torch.complex64, 3: torch.complex128}[vt]
    try:
        T = h.leaf_table()
        assert np.sum(T[:, 4] == 1) == (2 if eta > 1e-3 else 0) and np.all(T[T[:, 4] == 1, 5] > 0)
        # gather, a column pass and its sums a round, at most two group passes, the final sum
        assert h.gemv_launches(1, trans="T") >= 1 + 2 * 2 + 1
        rng = np.random.default_rng(1)
        for trans in ("N", "T", "C"):
            op = {"N": K, "T": K.T, "C": K.conj().T}[trans]
            for nrhs in (1, 3, 7, 11, 19):
                x = rng.standard_normal((n, nrhs)) + (1j * rng.standard_normal((n, nrhs)) if vt >= 2 else 0.0)
                xd = torch.from_numpy(np.ascontiguousarray(x.T)).to("cuda", dt)
                yd = torch.full_like(xd, float("nan"))
                h.gemv_device(xd.data_ptr(), yd.data_ptr(), nrhs, trans=trans)
                torch.cuda.synchronize()
                wide = xd.cpu().numpy().T.astype(K.dtype)
                _close(yd.cpu().numpy().T, op, wide, vt, eta < 1e-3)
                if not noalloc:
                    continue
                for _ in range(2):  # the array keeps the last call's rows
                    zd = torch.full_like(xd, float("nan"))
                    rc = h.gemv_device_noalloc(xd.data_ptr(), zd.data_ptr(), nrhs, trans=trans)
                    assert rc == 0, hb.load_library().hmat_b200_last_error()
                    torch.cuda.synchronize()
                    assert torch.equal(zd, yd), (trans, nrhs)
        # <H x, r> = <x, H^T r> to rounding, whatever the compression
        x, r = (rng.standard_normal((n, 5)).astype(h.dtype) for _ in range(2))
        a, b = h.gemv(x), h.gemv(r, trans="T")
        lhs, rhs = (a * r).sum(0), (x * b).sum(0)
        u = 2.0 ** -24 if vt in (0, 2) else 2.0 ** -53
        assert np.all(np.abs(lhs - rhs) <= 16.0 * u * np.sqrt(n) * (np.abs(r) * (np.abs(K) @ np.abs(x))).sum(0))
    finally:
        h.close()


@pytest.mark.parametrize("vt,n,leaf,eta,nrhs", [(0, 8192, 32, 1e-9, 5), (1, 4096, 8, 0.02, 1), (0, 4096, 8, 0.02, 16)])
def test_adjoint(hb, vt, n, leaf, eta, nrhs):
    import torch
    h, K = _problem(hb, vt, n, leaf, eta)
    try:
        rng = np.random.default_rng(2)
        x, r = (rng.standard_normal((n, nrhs)).astype(h.dtype) for _ in range(2))
        xd, rd = (torch.from_numpy(np.ascontiguousarray(v.T)).cuda() for v in (x, r))
        offs, total = h.payload_layout()
        dx = torch.full_like(xd, float("nan"))
        grad = torch.full((total,), float("nan"), dtype=xd.dtype, device="cuda")
        h.gemv_adjoint(xd.data_ptr(), rd.data_ptr(), nrhs, dx.data_ptr(), grad.data_ptr())
        torch.cuda.synchronize()
        _close(dx.cpu().numpy().T, K.T, r.astype(np.float64), vt, eta < 1e-3)
        g = grad.cpu().numpy()
        assert np.all(np.isfinite(g))
        T, pr, pc = h.leaf_table(), h.perm(), h.perm(cols=True)
        u = 2.0 ** -24 if vt == 0 else 2.0 ** -53
        rk = np.flatnonzero((T[:, 4] == 1) & (T[:, 5] > 0))
        tall = rk[np.argsort(-T[rk, 1])]
        full = np.flatnonzero(T[:, 4] == 0)
        for i in np.concatenate([full[:: max(1, len(full) // 20)], tall[:20], rk[:: max(1, len(rk) // 20)]]):
            r0, m, c0, nn, t, k = T[i]
            ri, xj = r[pr[r0:r0 + m]].astype(np.float64), x[pc[c0:c0 + nn]].astype(np.float64)
            if t == 0:
                parts = [(ri, xj, 0.0)]
            else:
                p = h.leaf_payload(i).astype(np.float64)
                A, B = p[:k * m].reshape(k, m).T, p[k * m:].reshape(k, nn).T
                parts = [(ri, B.T @ xj, np.abs(B).T @ np.abs(xj)), (xj, A.T @ ri, np.abs(A).T @ np.abs(ri))]
            at = offs[i]
            for a, b, mag in parts:
                got = g[at:at + a.shape[0] * b.shape[0]].reshape(b.shape[0], a.shape[0]).T
                at += got.size
                bound = 16.0 * u * np.sqrt(n) * (np.abs(a) @ np.maximum(np.abs(b), mag).T)
                assert np.all(np.abs(got - a @ b.T) <= bound + 1e-300), i
    finally:
        h.close()


def test_large_matrix(hb):
    """Beyond the allocation-free products' bound: 3 GB of leaves, many of them Rk leaves over several
    blocks, in rounds of at most half the leaves' bytes.  <H x, r> = <x, H^T r>: each side's error is below
    n u ||K|| ||x|| ||r||, and the norm below n (entries of at most 1, nugget aside)."""
    import torch
    n = 60000
    pts = np.random.default_rng(1).random((n, 3))
    hb.set_parameters(compressionMinLeafSize=0)
    torch.manual_seed(0)
    h = hb.HMatrix(pts, hb.kernel(hb.EXP_COV, ell=0.3, nugget=1e-6), leaf_size=12, eta=1.5, epsilon=1e-5)
    try:
        T = h.leaf_table()
        assert np.sum((T[:, 4] == 1) & (T[:, 1] > 12)) > 1000
        assert h.gemv_launches(1, trans="T") >= 1 + 3 * 2 + 1
        for nrhs in (1, 5, 16):
            x, r = (torch.randn((nrhs, n), dtype=torch.float64, device="cuda") for _ in range(2))
            y, z = torch.zeros_like(x), torch.zeros_like(x)
            torch.cuda.synchronize()
            h.gemv_device(x.data_ptr(), y.data_ptr(), nrhs)
            h.gemv_device(r.data_ptr(), z.data_ptr(), nrhs, trans="T")
            torch.cuda.synchronize()
            lhs, rhs = (y * r).sum(1), (x * z).sum(1)
            assert torch.all((lhs - rhs).abs() <= 2.0 * n * n * 2.0 ** -53 * x.norm(dim=1) * r.norm(dim=1))
            assert torch.all(lhs.abs() > 1e4 * (lhs - rhs).abs())
    finally:
        h.close()
