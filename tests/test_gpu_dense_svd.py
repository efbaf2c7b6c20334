"""Small admissible blocks compressed by SVD of the dense block (compressionMinLeafSize): ranks and
blocks against numpy's truncated SVD of the kernel matrix, over block sizes at the edges of the
shared-memory kernel (one point, odd sizes, 128 columns, larger blocks on the slab kernel), tall
and wide blocks, real and complex types."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # value type, points, row leaf, column leaf, min leaf
    (1, 300, 1, None, 100), (1, 400, 7, None, 100), (1, 900, 33, None, 100), (1, 1500, 64, None, 100),
    (1, 3000, 99, None, 100), (1, 3000, 128, None, 200), (1, 3000, 190, None, 400),
    (1, 3000, 120, 10, 400), (1, 3000, 9, 60, 400),
    (3, 700, 33, None, 100), (3, 2000, 99, None, 100), (3, 2000, 130, None, 300), (3, 2000, 80, 8, 300),
    (0, 1500, 64, None, 100), (2, 1500, 64, None, 100),
]


def kernel_matrix(vt, p, q, rows, cols):
    r = np.sqrt(((p[:, None, :] - q[None, :, :]) ** 2).sum(-1))
    if vt >= 2:
        return np.exp(1j * 5.0 * r) / (4.0 * np.pi * (r + 0.01))
    return np.exp(-r / 0.3) + 1e-6 * (rows[:, None] == cols[None, :])


@pytest.mark.parametrize("vt,n,leaf,leaf_cols,min_leaf", CASES)
def test_dense_svd_blocks(hb, vt, n, leaf, leaf_cols, min_leaf):
    pts = np.random.default_rng(n + leaf).random((n, 3))
    eps = 1e-4
    k = hb.kernel(hb.HELMHOLTZ_REG, delta=0.01, wavenumber=5.0) if vt >= 2 else hb.kernel(hb.EXP_COV, ell=0.3,
                                                                                        nugget=1e-6)
    hb.set_parameters(compressionMinLeafSize=min_leaf)
    try:
        h = hb.HMatrix(pts, k, value_type=vt, leaf_size=leaf, leaf_size_cols=leaf_cols, eta=2.0, epsilon=eps)
    finally:
        hb.set_parameters(compressionMinLeafSize=0)
    try:
        T = h.leaf_table()
        pr, pc = h.perm(), h.perm(cols=True)
        small = [i for i in range(len(T)) if T[i, 4] == 1 and max(T[i, 1], T[i, 3]) < min_leaf]
        assert small
        # every shape, and a spread of the rest
        shapes = {}
        for i in small:
            shapes.setdefault((T[i, 1], T[i, 3]), i)
        for i in sorted(set(list(shapes.values())[:20] + small[:: max(1, len(small) // 40)])):
            r0, m, c0, nn, _, rank = T[i]
            rows, cols = pr[r0:r0 + m], pc[c0:c0 + nn]
            M = kernel_matrix(vt, pts[rows], pts[cols], rows, cols)
            U, s, Vh = np.linalg.svd(M)
            kk = int((s > eps * s[0]).sum())
            best = (U[:, :kk] * s[:kk]) @ Vh[:kk]
            got = h.leaf_block(i)
            if vt in (1, 3):
                # rounding of an SVD in FP64 (a few k u sigma_0); ranks equal unless a singular
                # value sits on the threshold
                near = np.any(np.abs(s / (eps * s[0]) - 1.0) < 1e-9)
                assert near or rank == kk, (m, nn, rank, kk)
                assert near or np.linalg.norm(got - best, 2) <= 1e-12 * s[0]
            else:
                # the FP32 entries move singular values by up to sqrt(m n) 2^-23: the block may be
                # cut one singular value earlier or later
                assert np.linalg.norm(got - M, 2) <= (eps + 1e-5) * s[0]
    finally:
        h.close()


@pytest.mark.parametrize("vt,eps", [(1, 1e-5), (1, 1e-7), (1, 1e-9), (3, 1e-4), (3, 1e-6)])
def test_high_rank_cores(hb, vt, eps):
    """Ranks above the register buckets, whose cores are diagonalised in shared memory (up to 32, 64
    and 96 columns) or on the slab: the factors come out as U sqrt(S), V sqrt(S) with the singular
    values in order, and the block is within the tolerance of the kernel's."""
    pts = np.random.default_rng(5).random((2500, 3))
    k = hb.kernel(hb.HELMHOLTZ_REG, delta=0.01, wavenumber=5.0) if vt >= 2 else hb.kernel(hb.EXP_COV, ell=0.3,
                                                                                        nugget=1e-6)
    hb.set_parameters(compressionMinLeafSize=0)
    h = hb.HMatrix(pts, k, value_type=vt, leaf_size=110, eta=4.0, epsilon=eps)
    try:
        T = h.leaf_table()
        pr = h.perm()
        rk = [i for i in range(len(T)) if T[i, 4] == 1 and T[i, 5] > 0]
        rk.sort(key=lambda i: -T[i, 5])
        assert T[rk[0], 5] > (16 if vt >= 2 else 32)
        for i in rk[:: max(1, len(rk) // 25)]:
            r0, m, c0, nn, _, r = T[i]
            p = h.leaf_payload(i)
            A, B = p[:r * m].reshape(r, m).T, p[r * m:].reshape(r, nn).T
            # U sqrt(S): orthogonal columns of norm sqrt(sigma_j), the same for A and B.  A column
            # is formed as A M with errors of order k u sigma_0 / sqrt(sigma_j), sigma_j > eps sigma_0
            ga, gb = A.conj().T @ A, B.conj().T @ B
            s = np.real(np.diag(ga))
            tol = 64.0 * 2.0 ** -53 / eps * s[0] + 1e-12 * s[0]
            assert np.all(np.diff(s) <= tol) and np.all(s > 0.5 * eps * s[0])
            assert np.abs(ga - np.diag(s)).max() <= tol and np.abs(gb - np.diag(s)).max() <= tol
            rows, cols = pr[r0:r0 + m], pr[c0:c0 + nn]
            M = kernel_matrix(vt, pts[rows], pts[cols], rows, cols)
            # ACA's own stopping estimate and the truncation, each at eps
            assert np.linalg.norm(A @ B.T - M) <= 50.0 * eps * np.linalg.norm(M)
    finally:
        h.close()
