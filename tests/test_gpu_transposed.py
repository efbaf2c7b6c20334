"""Products ('N', 'T', 'C') against the stored leaves multiplied out in FP64:
block heights at the edges of the kernels' tiles (one row, odd, 64, 128, leaves cut into several
blocks), row and column trees of different leaf sizes, ranks above the first height class, every
right-hand-side tile and more than one, every type."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # value type, points, row leaf, column leaf, eta, epsilon
    (1, 1, 1, None, 2.0, 1e-6), (1, 40, 1, None, 2.0, 1e-6), (0, 300, 7, None, 2.0, 1e-6),
    (1, 700, 33, None, 2.0, 1e-8), (0, 1500, 64, None, 2.0, 1e-6), (1, 1500, 128, None, 2.0, 1e-4),
    (0, 1500, 190, None, 2.0, 1e-4), (1, 1500, 20, 90, 2.0, 1e-6), (0, 1500, 90, 20, 2.0, 1e-6),
    (1, 3000, 50, None, 6.0, 1e-8), (0, 3000, 100, None, 6.0, 1e-6),
    (2, 1200, 48, None, 2.0, 1e-5), (3, 1200, 48, None, 2.0, 1e-8), (3, 1500, 128, None, 6.0, 1e-6),
    (2, 1500, 60, 17, 4.0, 1e-5),
]


@pytest.mark.parametrize("vt,n,leaf,leaf_cols,eta,eps", CASES)
def test_transposed_products(hb, vt, n, leaf, leaf_cols, eta, eps):
    pts = np.random.default_rng(n + leaf).random((n, 3))
    k = (hb.kernel(hb.HELMHOLTZ_REG, delta=0.05, wavenumber=6.0) if vt >= 2 else
         hb.kernel(hb.EXP_COV, ell=0.3, nugget=1e-6))
    hb.set_parameters(compressionMinLeafSize=0)
    h = hb.HMatrix(pts, k, value_type=vt, leaf_size=leaf, leaf_size_cols=leaf_cols, eta=eta, epsilon=eps)
    try:
        T = h.leaf_table()
        H = np.zeros((n, n), np.complex128 if vt >= 2 else np.float64)
        offs, total = h.payload_layout()
        pr, pc = h.perm(), h.perm(cols=True)
        for i, (r0, m, c0, nn, _, _) in enumerate(T):
            H[np.ix_(pr[r0:r0 + m], pc[c0:c0 + nn])] = h.leaf_block(i)
        rng = np.random.default_rng(1)
        for trans in "NTC" if vt >= 2 else "NT":
            op = {"N": H, "T": H.T, "C": H.conj().T}[trans]
            for nrhs in (1, 2, 4, 5, 8, 11, 16, 21):
                x = rng.standard_normal((n, nrhs)) + (1j * rng.standard_normal((n, nrhs)) if vt >= 2 else 0.0)
                x = x.astype(h.dtype)
                y0 = rng.standard_normal((n, nrhs)).astype(h.dtype)
                want = 0.5 * (op @ x.astype(H.dtype)) + 2.0 * y0
                got = h.gemv(x, trans=trans, alpha=0.5, beta=2.0, y=y0)
                # sums of n products: n u |op| |x| bounds each entry; the factors of FP32 blocks
                # are multiplied out in FP32 above (another u)
                u = 2.0 ** -24 if vt in (0, 2) else 2.0 ** -53
                bound = 16.0 * u * (np.abs(op) @ np.abs(x) * np.sqrt(n) + np.abs(y0))
                assert np.all(np.abs(got - want) <= bound + 1e-300), (trans, nrhs, np.max(np.abs(got - want) / bound))
    finally:
        h.close()


@pytest.mark.parametrize("n,leaf,leaf_cols,eta,eps", [
    (1, 1, None, 2.0, 1e-6), (40, 1, None, 2.0, 1e-6), (300, 7, None, 2.0, 1e-6), (900, 32, None, 2.0, 1e-6),
    (900, 33, None, 2.0, 1e-6), (1500, 64, None, 2.0, 1e-6), (1500, 100, None, 2.0, 1e-4),
    (1500, 128, None, 2.0, 1e-4), (1500, 190, None, 2.0, 1e-4), (1500, 90, 20, 2.0, 1e-6),
    (3000, 50, None, 6.0, 1e-6)])
def test_single_fp32_product(hb, n, leaf, leaf_cols, eta, eps):
    """'N' with one FP32 right-hand side, on its own kernels, against the stored leaves in FP64."""
    pts = np.random.default_rng(n + leaf).random((n, 3))
    hb.set_parameters(compressionMinLeafSize=0)
    h = hb.HMatrix(pts, hb.kernel(hb.EXP_COV, ell=0.3, nugget=1e-6), value_type=0, leaf_size=leaf,
                   leaf_size_cols=leaf_cols, eta=eta, epsilon=eps)
    try:
        H = np.zeros((n, n))
        pr, pc = h.perm(), h.perm(cols=True)
        for i, (r0, m, c0, nn, _, _) in enumerate(h.leaf_table()):
            H[np.ix_(pr[r0:r0 + m], pc[c0:c0 + nn])] = h.leaf_block(i)
        rng = np.random.default_rng(1)
        for nrhs in (1, 17):  # 17: a tile of 16 and one of 1
            x, y0 = (rng.standard_normal((n, nrhs)).astype(np.float32) for _ in range(2))
            want = 0.5 * (H @ x.astype(np.float64)) + 2.0 * y0
            got = h.gemv(x, alpha=0.5, beta=2.0, y=y0)
            # the bound of test_transposed_products
            bound = 16.0 * 2.0 ** -24 * (np.abs(H) @ np.abs(x) * np.sqrt(n) + np.abs(y0))
            assert np.all(np.abs(got - want) <= bound + 1e-300), nrhs
    finally:
        h.close()
