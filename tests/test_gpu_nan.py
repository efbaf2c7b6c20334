"""NaN entries in admissible blocks fail the compression with a message, on every kernel that orders
singular values: the shared-memory SVDs of dense blocks (real, complex), the slab kernel, the cores
of low and of high rank.  The library multiplies correctly afterwards."""
import numpy as np
import pytest
from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vt", [0, 1, 2, 3])
@pytest.mark.parametrize("n,leaf", [(300, 20), (1600, 100), (2240, 140)])
def test_nan_kernel_parameter_fails_the_dense_svd(hb, vt, n, leaf):
    pts = np.random.default_rng(n).random((n, 3))
    nan = float("nan")
    bad = hb.kernel(hb.HELMHOLTZ_REG, delta=0.01, wavenumber=nan) if vt >= 2 else hb.kernel(hb.LAPLACE_REG, delta=nan)
    good = hb.kernel(hb.HELMHOLTZ_REG, delta=0.01, wavenumber=5.0) if vt >= 2 else hb.kernel(hb.LAPLACE_REG, delta=0.01)
    kw = dict(value_type=vt, leaf_size=leaf, eta=4.0, epsilon=1e-4)
    hb.set_parameters(compressionMinLeafSize=100000)  # every admissible block
    try:
        with pytest.raises(hb.HMatError, match="did not converge"):
            hb.HMatrix(pts, bad, **kw)
        h = hb.HMatrix(pts, good, **kw)
    finally:
        hb.set_parameters(compressionMinLeafSize=0)
    try:
        assert np.any(h.leaf_table()[:, 4] == 1)
        x = np.random.default_rng(1).standard_normal((n, 1))
        r = np.sqrt(((pts[:, None] - pts[None]) ** 2).sum(-1))
        K = (np.exp(5j * r) if vt >= 2 else 1.0) / (4.0 * np.pi * (r + 0.01))
        assert rel(h.gemv(x.astype(h.dtype)), K @ x) < 1e-3
    finally:
        h.close()


@pytest.mark.parametrize("vt,eps,least", [(1, 1e-3, 2), (1, 1e-7, 33), (3, 1e-3, 2), (3, 1e-5, 17)])
def test_nan_factor_fails_the_truncation(hb, vt, eps, least):
    """A stored factor column of NaN, read back and truncated again: the core of its leaf."""
    pts = np.random.default_rng(5).random((2500, 3))
    k = hb.kernel(hb.HELMHOLTZ_REG, delta=0.01, wavenumber=5.0) if vt >= 2 else hb.kernel(hb.EXP_COV, ell=0.3,
                                                                                        nugget=1e-6)
    hb.set_parameters(compressionMinLeafSize=0)
    h = hb.HMatrix(pts, k, value_type=vt, leaf_size=110, eta=4.0, epsilon=eps)
    try:
        T = h.leaf_table()
        i = int(np.argmax(np.where(T[:, 4] == 1, T[:, 5], -1)))
        assert T[i, 5] >= least
        p = h.leaf_payload(i)
        struct, data = h.dump()
    finally:
        h.close()
    m, rank = int(T[i, 1]), int(T[i, 5])
    bad = p.copy()
    bad[m * (rank - 1):m * rank] = float("nan")  # A's last column
    a, b = p[:m * rank].tobytes(), bad[:m * rank].tobytes()
    assert data.count(a) == 1
    g = hb.HMatrix.load(vt, struct, data.replace(a, b))
    try:
        with pytest.raises(hb.HMatError, match="did not converge"):
            g.truncate(eps)
    finally:
        g.close()
