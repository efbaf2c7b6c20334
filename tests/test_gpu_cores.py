"""Cores of high-rank leaves: a kernel variant by the leaf's own rank (shared memory up to 32, 64 and
96 columns, the slab above; complex cores to 82), every variant in one assembly, and factors that do
not depend on which leaves share a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _assemble(hb, vt, eps, n):
    pts = np.random.default_rng(5).random((n, 3))
    k = hb.kernel(hb.HELMHOLTZ_REG, delta=0.01, wavenumber=15.0) if vt >= 2 else hb.kernel(hb.EXP_COV, ell=0.3,
                                                                                         nugget=1e-6)
    hb.set_parameters(compressionMinLeafSize=0)
    return hb.HMatrix(pts, k, value_type=vt, leaf_size=140 if vt == 1 else 110, eta=4.0, epsilon=eps)


@pytest.mark.parametrize("vt,eps,classes", [(1, 1e-9, [(33, 64), (65, 96), (97, 128)]),
                                            (3, 1.8e-7, [(33, 64), (65, 82), (83, 128)])])
def test_factors_do_not_depend_on_the_batch(hb, monkeypatch, vt, eps, classes):
    """The stored factors truncated again, all in one batch and in batches of at most 64 MB (the
    smallest workspace): cores of every class, the same bytes."""
    h = _assemble(hb, vt, eps, 4000 if vt == 1 else 3500)
    try:
        T = h.leaf_table()
        struct, data = h.dump()
    finally:
        h.close()
    rk = T[(T[:, 4] == 1) & (T[:, 5] > 0)]
    for lo, hi in classes:
        assert np.any((rk[:, 5] >= lo) & (rk[:, 5] <= hi)), (lo, hi)
    if vt == 3:  # the second batch of 64 MB has no core of the slab's class (a real core has the
        # same bytes on every variant)
        at = np.cumsum((rk[:, 1] + rk[:, 3]) * rk[:, 5] * 16)
        assert np.any(at > 66 << 20) and not np.any(rk[at > 63.8 * 2 ** 20, 5] > 82)
    out = []
    for mb in ("8192", "64"):
        monkeypatch.setenv("HMAT_B200_WORKSPACE_MB", mb)
        g = hb.HMatrix.load(vt, struct, data)
        try:
            g.truncate(2.0 * eps)
            out.append((g.leaf_table(), g.dump()[1]))
        finally:
            g.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
