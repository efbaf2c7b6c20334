"""The scratch of device products: taken with the assembly for both directions, not by the first
product of each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vt", [0, 1])
def test_first_products_take_no_device_memory(hb, vt):
    import torch
    pts = np.random.default_rng(3).random((20000, 3))
    hb.set_parameters(compressionMinLeafSize=0)
    k = hb.kernel(hb.EXP_COV, ell=0.3, nugget=1e-6)
    kw = dict(value_type=vt, leaf_size=64, eta=2.0, epsilon=1e-4)
    dt = torch.float64 if vt == 1 else torch.float32
    x = torch.from_numpy(np.random.default_rng(4).standard_normal((16, len(pts)))).to("cuda", dt)
    y = torch.zeros_like(x)
    h, other = hb.HMatrix(pts, k, **kw), hb.HMatrix(pts, k, **kw)
    try:
        for t in "NT":  # another matrix: the kernels of both directions are loaded
            other.gemv_device(x.data_ptr(), y.data_ptr(), 16, trans=t)
        torch.cuda.synchronize()
        for t in "NT":
            before = torch.cuda.mem_get_info()[0]
            h.gemv_device(x.data_ptr(), y.data_ptr(), 16, trans=t)
            torch.cuda.synchronize()
            # the rows of x alone, 16 right-hand sides: 1.3 MB in FP32; a graph may take a page
            assert before - torch.cuda.mem_get_info()[0] <= 2 << 20, t
    finally:
        h.close()
        other.close()
