"""Weight gradients on the tensor cores (k_dweight_tc) against the CUDA-core kernel's: one tile row a block and
many, ranges that end inside a strip, image and strip borders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nimg,crop", [(1, 64), (2, 64), (3, 128), (5, 192), (8, 256)])
def test_tensor_core_weight_gradients(gpu, nimg, crop):
    from simuverse_gb300.closure import Closure

    rng = np.random.default_rng(nimg)
    c = Closure(crop, crop, seed=3, inputs="eq", target="stress", projection="cell")
    c.reserve(nimg, crop, nimg)
    feats = rng.standard_normal((nimg, crop, crop, 9))
    targets = 0.3 * rng.standard_normal((nimg, crop, crop, 9))
    g = {}
    for kernel in ("layers", "fused"):
        c.set_kernel(kernel)
        _, g[kernel] = c.loss_grad(feats, targets)
        c.status()
    off, prev = 0, 0.0
    for n in (9 * 9 * 32, 32, 9 * 32 * 32, 32, 9 * 32 * 9, 9):
        a, b = (g[k][off:off + n].astype(np.float64) for k in ("layers", "fused"))
        off += n
        # both sum FP32 products of the same BF16 values in FP32, in another order: 2^-24 times the
        # roots of some 10^5 terms of either sign.  (The stress loss does not depend on the last bias.)
        scale = max(np.linalg.norm(a), prev if n in (32, 9) else 0.0)
        assert np.linalg.norm(a - b) <= 2e-5 * scale, n
        prev = np.linalg.norm(a)
    c.close()
