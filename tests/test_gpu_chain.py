"""Scalar products with a product state run as one launch over the chain: against the oracle for
either side being the product, ragged bonds, long and short chains, and a bond beyond the
kernel's range (the general path)."""
import numpy as np
import pytest

from gpu_util import crand
from oracle import mps_ref as R

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("na,d,chi", [(1, 2, 1), (2, 3, 3), (7, 2, 5), (12, 4, 97), (9, 4, 512), (13, 5, 400), (40, 2, 17), (256, 2, 4),
                                      (257, 2, 3), (5, 4, 600)])
def test_product_scalar_products_match_oracle(gpu_ctx, na, d, chi):
    from mpsb200 import core as K
    rng = np.random.default_rng(na * 1000 + chi)
    dims = [1] + [chi if na < 9 else min(chi, 2 * d ** min(k, 9), 2 * d ** min(na - k, 9)) for k in range(1, na)] + [1]
    B = [crand(rng, dims[k], d, dims[k + 1]) / np.sqrt(d * dims[k]) for k in range(na)]
    f = [crand(rng, 1, d, 1) for _ in range(na)]
    mB, mf = K.MPS.from_sites(B, gpu_ctx), K.MPS.from_sites(f, gpu_ctx)
    # the chain of absolute values bounds the rounding of any order of summation
    size = R.scal_prod_no_conj([abs(x).astype(complex) for x in f], [abs(x).astype(complex) for x in B]).real
    tol = 8 * EPS * size * sum(dims[k] * d for k in range(na))
    for a, b, ma, mb in ((f, B, mf, mB), (B, f, mB, mf)):
        assert abs(K.scal_prod_no_conj(ma, mb) - R.scal_prod_no_conj(a, b)) <= tol
        assert abs(K.scal_prod(ma, mb) - R.scal_prod(a, b)) <= tol
