"""The contraction with one MPO tensor (second half of prod_AOR and prod_AOL) at the edges of its
32-wide columns, its 2 / 4 / 8 outputs per thread and its groups of outputs."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import crand, empty_dev, from_dev, to_dev
from oracle import mps_ref as R

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("X,Y,d,wL,wR", [
    (1, 1, 1, 1, 1), (31, 3, 2, 1, 5), (32, 2, 3, 7, 1), (33, 40, 2, 5, 3), (65, 64, 4, 2, 2), (300, 70, 2, 9, 9),
    (96, 500, 4, 4, 4), (40, 9, 2, 33, 33), (33, 300, 2, 33, 33),
])
@pytest.mark.parametrize("right", [True, False])
def test_mpo_tile_edges(gpu_ctx, X, Y, d, wL, wR, right):
    import torch
    from mpsb200 import _lib
    chi = 6
    rng = np.random.default_rng(X + 1000 * Y + wL + 10 * wR + right)
    O = crand(rng, wL, d, wR, d)
    if right:   # x = chiL, y = chiR0
        A, E = crand(rng, X, d, chi), crand(rng, chi, wR, Y)
        prod, name, args = R.prod_AOR, "mpsb_op_prod_AOR", (X, d, chi, wL, wR, Y)
    else:       # x = chiL0, y = chiR
        A, E = crand(rng, chi, d, Y), crand(rng, chi, wL, X)
        prod, name, args = R.prod_AOL, "mpsb_op_prod_AOL", (chi, d, Y, wL, wR, X)
    ref = prod(A, O, E)
    dA, dO, dE, dout = to_dev(A), to_dev(O), to_dev(E), empty_dev(ref.shape)
    torch.cuda.synchronize()
    _lib.call(name, gpu_ctx.h, *(C.c_void_p(t.data_ptr()) for t in (dA, dO, dE, dout)), *args)
    gpu_ctx.sync()
    # sums of chi and of d w complex products (4 roundings a term), on both sides
    K = d * (wR if right else wL)
    bound = 2 * 4 * (chi + K + 4) * EPS * prod(abs(A), abs(O), abs(E)).real
    assert np.all(np.abs(from_dev(dout, ref.shape) - ref) <= bound)
