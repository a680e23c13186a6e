"""QR at the edges of its kernel's tilings: one, two and many CTAs of a cluster, partial panels,
full and ragged column chunks, row counts on and off the CTA grid, outer panels of the blocked
form -- against LAPACK, and batched against one by one."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import crand, empty_dev, from_dev, to_dev
from oracle import mps_ref as R

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _qr(ctx, X):
    import torch
    from mpsb200 import _lib
    m, n = X.shape
    dX, dQ, dR = to_dev(X), empty_dev((m, n)), empty_dev((n, n))
    torch.cuda.synchronize()
    _lib.call("mpsb_op_qr", ctx.h, *(C.c_void_p(t.data_ptr()) for t in (dX, dQ, dR)), m, n)
    ctx.sync()
    return from_dev(dQ, (m, n)), from_dev(dR, (n, n))


# 31..33: one CTA to two; 64/65: two to three; 15..17, 31..33 columns: partial panels; 512 x 285 and
# 286: the widest matrix of one cluster at 16 CTAs and the narrowest blocked one; 545 x 40: two rows
# per lane; 2048 x 70: four, two outer panels; 1920 x 64: 15 CTAs
@pytest.mark.parametrize("m,n", [(15, 15), (31, 16), (32, 17), (33, 31), (64, 33), (65, 16), (97, 80), (320, 97),
                                 (512, 200), (512, 285), (512, 286), (513, 129), (545, 40), (1030, 65), (1920, 64),
                                 (2048, 70)])
def test_qr_edges_match_lapack(gpu_ctx, m, n):
    rng = np.random.default_rng(100 * m + n)
    X = crand(rng, m, n)
    q, r = R.julia_qr(X)
    Q, Rr = _qr(gpu_ctx, X)
    # two backward-stable factorisations of X differ by O(eps) ||X|| in R and O(eps) cond(X) in Q
    s = np.linalg.svd(X, compute_uv=False)
    tol = 10 * EPS * n * s[0] / s[-1]
    assert np.linalg.norm(Q - q, 2) <= tol
    assert np.linalg.norm(Rr - r, 2) <= tol * s[0]
    assert np.linalg.norm(Q.conj().T @ Q - np.eye(n), 2) <= 10 * EPS * n
    assert np.linalg.norm(Q @ Rr - X, 2) <= 10 * EPS * n * s[0]


@pytest.mark.parametrize("chi", [20, 290])
def test_batched_sweep_qr_equals_one_by_one(gpu_ctx, chi):
    """A sweep pair on a batch of three (its QRs in one launch per site; chi = 290 blocked) computes
    each copy as a batch of one does."""
    from mpsb200 import core as K
    na, d = 20, 2
    dims = K._dims_rule(na, chi, d)
    rng = np.random.default_rng(chi)
    states = [[crand(rng, dims[k], d, dims[k + 1]) / np.sqrt(dims[k] * d) for k in range(na)] for _ in range(3)]
    one = np.eye(d, dtype=np.complex128).reshape(1, d, 1, d)
    H = K.MPO.from_sites([one] * na, gpu_ctx)

    def run(copies):
        A = K.MPS(dims, d, gpu_ctx, batch=len(copies))
        for b, sites in enumerate(copies):
            for k, a in enumerate(sites):
                A.set_site_copy(b, k, a)
        A0 = A.clone()
        K.compress_var_apply_H_(A0, K.build_env(dims, dims, [1] * (na + 1), gpu_ctx, batch=len(copies)), A, A, H, 1)
        return [A0.sites_copy(b) for b in range(len(copies))]

    for got, alone in zip(run(states), [run([s])[0] for s in states]):
        assert all(np.array_equal(x, y) for x, y in zip(got, alone))
