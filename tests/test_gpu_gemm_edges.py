"""The FP64 GEMM at the edges of its 32 x 32 x 16 tiles, for every layout and conjugation, with the K
splits its rule picks for few tiles, and through the stride forms that a tensor map does not
describe (both strides beyond one, broadcast, reversed)."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import crand, from_dev, to_dev

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
AL, BE = 0.75 - 0.5j, -0.25 + 1.0j


def _gemm(ctx, M, N, K, a, sa, ca, b, sb, cb, c):
    """c (M x N, column-major) <- AL op(A) op(B) + BE c; a, b: (flat buffer, element offset), sa, sb: strides."""
    import torch
    from mpsb200 import _lib
    da, db, dc = to_dev(a[0]), to_dev(b[0]), to_dev(c)
    al, be = (np.array([z.real, z.imag]) for z in (AL, BE))
    p = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    torch.cuda.synchronize()
    _lib.call("mpsb_op_zgemm", ctx.h, M, N, K, C.c_void_p(da.data_ptr() + 16 * a[1]), sa[0], sa[1], ca,
              C.c_void_p(db.data_ptr() + 16 * b[1]), sb[0], sb[1], cb, C.c_void_p(dc.data_ptr()), 1, M, p(al), p(be), 0)
    ctx.sync()
    return from_dev(dc, (M, N))


def _check(got, A, B, c):
    # each entry is a sum of 4 K real products (as two chains) plus the scaling: |error| <= gamma |A||B|
    K = A.shape[1]
    bound = 4 * (K + 8) * EPS * (abs(AL) * (np.abs(A) @ np.abs(B)) + abs(BE) * np.abs(c)) * 2
    assert np.all(np.abs(got - (AL * (A @ B) + BE * c)) <= bound)


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 33, 15), (31, 32, 16), (32, 31, 17), (33, 65, 31), (64, 64, 512), (5, 7, 1000),
                                   (96, 100, 255), (129, 40, 48)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_gemm_tile_edges(gpu_ctx, M, N, K, ta, tb):
    rng = np.random.default_rng(M + 100 * N + 10000 * K + ta + 2 * tb)
    ca, cb = ta ^ (M & 1), tb
    sA, sB, c = crand(rng, *((K, M) if ta else (M, K))), crand(rng, *((N, K) if tb else (K, N))), crand(rng, M, N)
    A, B = (sA.T if ta else sA), (sB.T if tb else sB)
    got = _gemm(gpu_ctx, M, N, K, (sA, 0), (K, 1) if ta else (1, M), ca, (sB, 0), (N, 1) if tb else (1, K), cb, c)
    _check(got, A.conj() if ca else A, B.conj() if cb else B, c)


@pytest.mark.parametrize("M,N,K", [(40, 35, 33), (7, 70, 200)])
def test_gemm_stride_forms(gpu_ctx, M, N, K):
    rng = np.random.default_rng(M * N + K)
    A, B, c = crand(rng, M, K), crand(rng, K, N), crand(rng, M, N)
    # every other element of both indices
    wide = np.zeros((2 * M, 2 * K), dtype=complex)
    wide[::2, ::2] = A
    _check(_gemm(gpu_ctx, M, N, K, (wide, 0), (2, 4 * M), 0, (B, 0), (1, K), 0, c), A, B, c)
    # rows reversed, columns reversed
    _check(_gemm(gpu_ctx, M, N, K, (A, M - 1), (-1, M), 0, (B, 0), (1, K), 0, c), A[::-1], B, c)
    _check(_gemm(gpu_ctx, M, N, K, (A, 0), (1, M), 0, (B, K * (N - 1)), (1, -K), 0, c), A, B[:, ::-1], c)
    # one column of B for all
    _check(_gemm(gpu_ctx, M, N, K, (A, 0), (1, M), 0, (B, 0), (1, 0), 0, c), A, np.repeat(B[:, :1], N, 1), c)
