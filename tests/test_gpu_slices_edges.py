"""The split-precision GEMM at the edges of its slicing: rows per CTA, columns beyond the rows that fit
in shared memory (two passes for one or both operands), every layout, conjugation, rows far apart in
scale and of zeros."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import crand, empty_dev, from_dev, to_dev

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("M,N,K,slices", [(1, 1, 1, 6), (129, 33, 31, 3), (7, 300, 97, 7), (257, 65, 33, 6), (640, 500, 160, 6),
                                          (40, 30, 790, 5), (36, 70, 6300, 4)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_slicing_edges(gpu_ctx, M, N, K, slices, ta, tb):
    import torch
    from mpsb200 import _lib
    rng = np.random.default_rng(M + 10 * N + 100 * K + ta + 2 * tb)
    ca, cb = ta ^ (M & 1), tb
    sA, sB = crand(rng, *((K, M) if ta else (M, K))), crand(rng, *((N, K) if tb else (K, N)))
    A, B = (sA.T if ta else sA), (sB.T if tb else sB)
    A *= 2.0 ** rng.integers(-40, 40, size=(M, 1))
    B *= 2.0 ** rng.integers(-40, 40, size=(1, N))
    A[M // 2] = 0
    dA, dB, dC = to_dev(sA), to_dev(sB), empty_dev((M, N))
    one, zero = (np.array([v, 0.0]) for v in (1.0, 0.0))
    p = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    sa, sb = ((K, 1) if ta else (1, M)), ((N, 1) if tb else (1, K))
    torch.cuda.synchronize()
    _lib.call("mpsb_op_zgemm", gpu_ctx.h, M, N, K, C.c_void_p(dA.data_ptr()), *sa, ca, C.c_void_p(dB.data_ptr()), *sb, cb,
              C.c_void_p(dC.data_ptr()), 1, M, p(one), p(zero), slices)
    gpu_ctx.sync()
    got = from_dev(dC, (M, N))
    ref = (A.conj() if ca else A) @ (B.conj() if cb else B)
    # a row's digits stop at 2^(E - 7 S), E <= 1 + log2 of its largest component; the slice products of
    # levels >= S are dropped; 2 K real products a component; plus both sides' FP64 sums
    top = lambda X, ax: 2 * np.maximum(abs(X.real), abs(X.imag)).max(axis=ax)  # noqa: E731
    bound = 2 ** 1.5 * K * (slices + 2.1) * 2.0 ** (-7 * slices) * np.outer(top(A, 1), top(B, 0))
    bound += 4 * (K + slices + 4) * EPS * (abs(A) @ abs(B))
    assert np.all(abs(got - ref) <= bound)
