"""The allocation-free Gram product at sizes that take its two tile orders (64 and 32), with
remainders, in one and several K chunks, against NumPy.

Every entry is a sum of K products: here and in NumPy |ΔS_ij| ≤ (K + 16)·eps·(|P|ᵀ|P|)_ij."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("m,K", [(1, 1), (5, 333), (33, 127), (61, 129), (317, 2049), (1000, 515), (1999, 4097),
                                 (2048, 1001)])
def test_gram(m, K):
    import torch
    from sdpx_b200.cuda_backend import load_library
    lib = load_library()
    P = np.random.default_rng(m + K).standard_normal((K, m))
    d = torch.from_numpy(np.ascontiguousarray(P.T)).cuda()
    S = torch.full((m, m), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = lib.sdpx_b200_gram_noalloc(ctypes.c_void_p(d.data_ptr()), ctypes.c_int64(K), ctypes.c_int32(m),
                                    ctypes.c_void_p(S.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    got = S.cpu().numpy()
    assert np.array_equal(got, got.T)
    assert (np.abs(got - P.T @ P) <= (2 * K + 32) * EPS * (np.abs(P).T @ np.abs(P))).all()
