"""The ct-pt matmul's CRT fold at every remainder of the modulus count by four (it takes the moduli in
groups of four), on primes below 2^52, against the CUDA-core contraction and the CPU oracle."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("wbits", [1, 9, 17, 25, 33, 39])  # 7 to 12 moduli
def test_crt_groups_match_oracle(wbits):
    import torch

    from shmoai_b200._lib import check, lib
    from shmoai_b200.ckks import CKKSContext, to_device, to_host

    primes = [int(p) for p in O.gen_primes(12, [51, 46, 46, 51])]
    ctx = CKKSContext(12, primes=primes, n_special=1)
    n_in, n_out, L, n = 8, 3, 3, 4096
    rng = np.random.default_rng(wbits)
    q = np.array(primes[:L], dtype=np.uint64)[None, None, :, None]
    X = rng.integers(0, 1 << 63, size=(n_in, 2, L, n), dtype=np.uint64) % q
    X[:, :, :, :64] = q - np.uint64(1)
    X[:, :, :, 64:128] = 0
    W = rng.integers(-(1 << wbits), 1 << wbits, size=(n_in, n_out), dtype=np.int64)
    W[:, 0] = (1 << wbits) - 1
    W[:, 1] = -(1 << wbits)
    Xd, Wd = to_device(X), torch.from_numpy(W).cuda()
    Y = to_host(ctx.ctpt_matmul(Xd, Wd))
    Yc = torch.empty(n_out, 2, L, n, dtype=torch.int64, device="cuda")
    check(lib().shm_ctpt_matmul_cuda_core(ctx._h, ctypes.c_void_p(Xd.data_ptr()), ctypes.c_void_p(Wd.data_ptr()),
                                          ctypes.c_void_p(Yc.data_ptr()), n_in, n_out, L,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert np.array_equal(Y, to_host(Yc))
    assert np.array_equal(Y, O.Oracle(12, primes, 3, 1).ctpt_matmul(X, W))
    ctx.close()
