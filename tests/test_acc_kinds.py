"""The three ways of holding sums of products (Acc): their arithmetic restated in C over the ranges they are used
for (CPU), and calls that take each of them against the oracle or the separate operations (GPU)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="no C compiler")
def test_kinds_exact(tmp_path):
    exe = str(tmp_path / "acc_kinds_check")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "native", "acc_kinds_check.c"), "-lm"],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


def _open(bits, n_special):
    from shmoai_b200.ckks import CKKSContext

    ctx = CKKSContext(12, bits=bits, n_special=n_special)
    rng = np.random.default_rng(sum(bits))

    def res(*shape, L):
        return rng.integers(0, 1 << 62, (*shape, L, ctx.n), dtype=np.uint64) % ctx.primes[:L].astype(np.uint64)[:, None]

    return ctx, res


@pytest.mark.gpu
@pytest.mark.parametrize("bits,n_special", [
    ([52] + [30] * 9 + [52], 1), ([51] + [30] * 15 + [40], 1),  # inner products in halves below 2^40, 10 and 16 digits
    ([52] + [27] * 9 + [52], 1),                                # ... and below 2^28: 128 bits
    ([50] + [40] * 10 + [50] * 9, 9), ([52] + [28] * 10 + [52] * 9, 9)])  # conversions of nine limbs: split at 32
def test_keyswitch_over_prime_sizes(bits, n_special):
    import torch

    from oracle import oracle as O
    from shmoai_b200.ckks import to_device, to_host

    ctx, res = _open(bits, n_special)
    orc = O.Oracle(12, ctx.primes, ctx.nq, ctx.np)
    L = ctx.dnum * n_special
    key, d = res(ctx.dnum, 2, L=len(ctx.primes)), res(2, L=L)
    d[0] = ctx.primes[:L, None] - np.uint64(1)
    got = to_host(ctx.keyswitch(to_device(d), to_device(key)))
    torch.cuda.synchronize()
    for i in range(2):
        assert np.array_equal(got[i], orc.keyswitch(d[i], key)), i
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [[51, 46, 46, 51], [52, 30, 30, 52], [50, 27, 40, 50], [60, 50, 50, 60]])
@pytest.mark.parametrize("k", [1, 5, 32])
def test_accumulated_products(bits, k):
    """Sums of tensor and plaintext products against the products added one by one."""
    import torch

    from shmoai_b200._lib import check, lib
    from shmoai_b200.ckks import to_device

    P, U = ctypes.c_void_p, ctypes.c_uint32
    L_ = lib()
    L_.shm_multiply_accumulate.argtypes = [P, P, P, U, ctypes.c_int, P, U, U, ctypes.c_int, P]
    ctx, res = _open(bits, 1)
    L = ctx.nq
    A, B = ([to_device(res(2, 2, L=L)) for _ in range(k)] for _ in range(2))
    A[0][:] = B[0][:] = to_device(np.broadcast_to(ctx.primes[:L, None] - np.uint64(1), (2, 2, L, ctx.n)))
    pt = [to_device(res(L=L)) for _ in range(k)]
    st = P(torch.cuda.current_stream().cuda_stream)
    ptrs = lambda ts: (P * k)(*[t.data_ptr() for t in ts])
    out3, out2 = ctx.empty(2, 3, L, ctx.n), ctx.empty(2, 2, L, ctx.n)
    check(L_.shm_multiply_accumulate(ctx._h, ptrs(A), ptrs(B), k, 0, P(out3.data_ptr()), 2, L, 0, st))
    check(L_.shm_multiply_plain_accumulate(ctx._h, ptrs(A), ptrs(pt), k, P(out2.data_ptr()), 4, L, 0, st))
    want3, want2 = ctx.multiply(A[0], B[0]), ctx.multiply_plain(A[0], pt[0])
    for t in range(1, k):
        want3 = ctx.add(want3, ctx.multiply(A[t], B[t]))
        want2 = ctx.add(want2, ctx.multiply_plain(A[t], pt[t]))
    torch.cuda.synchronize()
    assert torch.equal(out3, want3) and torch.equal(out2, want2)
    ctx.close()
