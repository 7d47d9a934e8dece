"""The key-switch inner products' three summations: their arithmetic restated in C (CPU), and key switches
that take each of them against the oracle (GPU)."""
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="no C compiler")
def test_sums_exact():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "ip_sums_check")
        subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "native", "ip_sums_check.c"),
                        "-lm"], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("digits,bits", [
    (1, 51), (7, 51), (8, 51), (8, 46),  # doubles: up to eight digits below 2^51
    (9, 51), (16, 46), (4, 52),          # 26-bit halves: more digits, or primes up to 2^52
    (8, 36), (9, 36), (3, 55)])          # primes below 2^40 on doubles, then 128 bits; above 2^52
def test_digit_counts_match_oracle(digits, bits):
    """One special prime: a digit per limb.  Hoisted rotations (permuted reads) and a shared-a rotation
    (the multi-half kernel) besides the plain key switch."""
    import torch

    from oracle import oracle as O
    from shmoai_b200.ckks import CKKSContext, to_device, to_host

    ctx = CKKSContext(12, bits=[bits] * (digits + 1), n_special=1)
    orc = O.Oracle(12, ctx.primes, ctx.nq, ctx.np)
    rng = np.random.default_rng(digits * 64 + bits)
    pr = ctx.primes.astype(np.uint64)

    def res(*shape, L):
        return rng.integers(0, 1 << 62, (*shape, L, ctx.n), dtype=np.uint64) % pr[:L][:, None]

    L, n = digits, 3
    key, shk = res(ctx.dnum, 2, L=len(pr)), res(ctx.dnum, n + 1, L=len(pr))
    ct, sh = res(2, 2, L=L), res(2, n + 1, L=L)
    ct[0] = pr[:L, None] - np.uint64(1)
    elt = ctx.galois_elt(1)
    ks = to_host(ctx.keyswitch(to_device(np.ascontiguousarray(ct[:, 1])), to_device(key)))
    hoisted = to_host(ctx.apply_galois_hoisted(to_device(ct), [elt], [to_device(key)])[0])
    rot = to_host(ctx.shared_rotate_hoisted(to_device(sh), [elt], [to_device(shk)])[0])
    torch.cuda.synchronize()
    for i in range(2):
        assert np.array_equal(ks[i], orc.keyswitch(ct[i, 1], key))
        assert np.array_equal(hoisted[i], orc.apply_galois_hoisted(ct[i], [elt], [key])[0])
        assert np.array_equal(rot[i], orc.shared_rotate_hoisted(sh[i], [elt], [shk])[0])
    ctx.close()
