"""Base conversion by byte products (conv.cu): its quotient arithmetic restated in Python (CPU), and the
key switch through it against the oracle over digit sizes, short last digits and prime sizes (GPU)."""
import random

import numpy as np
import pytest

LIM51, LIM61 = 1 << 51, 1 << 61


def _step(ys, cs, q):
    """One coefficient as the kernel forms it: the double or integer it stores, from the byte sums."""
    sums = [0] * 8
    for y, c in zip(ys, cs):
        for b in range(8):
            k = (c << (8 * b)) % q
            for o in range(8):
                sums[o] += ((y >> (8 * b)) & 255) * ((k >> (8 * o)) & 255)
    assert max(sums) < 1 << 22
    u = [sums[2 * i] + (sums[2 * i + 1] << 8) for i in range(4)]
    low = u[0] + (u[1] << 16)
    t = u[2] + (low >> 32)
    high = t + (u[3] << 16)
    assert t < 1 << 32 and high < 1 << 52
    hd, k32 = float(high), 4294967296.0 * (1.0 / float(q))
    Q = int(np.rint(np.float64(hd) * np.float64(k32)))  # below 2^14: the fma's rounding to an integer
    return ((high << 32) | (low & 0xFFFFFFFF)) - Q * q


@pytest.mark.parametrize("qbits", [20, 30, 40, 46, 50, 51, 57, 60, 61])
def test_quotient_bound(qbits):
    rng = random.Random(qbits)
    for slots in (1, 5, 6, 8):
        for _ in range(60):
            q = rng.randrange(1 << (qbits - 1), 1 << qbits) | 1
            top = rng.choice([1 << 46, LIM51, LIM61])
            ys = [rng.choice([0, top - 1, rng.randrange(top)]) for _ in range(slots)]
            cs = [rng.choice([q - 1, 1, rng.randrange(q)]) for _ in range(slots)]
            r = _step(ys, cs, q)
            assert (r - sum(y * c for y, c in zip(ys, cs))) % q == 0
            # within q/2 + 2^32 of zero (the quotient sees high alone); one rounding of a quotient below 2^14
            assert abs(r) <= q // 2 + (1 << 33)
            if q >= LIM51:
                assert 0 <= r + (q if r < 0 else 0) < q


def _context(n_special, bits, log_n):
    from oracle import oracle as O
    from shmoai_b200.ckks import CKKSContext

    ctx = CKKSContext(log_n, bits=bits, n_special=n_special)
    return ctx, O.Oracle(log_n, ctx.primes, ctx.nq, ctx.np)


@pytest.mark.gpu
@pytest.mark.parametrize("log_n,n_special,qb,pb", [
    (12, 1, 40, 60), (12, 3, 46, 51), (12, 5, 51, 51), (12, 6, 30, 40), (12, 7, 50, 60), (12, 8, 50, 60),
    (12, 9, 40, 45),  # more limbs than the tensor-core conversion's slots: the load transform
    (16, 2, 46, 51), (16, 5, 51, 51)])
def test_keyswitch_matches_oracle(log_n, n_special, qb, pb):
    """Full and short last digits, an odd batch; rotations through the same ModUp."""
    import torch

    from shmoai_b200.ckks import to_device, to_host

    nq = 2 * n_special + 1 if n_special > 1 else 4
    bits = [min(qb + 4, 60)] + [qb] * (nq - 1) + [pb] * n_special
    ctx, orc = _context(n_special, bits, log_n)
    rng = np.random.default_rng(n_special * 100 + qb)
    pr = ctx.primes

    def res(*shape, L):
        return rng.integers(0, 1 << 62, (*shape, L, ctx.n), dtype=np.uint64) % pr[:L].astype(np.uint64)[:, None]

    key = res(ctx.dnum, 2, L=len(pr))
    for L in sorted({2 * n_special, n_special + 1, max(1, n_special - 1)} & set(range(1, ctx.dnum * n_special + 1))):
        d = res(3, L=L)
        d[1] = pr[:L, None] - np.uint64(1)
        got = to_host(ctx.keyswitch(to_device(d), to_device(key)))
        torch.cuda.synchronize()
        for i in range(3):
            assert np.array_equal(got[i], orc.keyswitch(d[i], key)), (L, i)
    ctx.close()
