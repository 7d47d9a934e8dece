"""The base conversion's pipeline over several coefficient tiles per CTA, and its column of overflow counts, against
the oracle; rotations through the same ModUp."""
import numpy as np
import pytest


def _open(log_n, bits, n_special):
    from oracle import oracle as O
    from shmoai_b200.ckks import CKKSContext

    ctx = CKKSContext(log_n, bits=bits, n_special=n_special)
    rng = np.random.default_rng(n_special * 64 + log_n)

    def res(*shape, L):
        return rng.integers(0, 1 << 62, (*shape, L, ctx.n), dtype=np.uint64) % ctx.primes[:L].astype(np.uint64)[:, None]

    return ctx, O.Oracle(log_n, ctx.primes, ctx.nq, ctx.np), res


def tiles_of(sets, log_n, sms=148):
    """conv_rows' rule: as many tiles of 256 coefficients per CTA as leave 16 CTAs per SM."""
    blocks, t = (1 << log_n) // 256, 1
    while t < 32 and t * 2 <= blocks and sets * (blocks // (t * 2)) >= 16 * sms:
        t *= 2
    return t


def test_batches_reach_the_tile_counts():
    assert [tiles_of(2 * n, 12) for n in (147, 148, 296, 592, 1184)] == [1, 2, 4, 8, 16]
    assert [tiles_of(2 * n, 16) for n in (9, 10, 19, 37)] == [1, 2, 4, 8]


# a key switch of two digits (one full, one short) converts 2 n sets up and 2 n down
@pytest.mark.gpu
@pytest.mark.parametrize("log_n,n", [(12, 148), (12, 296), (12, 592), (12, 1184), (16, 10), (16, 19), (16, 37)])
def test_keyswitch_batches(log_n, n):
    import torch

    from shmoai_b200.ckks import to_device, to_host

    ctx, orc, res = _open(log_n, [51] + [46] * 3 + [51] * 2, 2)
    L, k = 3, 5  # k different polynomials, repeated in an order that puts each into many sets
    key, d = res(ctx.dnum, 2, L=len(ctx.primes)), res(k, L=L)
    d[1] = ctx.primes[:L, None] - np.uint64(1)
    order = (np.arange(n) * 3 + np.arange(n) // k) % k
    key_d, d_d = to_device(key), to_device(d)
    got = ctx.keyswitch(d_d[torch.from_numpy(order).cuda()].contiguous(), key_d)
    want = to_device(np.stack([orc.keyswitch(d[i], key) for i in range(k)]))
    torch.cuda.synchronize()
    assert torch.equal(got, want[torch.from_numpy(order).cuda()])
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n_special,qb,pb", [(1, 40, 51), (3, 46, 51), (6, 46, 51), (6, 50, 60), (7, 46, 51), (8, 50, 60)])
def test_relin_rescale_digit_sizes(n_special, qb, pb):
    """n_special + 1 limbs and the overflow count: all eight slots at 6, the transform's load from 7 on."""
    import ctypes

    import torch

    from shmoai_b200._lib import check, lib
    from shmoai_b200.ckks import to_device, to_host

    P, U = ctypes.c_void_p, ctypes.c_uint32
    L_ = lib()
    L_.shm_relinearize_rescale.argtypes = [P, P, P, P, U, U, P, ctypes.c_size_t, P]
    nq = max(2 * n_special, 3)
    ctx, orc, res = _open(12, [min(qb + 4, 60)] + [qb] * (nq - 1) + [pb] * n_special, n_special)
    key = res(ctx.dnum, 2, L=len(ctx.primes))
    for L in (2, nq - 1):
        ct3 = res(2, 3, L=L)
        ct3[0] = ctx.primes[:L, None] - np.uint64(1)
        x, k_d, out = to_device(ct3), to_device(key), ctx.empty(2, 2, L - 1, ctx.n)
        ws = ctx.empty(ctx.workspace_bytes("keyswitch", 2, L) // 8)
        check(L_.shm_relinearize_rescale(ctx._h, P(x.data_ptr()), P(k_d.data_ptr()), P(out.data_ptr()), 2, L,
                                         P(ws.data_ptr()), ws.numel() * 8, P(torch.cuda.current_stream().cuda_stream)))
        got = to_host(out)
        for i in range(2):
            assert np.array_equal(got[i], orc.rescale(orc.relinearize(ct3[i], key))), (L, i)
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n_special,qb,pb", [(2, 46, 51), (8, 50, 60), (9, 46, 51)])
def test_rotations_match_oracle(n_special, qb, pb):
    import torch

    from shmoai_b200.ckks import to_device, to_host

    nq = 2 * n_special
    ctx, orc, res = _open(12, [min(qb + 4, 58)] + [qb] * (nq - 1) + [min(pb, 58)] * n_special, n_special)
    L = nq - 1
    key, ct = res(ctx.dnum, 2, L=len(ctx.primes)), res(3, 2, L=L)
    elt = ctx.galois_elt(-3)
    got = to_host(ctx.rotate(to_device(ct), -3, to_device(key)))
    torch.cuda.synchronize()
    for i in range(3):
        assert np.array_equal(got[i], orc.apply_galois_ct(ct[i], elt, key)), i
    ctx.close()
