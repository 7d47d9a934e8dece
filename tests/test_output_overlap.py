"""Outputs that lie over the rows a key switch has extended (the c1 or shared a rows, which no later step
of the call needs): each call gives what it gives with outputs of their own."""
import ctypes

import numpy as np
import pytest

P, U, SZ = ctypes.c_void_p, ctypes.c_uint32, ctypes.c_size_t


def _setup(n_special, n_groups, H, rows_after):
    """Context, keys and a buffer with the input at its head and room behind it."""
    import torch

    from shmoai_b200.ckks import CKKSContext

    nq = 2 * n_special
    ctx = CKKSContext(12, bits=[50] + [45] * (nq - 1) + [50] * n_special, n_special=n_special)
    L = nq - 1  # a short last digit
    rng = np.random.default_rng(n_special * 10 + n_groups)

    def res(*shape, L):
        x = rng.integers(0, 1 << 62, (*shape, L, ctx.n), dtype=np.uint64) % ctx.primes[:L].astype(np.uint64)[:, None]
        return torch.from_numpy(x.view(np.int64)).cuda()

    x = res(n_groups, H, L=L)
    buf = ctx.empty(x.numel() + rows_after * L * ctx.n)
    buf[:x.numel()] = x.view(-1)
    return ctx, L, x, buf, res


def _ptrs(ts):
    return (P * len(ts))(*[t.data_ptr() for t in ts])


@pytest.mark.gpu
@pytest.mark.parametrize("n_special", [2, 9])  # conversions by byte products, and in the transform's load
@pytest.mark.parametrize("n_groups", [1, 2])
@pytest.mark.parametrize("op", ["hoisted", "shared", "backward", "shared_ext"])
def test_output_over_extended_rows(op, n_groups, n_special):
    import torch

    from shmoai_b200._lib import check, lib

    L_ = lib()
    n = 1 if op == "hoisted" else 3  # members: the extended row is the last of a group's n + 1
    H = n + 1
    ctx, L, x, buf, res = _setup(n_special, n_groups, H, n_groups * 2 * H * 3)
    ln, LP = L * ctx.n, L + ctx.np
    st = P(torch.cuda.current_stream().cuda_stream)
    over = buf[(n_groups * H - 1) * ln:]  # begins at the last group's extended row
    elts = (U * 2)(ctx.galois_elt(1), ctx.galois_elt(2))
    if op == "backward":
        keys = [res(ctx.dnum, 2, L=len(ctx.primes)) for _ in range(n)]
        size = n_groups * n * 2 * ln
        ws = ctx.empty(L_.shm_fmt_switch_backward_workspace_bytes(ctx._h, n_groups, n, L) // 8)

        def call(src, outs):
            check(L_.shm_fmt_switch_backward(ctx._h, P(src.data_ptr()), n_groups, n, _ptrs(keys), P(outs[0].data_ptr()),
                                             L, P(ws.data_ptr()), ws.numel() * 8, st))
    elif op == "hoisted":
        keys = [res(ctx.dnum, 2, L=len(ctx.primes)) for _ in range(2)]
        size = n_groups * 2 * ln
        ws = ctx.empty(L_.shm_apply_galois_hoisted_workspace_bytes(ctx._h, n_groups, L) // 8)

        def call(src, outs):
            check(L_.shm_apply_galois_hoisted(ctx._h, P(src.data_ptr()), 2, elts, _ptrs(keys), _ptrs(outs), n_groups, L,
                                              P(ws.data_ptr()), ws.numel() * 8, st))
    else:
        keys = [res(ctx.dnum, H, L=len(ctx.primes)) for _ in range(2)]
        ext = op == "shared_ext"
        size = n_groups * H * (LP if ext else L) * ctx.n
        if ext:
            L_.shm_shared_rotate_ext_workspace_bytes.restype = SZ
            L_.shm_shared_rotate_ext_workspace_bytes.argtypes = [P, U, U, U]
            L_.shm_shared_rotate_ext.argtypes = [P, P, ctypes.c_int, U, U, U, P, P, P, U, P, SZ, P]
            ws = ctx.empty(L_.shm_shared_rotate_ext_workspace_bytes(ctx._h, n_groups, n, L) // 8)
        else:
            ws = ctx.empty(L_.shm_shared_rotate_workspace_bytes(ctx._h, n_groups, n, L) // 8)

        def call(src, outs):
            if ext:
                check(L_.shm_shared_rotate_ext(ctx._h, P(src.data_ptr()), 0, n_groups, n, 2, elts, _ptrs(keys),
                                               _ptrs(outs), L, P(ws.data_ptr()), ws.numel() * 8, st))
            else:
                check(L_.shm_shared_rotate_hoisted(ctx._h, P(src.data_ptr()), n_groups, n, 2, elts, _ptrs(keys),
                                                   _ptrs(outs), L, P(ws.data_ptr()), ws.numel() * 8, st))
    assert over.numel() >= size
    want = [ctx.empty(size), ctx.empty(size)]
    call(x, want)
    got = [over[:size], ctx.empty(size)]
    call(buf, got)
    torch.cuda.synchronize()
    for e in range(1 if op == "backward" else 2):
        assert torch.equal(got[e], want[e]), e
    ctx.close()
