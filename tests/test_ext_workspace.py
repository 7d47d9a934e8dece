"""The extended Sh-Rot's workspace: no more than the call uses (its inner products go straight to the outputs), and
nothing is written beyond it."""
import ctypes

import numpy as np
import pytest

P, U, SZ = ctypes.c_void_p, ctypes.c_uint32, ctypes.c_size_t


@pytest.mark.gpu
@pytest.mark.parametrize("n_groups,n,L", [(1, 1, 1), (3, 4, 5), (2, 8, 8)])
@pytest.mark.parametrize("in_ext", [0, 1])
def test_shared_rotate_ext_workspace(n_groups, n, L, in_ext):
    import torch

    from shmoai_b200._lib import check, lib
    from shmoai_b200.ckks import CKKSContext

    L_ = lib()
    L_.shm_shared_rotate_ext_workspace_bytes.restype = SZ
    L_.shm_shared_rotate_ext_workspace_bytes.argtypes = [P, U, U, U]
    L_.shm_shared_rotate_ext.argtypes = [P, P, ctypes.c_int, U, U, U, P, P, P, U, P, SZ, P]
    ctx = CKKSContext(12, bits=[50] + [45] * 7 + [50] * 2, n_special=2)
    N, LP, beta, H = ctx.n, L + 2, (L + 1) // 2, n + 1
    rng = np.random.default_rng(L)

    def res(*shape, primes):
        x = rng.integers(0, 1 << 62, (*shape, len(primes), N), dtype=np.uint64) % primes.astype(np.uint64)[:, None]
        return torch.from_numpy(x.view(np.int64)).cuda()

    x = res(n_groups, H, primes=np.concatenate([ctx.primes[:L], ctx.primes[ctx.nq:]]) if in_ext else ctx.primes[:L])
    keys = [res(ctx.dnum, H, primes=ctx.primes) for _ in range(2)]
    elts = (U * 2)(ctx.galois_elt(1), ctx.galois_elt(2))
    need = L_.shm_shared_rotate_ext_workspace_bytes(ctx._h, n_groups, n, L)
    assert need == 8 * n_groups * N * (L + beta * LP + LP + 2 * L)
    st = P(torch.cuda.current_stream().cuda_stream)

    def call(ws, size):
        outs = [ctx.empty(n_groups, H, LP, N) for _ in keys]
        ptrs = lambda ts: (P * 2)(*[t.data_ptr() for t in ts])
        check(L_.shm_shared_rotate_ext(ctx._h, P(x.data_ptr()), in_ext, n_groups, n, 2, elts, ptrs(keys), ptrs(outs), L,
                                       P(ws.data_ptr()), size, st))
        return outs

    wide = torch.full((2 * need // 8,), 0x5A5A5A5A, dtype=torch.int64, device="cuda")
    want = call(wide, wide.numel() * 8)
    tight = torch.full((need // 8 + 2 * N,), 0x5A5A5A5A, dtype=torch.int64, device="cuda")
    got = call(tight, need)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert bool((tight[need // 8:] == 0x5A5A5A5A).all()) and bool((wide[need // 8:] == 0x5A5A5A5A).all())
    ctx.close()
