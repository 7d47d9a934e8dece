"""Chains longer than a key switch takes: a context holds no conversion tables for levels that refuse one, and the
operations that take every level agree between levels."""
import ctypes

import numpy as np
import pytest

P, U, SZ = ctypes.c_void_p, ctypes.c_uint32, ctypes.c_size_t
NQ, NP, N = 120, 2, 4096


@pytest.mark.gpu
def test_context_memory():
    import torch

    from shmoai_b200.ckks import CKKSContext

    CKKSContext(12, bits=[50, 45, 50], n_special=1).close()  # the library's module is loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx = CKKSContext(12, bits=[50] + [45] * (NQ - 1) + [50] * NP, n_special=NP)
    used = before - torch.cuda.mem_get_info()[0]
    twiddles = (NQ + NP) * 8 * N * (4 + 2 * (1 + 1 / 8))
    conv = sum((-(-L // NP)) * (L + NP) * NP * 8 for L in range(1, NQ + 1))  # the load transform's constants
    levels = sum(L * (32 + 16 * 8 + (NP + 3) * 8) for L in range(1, NQ + 1)) + NQ * NQ * 16
    conv_bytes = sum((-(-L // NP) * (L + NP) + L) * 512 for L in range(1, 2 * 16 + 1))  # up to 16 digits
    assert used < twiddles + conv + levels + conv_bytes + 256 * 9 * NQ + (16 << 20), used  # 2 MB granules
    ctx.close()


@pytest.mark.gpu
def test_moddown_agrees_between_levels():
    import torch

    from shmoai_b200._lib import check, lib
    from shmoai_b200.ckks import CKKSContext

    L_ = lib()
    L_.shm_moddown_ext.argtypes = [P, P, P, U, U, P, SZ, P]
    L_.shm_moddown_ext_workspace_bytes.restype = SZ
    L_.shm_moddown_ext_workspace_bytes.argtypes = [P, U, U]
    ctx = CKKSContext(12, bits=[50] + [45] * (NQ - 1) + [50] * NP, n_special=NP)
    rng = np.random.default_rng(5)
    x = rng.integers(0, 1 << 62, (2, NQ + NP, N), dtype=np.uint64) % ctx.primes.astype(np.uint64)[:, None]

    def moddown(L):
        e = torch.from_numpy(np.concatenate([x[:, :L], x[:, NQ:]], axis=1).view(np.int64)).cuda()
        out = ctx.empty(2, L, N)
        ws = ctx.empty(L_.shm_moddown_ext_workspace_bytes(ctx._h, 2, L) // 8)
        check(L_.shm_moddown_ext(ctx._h, P(e.data_ptr()), P(out.data_ptr()), 2, L, P(ws.data_ptr()), ws.numel() * 8,
                                 P(torch.cuda.current_stream().cuda_stream)))
        return out

    whole = moddown(NQ)
    for L in (1, 30, 63, 64, 119):
        assert torch.equal(moddown(L), whole[:, :L]), L
    d = ctx.empty(1, 40, N)
    with pytest.raises(Exception, match="shape too large|more key digits"):
        ctx.keyswitch(d, d)  # 20 digits
    ctx.close()
