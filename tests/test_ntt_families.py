"""The NTT's FP64 passes: their arithmetic restated in C against exact integers (CPU), and the kernels
against the oracle at the edges of the butterfly families (GPU)."""
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="no C compiler")
def test_fp64_passes_exact():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "ntt_passes_check")
        subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "native", "ntt_passes_check.c"), "-lm"], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    lines = [x for x in r.stdout.splitlines() if x.startswith("q=")]
    assert len(lines) == 96 and all("mismatches 0, out of range 0" in x for x in lines), r.stdout


def _is_prime(n):
    """Miller-Rabin with the bases that decide every n below 2^64."""
    for p in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        if n % p == 0:
            return n == p
    d, r = n - 1, 0
    while d % 2 == 0:
        d, r = d // 2, r + 1
    for b in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        y = pow(b, d, n)
        if y in (1, n - 1):
            continue
        for _ in range(r - 1):
            y = y * y % n
            if y == n - 1:
                break
        else:
            return False
    return True


def _primes_near(limit, log_n, k):
    """The k largest primes = 1 mod 2N below `limit`."""
    step, out = 2 << log_n, []
    q = (limit - 2) // step * step + 1
    while len(out) < k:
        if _is_prime(q):
            out.append(q)
        q -= step
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("log_n", [12, 16])
@pytest.mark.parametrize("families", ["small", "large", "all"])
def test_family_edges_match_oracle(log_n, families):
    """Primes at both sides of every family limit, in the instantiation of each set of families; inputs
    at 0, q/2, q - 1 and random; the largest limb count of a launch's odd batch."""
    import torch

    from oracle import oracle as O
    from shmoai_b200.ckks import CKKSContext, to_device, to_host

    lim = {"grow64": (1 << 52) // 36, "c": 1 << 51, "grow": 1 << 57, "top": 1 << 61}
    pr = []
    if families in ("small", "all"):
        pr += _primes_near(1 << 30, log_n, 1) + _primes_near(lim["grow64"], log_n, 2)
    pr += _primes_near(lim["grow64"] + (1 << 24), log_n, 1) + _primes_near(lim["c"], log_n, 2)
    if families in ("large", "all"):
        pr += _primes_near(lim["c"] + (1 << 24), log_n, 1) + _primes_near(lim["grow"], log_n, 1)
        pr += _primes_near(lim["top"], log_n, 1)
    pr = list(dict.fromkeys(pr))
    n, L, rng = 1 << log_n, len(pr), np.random.default_rng(7)
    q = np.array(pr, dtype=np.uint64)[None, :, None]
    x = rng.integers(0, 1 << 63, (5, L, n), dtype=np.uint64) % q
    edge = np.concatenate([np.zeros_like(q), q // np.uint64(2), q - np.uint64(1)])
    x[1] = np.take_along_axis(np.broadcast_to(edge, (3, L, n)), rng.integers(0, 3, (1, L, n)), axis=0)[0]
    x[2] = (q - np.uint64(1))[0]
    ctx, orc = CKKSContext(log_n, primes=pr), O.Oracle(log_n, np.array(pr, dtype=np.uint64), L, 0)
    fwd, inv = to_host(ctx.ntt_forward_(to_device(x))), to_host(ctx.ntt_inverse_(to_device(x)))
    torch.cuda.synchronize()
    for p in range(x.shape[0]):
        assert np.array_equal(fwd[p], orc.ntt(x[p])), (p, "forward")
        assert np.array_equal(inv[p], orc.intt(x[p])), (p, "inverse")
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("polys,limbs", [(1, 1), (37, 4), (593, 1)])
def test_every_tile_matches_oracle(polys, limbs):
    """One row, the SMs' count and a row beyond whole waves, under the default tile and every tile set by
    hand."""
    from oracle import oracle as O
    from shmoai_b200._lib import check, lib
    from shmoai_b200.ckks import CKKSContext, to_device, to_host

    pr = _primes_near(1 << 46, 12, 3) + _primes_near(1 << 51, 12, 1)
    rng = np.random.default_rng(11)
    x = rng.integers(0, 1 << 63, (polys, limbs, 4096), dtype=np.uint64) % np.array(pr[:limbs], np.uint64)[None, :, None]
    orc = O.Oracle(12, np.array(pr, dtype=np.uint64), len(pr), 0)
    want = np.stack([orc.ntt(v) for v in x])
    ctx = CKKSContext(12, primes=pr)
    for tile in (None, 0, 1, 2, 3):
        if tile is not None:
            check(lib().shm_tune_set(ctx._h, 0, tile))
        d = ctx.ntt_forward_(to_device(x))
        assert np.array_equal(to_host(d), want), (tile, "forward")
        assert np.array_equal(to_host(ctx.ntt_inverse_(d)), x), (tile, "inverse")
    ctx.close()
