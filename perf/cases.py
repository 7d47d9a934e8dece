"""Timing cases of the CKKS evaluation core: what a program that uses this framework has it do.

Every case goes through a public entry point of ``shmoai_b200.ckks.CKKSContext`` (the kernel ABI on
device tensors) or ``shmoai_b200.host`` (the C++ evaluator and bootstrapper).  Outputs are uint64
residues (as int64 bit patterns), so two versions of the library are compared bit for bit.

Prime chains:
  boot  N = 2^16, Q = [51] + 20 x [46] + 14 x [51], P = 5 x [51] (dnum 7): the bootstrapping chain
  prim  N = 2^16, Q = [60] + 23 x [50], P = 8 x [60] (dnum 3): the evaluator primitives' chain
  layer N = 2^16, Q = [51] + 23 x [46] + 11 x [51], P = 5 x [51]: the BERT layer's chain
  tiny  N = 2^12, Q = [60] + 5 x [40], P = 2 x [60]: the small ring of the tests
"""
import functools
import math

import numpy as np
import torch

from shmoai_b200.ckks import CKKSContext
from shmoai_b200.host import Bootstrapper, Host

CHAINS = {
    "boot": dict(log_n=16, bits=[51] + [46] * 20 + [51] * 14 + [51] * 5, n_special=5),
    "prim": dict(log_n=16, bits=[60] + [50] * 23 + [60] * 8, n_special=8),
    "layer": dict(log_n=16, bits=[51] + [46] * 23 + [51] * 11 + [51] * 5, n_special=5),
    "tiny": dict(log_n=12, bits=[60] + [40] * 5 + [60] * 2, n_special=2),
}
SCALE = 2.0 ** 46


def listed():
    return [
        # the smallest evaluator call: one ciphertext at the bootstrap's input level to coefficient
        # form and back (two polynomials of four limbs each way); latency counts
        dict(name="ntt_1ct_4limbs", op="ntt", chain="boot", polys=2, L=4),
        # a large batch of limbs at the top level, both directions (what a bootstrap's key switches do)
        dict(name="ntt_117polys_35limbs", op="ntt", chain="boot", polys=117, L=35),
        # HRotate of a single ciphertext on the primitives' chain (60-bit special primes)
        dict(name="rotate_1ct_24limbs", op="rotate", chain="prim", cts=1, L=24, step=1),
        # a ragged rotation batch in the middle of the bootstrapping chain, as the serving loop forms them
        dict(name="rotate_5cts_17limbs", op="rotate", chain="boot", cts=5, L=17, step=-3),
        # one ciphertext product with relinearisation and rescale on the primitives' chain
        dict(name="mul_1ct_24limbs", op="mul", chain="prim", cts=1, L=24),
        # a batch of products at EvalMod's levels
        dict(name="mul_16cts_27limbs", op="mul", chain="boot", cts=16, L=27),
        # baby steps of a CoeffToSlot layer on shared-a groups of eight: three hoisted rotations
        dict(name="shrotate_4x8_35limbs", op="shrotate", chain="boot", groups=4, members=8, L=35, elts=3),
        # bias / mask work of a layer: plaintext product, sum and rescale of a column block
        dict(name="plain_24cts_13limbs", op="plain", chain="layer", cts=24, L=13),
        # a small ragged projection
        dict(name="ctpt_100x70_7limbs", op="ctpt", chain="layer", n_in=100, n_out=70, L=7),
        # the hidden-size projection of BERT-base at 13 limbs
        dict(name="ctpt_768x768_13limbs", op="ctpt", chain="boot", n_in=768, n_out=768, L=13),
        # GELU on a block of ciphertexts (degree-24 series, six levels)
        dict(name="gelu_8cts_12limbs", op="gelu", chain="boot", cts=8, L=12),
        # a whole call: shared-a bootstrapping of two groups of four ciphertexts
        dict(name="boot_8cts_groups4", op="boot", chain="boot", cts=8, members=4),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    """Another case of the same ranges: mostly the single operations, now and then a whole call."""
    op = rng.choice(["ntt", "ntt", "rotate", "rotate", "mul", "mul", "shrotate", "fmt", "plain", "ctpt", "ctpt", "gelu",
                     "boot"])
    if op in ("ntt", "rotate", "mul", "plain"):
        chain = rng.choice(["boot", "boot", "layer", "prim", "tiny"])
        c = CHAINS[chain]
        nq = len(c["bits"]) - c["n_special"]
        L = rng.randint(2, nq)
        if op == "ntt":
            return dict(op=op, chain=chain, polys=_log_int(rng, 1, 4000 // L), L=rng.randint(1, nq))
        cts = _log_int(rng, 1, 24)
        if op == "rotate":
            return dict(op=op, chain=chain, cts=cts, L=L, step=rng.choice([-7, -1, 1, 2, 5, 64, 900]))
        return dict(op=op, chain=chain, cts=cts, L=L)
    if op == "shrotate":
        return dict(op=op, chain="boot", groups=_log_int(rng, 1, 6), members=rng.choice([2, 4, 5, 8]),
                    L=rng.randint(2, 35), elts=rng.randint(1, 3))
    if op == "fmt":
        return dict(op=op, chain="boot", groups=_log_int(rng, 1, 4), members=rng.choice([2, 4, 7]),
                    L_fwd=rng.randint(2, 4), L_back=rng.randint(2, 35))
    if op == "ctpt":
        return dict(op=op, chain=rng.choice(["boot", "layer"]), n_in=_log_int(rng, 8, 768), n_out=_log_int(rng, 8, 768),
                    L=rng.randint(2, 13))
    if op == "gelu":
        return dict(op=op, chain="boot", cts=_log_int(rng, 1, 16), L=rng.randint(8, 20))
    members = rng.choice([0, 2, 4])
    return dict(op=op, chain="boot", cts=rng.randint(1, 4) if members == 0 else members * rng.randint(1, 8 // members),
                members=members)


# ---------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _context(chain):
    """A program keeps one context per prime chain."""
    c = CHAINS[chain]
    return CKKSContext(c["log_n"], bits=c["bits"], n_special=c["n_special"])


def _primes(ctx):
    return torch.tensor(ctx.primes.astype(np.int64), device=ctx.device)


def _residues(gen, ctx, shape, primes):
    """Uniform residues [..., limbs, N]: ciphertexts and keys look uniform."""
    x = torch.empty(*shape, primes.numel(), ctx.n, dtype=torch.int64, device=ctx.device)
    flat = x.view(-1, primes.numel(), ctx.n)
    for i in range(0, flat.shape[0], 64):  # in blocks: the scratch stays small
        b = flat[i:i + 64]
        b.random_(0, 1 << 62, generator=gen)
        b.remainder_(primes.view(-1, 1))
    return x


def prepare(case, seed):
    op = case["op"]
    if op in ("gelu", "boot"):
        return _prepare_host(case, seed)
    ctx = _context(case["chain"])
    gen = torch.Generator(device=ctx.device).manual_seed(seed)
    pr = _primes(ctx)

    def ct(L, *shape):
        return _residues(gen, ctx, shape, pr[:L])

    def key(*shape):
        return _residues(gen, ctx, shape, pr)

    s = dict(op=op, ctx=ctx)
    if op == "ntt":  # two buffers, transformed in place
        s.update(x=ct(case["L"], case["polys"]), y=ct(case["L"], case["polys"]))
    elif op == "rotate":
        s.update(a=ct(case["L"], case["cts"], 2), step=case["step"], key=key(ctx.dnum, 2))
    elif op == "mul":
        s.update(a=ct(case["L"], case["cts"], 2), b=ct(case["L"], case["cts"], 2), key=key(ctx.dnum, 2))
    elif op == "plain":
        s.update(a=ct(case["L"], case["cts"], 2), b=ct(case["L"], case["cts"], 2), pt=ct(case["L"]))
    elif op == "shrotate":
        n = case["members"]
        s.update(a=ct(case["L"], case["groups"], n + 1), elts=[ctx.galois_elt(k) for k in (1, 2, 3)[:case["elts"]]],
                 keys=[key(ctx.dnum, n + 1) for _ in range(case["elts"])])
    elif op == "fmt":
        n, G = case["members"], case["groups"]
        s.update(n=n, a=ct(case["L_fwd"], G * n, 2), sh=ct(case["L_back"], G, n + 1), fkey=key(n, n + 1),
                 keys=[key(ctx.dnum, 2) for _ in range(n)])
    elif op == "ctpt":
        w = torch.randn(case["n_in"], case["n_out"], dtype=torch.float64, device=ctx.device, generator=gen)
        s.update(a=ct(case["L"], case["n_in"], 2), w=torch.round(w * 0.02 * 2.0 ** 40).to(torch.int64))
    return s


def _prepare_host(case, seed):
    """Keys and encrypted inputs of one user."""
    c = CHAINS[case["chain"]]
    h = Host(c["log_n"], bits=c["bits"], n_special=c["n_special"], hamming_weight=192, seed=seed)
    h.gen_relin_key()
    rng = np.random.default_rng(seed)
    slots = h.n // 2
    if case["op"] == "gelu":
        z = rng.uniform(-8.0, 8.0, (case["cts"], slots))
        return dict(op="gelu", host=h, ct=h.encrypt(z, SCALE, case["L"]))
    bs = Bootstrapper(h, SCALE, 4)
    if case["members"]:
        h.gen_shared_keys(case["members"], bs.galois_elts())
    else:
        h.gen_galois_keys(bs.galois_elts())
    z = rng.uniform(-1.0, 1.0, (case["cts"], slots)) + 1j * rng.uniform(-1.0, 1.0, (case["cts"], slots))
    return dict(op="boot", host=h, bs=bs, ct=h.encrypt(z, SCALE, 4), members=case["members"])


class _View:
    """A ciphertext batch of the host library as a CUDA array."""

    def __init__(self, ct):
        self.ct = ct
        self.__cuda_array_interface__ = dict(shape=(ct.count, ct.size, ct.level, ct.host.n), typestr="<i8",
                                             data=(ct.device_ptr(), False), version=3)


def _tensor(ct):
    return torch.as_tensor(_View(ct), device="cuda")


def run(s):
    op = s["op"]
    if op == "gelu":
        return _tensor(s["host"].gelu(s["ct"]))
    if op == "boot":
        return _tensor(s["bs"].run(s["ct"], s["members"]))
    ctx = s["ctx"]
    if op == "ntt":
        return ctx.ntt_inverse_(s["x"]), ctx.ntt_forward_(s["y"])
    if op == "rotate":
        return ctx.rotate(s["a"], s["step"], s["key"])
    if op == "mul":
        return ctx.rescale(ctx.relinearize(ctx.multiply(s["a"], s["b"]), s["key"]))
    if op == "plain":
        return ctx.rescale(ctx.add(ctx.multiply_plain(s["a"], s["pt"]), s["b"]))
    if op == "shrotate":
        return ctx.shared_rotate_hoisted(s["a"], s["elts"], s["keys"])
    if op == "fmt":
        return ctx.fmt_forward(s["a"], s["n"], s["fkey"]), ctx.fmt_backward(s["sh"], s["keys"])
    return ctx.ctpt_matmul(s["a"], s["w"])


def exact(case, seed):
    """Every output is a residue (a whole number), which stays equal: there is no rounding to compare."""
    return None


# ---------------------------------------------------------------------------


def work(case):
    """Bytes: inputs, keys and outputs once.  Flops: three operations for a butterfly (a modular
    product, a sum, a difference), two for a modular multiply-add."""
    c = CHAINS[case["chain"]]
    n, P = 1 << c["log_n"], c["n_special"]
    nq = len(c["bits"]) - P
    limb = 8 * n
    ntt = 3 * n // 2 * c["log_n"]  # one limb's transform
    mac = 2 * n

    def modup(L):
        beta = -(-L // P)
        return L * ntt + (beta * (L + P) - L) * (ntt + P * mac)

    def moddown(L):
        return P * ntt + L * (ntt + P * mac) + L * mac

    def switch(L, halves):  # inner products and ModDowns of one extension, `halves` outputs
        return halves * (-(-L // P) * (L + P) * mac + moddown(L))

    def key(L, halves):
        return -(-L // P) * halves * (L + P) * limb

    op = case["op"]
    if op == "ntt":
        rows = case["polys"] * case["L"]
        return dict(bytes=4 * rows * limb, flops=2 * rows * ntt)
    if op == "rotate":
        L, k = case["L"], case["cts"]
        return dict(bytes=4 * k * L * limb + key(L, 2), flops=k * (modup(L) + switch(L, 2)))
    if op == "mul":
        L, k = case["L"], case["cts"]
        return dict(bytes=k * (4 * L + 2 * (L - 1)) * limb + key(L, 2),
                    flops=k * (4 * L * mac + modup(L) + switch(L, 2) + 2 * (L * ntt + (L - 1) * mac)))
    if op == "plain":
        L, k = case["L"], case["cts"]
        return dict(bytes=(k * (4 * L + 2 * (L - 1)) + L) * limb, flops=2 * k * (L * mac + L * ntt + (L - 1) * mac))
    if op == "shrotate":
        L, G, n1, e = case["L"], case["groups"], case["members"] + 1, case["elts"]
        return dict(bytes=(1 + e) * G * n1 * L * limb + e * key(L, n1), flops=G * (modup(L) + e * switch(L, n1)))
    if op == "fmt":
        G, m, L, B = case["groups"], case["members"], case["L_fwd"], case["L_back"]
        return dict(bytes=G * ((3 * m + 1) * L + (3 * m + 1) * B) * limb + m * (m + 1) * (L + P) * limb + m * key(B, 2),
                    flops=G * (m * ((L + P) * ntt + P * L * mac) + (m + 1) * (m * (L + P) * mac + moddown(L)) + modup(B)
                               + m * switch(B, 2)))
    if op == "ctpt":
        i, o, L = case["n_in"], case["n_out"], case["L"]
        return dict(bytes=2 * (i + o) * L * limb + 8 * i * o, flops=2 * L * i * o * mac)
    if op == "gelu":  # nine products of the degree-24 series on falling levels, six rescales
        k, L = case["cts"], case["L"]
        levels = [L - 1, L - 2, L - 2, L - 3, L - 3, L - 3, L - 3, L - 4, L - 5]
        return dict(bytes=k * 2 * (L + L - 6) * limb + key(L - 1, 2),
                    flops=k * sum(4 * x * mac + modup(x) + switch(x, 2) + 2 * x * ntt for x in levels))
    # boot: the relinearisation key and the rotation keys of the six slot-transform layers (about
    # thirteen rotations each, three layers at 4..2 primes, three at the top), fifteen products on
    # both halves from the top down, the ciphertexts
    k, m = case["cts"], case["members"]
    g, h = (k // m, m + 1) if m else (k, 2)
    low, top = [4, 3, 2], [nq, nq - 1, nq - 2]
    rot = sum(g * (7 * modup(x) + 13 * switch(x, h)) for x in low + top)
    mul = 2 * k * sum(4 * x * mac + modup(x) + switch(x, 2) + 2 * x * ntt for x in [nq - 3 - i // 2 for i in range(15)])
    return dict(bytes=k * 2 * (4 + 23) * limb + key(nq, 2) + sum(13 * key(x, h) for x in low + top), flops=rot + mul)
