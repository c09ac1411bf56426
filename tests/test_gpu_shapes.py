"""Edges of the launch shapes and of the kernels' tiles: operand lengths around the limbs
taken per step, moduli counts around a warp, a CTA, a cluster and the grid, gcd lengths around
the recovery's panel, and batches around the counts at which their shape changes.  Digits
against the oracle's, gcds against Python's, exactly."""
import math
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(rng, nbits):
    return rng.getrandbits(nbits) | (1 << (nbits - 1)) | 1


def _oracle_digits(oracle, u, v, L, mods, nq=None):
    a, b = max(u, v), min(u, v)
    st, dig, _, _ = oracle.modgcd(a, b, L, mods, nq or oracle.num_moduli_needed(a.bit_length(), L))
    assert st == 0
    return dig


@pytest.mark.parametrize("L", [22, 27, 32])
def test_operand_lengths(mgcd, oracle, L):
    """1 to 10 limbs (four or two are taken per step), random and all-ones, alone and together."""
    rng = random.Random(100 + L)
    mods = oracle.gen_moduli(L, 512)
    us, vs = [], []
    for n in range(1, 11):
        for m in range(1, n + 1):
            us += [_exact(rng, 32 * n), (1 << 32 * n) - 1]
            vs += [_exact(rng, 32 * m), (1 << 32 * m) - 1]
    with mgcd.Device(0, L) as dev:
        assert dev.gcd_batch(us, vs) == [math.gcd(u, v) for u, v in zip(us, vs)]
        for i in range(0, len(us), 7):
            assert dev.gcd_digits(us[i], vs[i]) == _oracle_digits(oracle, us[i], vs[i], L, mods)


@pytest.mark.parametrize("L", [27, 32])
def test_single_pair_moduli_counts(mgcd, oracle, L):
    """A single pair's moduli (forced counts are multiples of 256) at the one-CTA limit, at
    clusters of one and more moduli per thread of a warp, and on the grid."""
    rng = random.Random(200 + L)
    mods = oracle.gen_moduli(L, 16640)
    g = _exact(rng, 150)
    u, v = g * _exact(rng, 250), g * _exact(rng, 200)
    with mgcd.Device(0, L) as dev:
        for nq in (256, 512, 768, 1024, 3840, 4096, 4352, 7936, 8192, 8448, 16128, 16384, 16640):
            dev.test_force_moduli(nq)
            assert dev.gcd_digits(u, v) == _oracle_digits(oracle, u, v, L, mods, nq), nq


@pytest.mark.parametrize("L", [27, 32])
def test_recovery_panels(mgcd, oracle, L):
    """gcds of about 1 to 97 digits around the panel's 32, a divisor of the other operand, and
    gcds that are products of moduli of the table (residues that are zero from the start)."""
    rng = random.Random(300 + L)
    mods = oracle.gen_moduli(L, 1024)
    pairs = [(u * g, v * g) for k in (0, 1, 30, 31, 32, 33, 63, 64, 65, 97)
             for g, u, v in [(_exact(rng, max(1, (L - 1) * k)), _exact(rng, 900), _exact(rng, 700))]]
    d = _exact(rng, 33 * (L - 1))
    pairs += [(d * _exact(rng, 800), d), (d, d)]
    for idx in ([0], [0, 1], [31, 32, 255], list(range(40))):
        p = 1
        for i in idx:
            p *= int(mods[i])
        pairs.append((p * _exact(rng, 700), p * _exact(rng, 600)))
    us, vs = [p[0] for p in pairs], [p[1] for p in pairs]
    with mgcd.Device(0, L) as dev:
        for u, v in pairs:
            assert dev.gcd_digits(u, v) == _oracle_digits(oracle, u, v, L, mods)
        assert dev.gcd_batch(us, vs) == [math.gcd(u, v) for u, v in pairs]              # spread
        assert dev.gcd_batch(us * 8, vs * 8) == [math.gcd(u, v) for u, v in pairs] * 8   # K per CTA


@pytest.mark.parametrize("L,tuned", [(22, False), (27, True), (32, True), (32, False)])
def test_small_batches_spread(mgcd, oracle, L, tuned):
    """Batches up to and just above half as many pairs as SMs, of every size class, with and
    without growth: exact gcds, and the digits of the moduli count that is reported."""
    rng = random.Random(400 + L)
    bits = [300, 2000, 5000, 9000, 18000, 40000] * 13
    pairs = []
    for nb in bits:
        g = _exact(rng, nb // 4)
        pairs.append((g * _exact(rng, nb - nb // 4), g * _exact(rng, nb // 2)))
    mods = oracle.gen_moduli(L, 8192)
    with mgcd.Device(0, L) as dev:
        if tuned:
            dev.load_tuning(mgcd.default_tuning_path(dev))
        for n, extra in ((1, 0), (2, 1), (6, 0), (61, 0), (75, 1), (76, 0), (77, 0), (78, 0)):
            us, vs = [p[0] for p in pairs[:n]], [p[1] for p in pairs[:n]]
            if extra:                               # one pair of the cluster class
                g = _exact(rng, 100000)
                us.append(g * _exact(rng, 80000))
                vs.append(g * _exact(rng, 1500))
            assert dev.gcd_batch(us, vs) == [math.gcd(u, v) for u, v in zip(us, vs)], n
            for i in range(n if n <= 6 else 0):     # (in a fuller batch a set may have grown)
                dig, nq = dev.batch_pair_digits(i)
                assert dig == _oracle_digits(oracle, us[i], vs[i], L, mods, nq)


@pytest.mark.parametrize("n,big", [(2431, 0), (2432, 1), (4864, 0), (4864, 1)])
def test_class0_counts(mgcd, n, big):
    """Queues of size class 0 around its shape's limits, with and without a pair whose set may
    pass 1,024 moduli."""
    rng = random.Random(500 + n)
    us, vs = [], []
    for _ in range(n - big):
        nb = rng.randint(100, 1500)
        g = _exact(rng, rng.randint(1, nb // 2))
        us.append(g * _exact(rng, nb))
        vs.append(g * _exact(rng, rng.randint(1, nb)))
    if big:
        us.append(_exact(rng, 6000))
        vs.append(_exact(rng, 5000))
    with mgcd.Device(0, 32) as dev:
        exp = [math.gcd(u, v) for u, v in zip(us, vs)]
        assert dev.gcd_batch(us, vs) == exp
        dev.load_tuning(mgcd.default_tuning_path(dev))
        assert dev.gcd_batch(us, vs) == exp


@pytest.mark.parametrize("n", [1215, 1216])
def test_class1_counts(mgcd, n):
    rng = random.Random(600 + n)
    us, vs = [], []
    for _ in range(n):
        nb = rng.randint(8000, 12000)
        g = _exact(rng, rng.randint(1, nb // 2))
        us.append(g * _exact(rng, nb - g.bit_length()))
        vs.append(g * _exact(rng, rng.randint(100, nb - g.bit_length())))
    with mgcd.Device(0, 27) as dev:
        dev.load_tuning(mgcd.default_tuning_path(dev))
        assert dev.gcd_batch(us, vs) == [math.gcd(u, v) for u, v in zip(us, vs)]


@pytest.mark.parametrize("bits", [2000, 2500, 4000, 4500, 6500, 30000])
def test_noalloc_on_one_cta_and_on_clusters(mgcd, bits):
    """Up to 512 moduli on one CTA, more on a cluster of 256-modulus CTAs: the regular entry
    point's digits."""
    torch = pytest.importorskip("torch")
    rng = random.Random(700 + bits)
    g = _exact(rng, bits // 3)
    u, v = g * _exact(rng, bits - bits // 3), g * _exact(rng, bits // 3)
    a, b = mgcd.to_limbs(u), mgcd.to_limbs(v)
    cap = mgcd.moduli_needed(32 * max(len(a), len(b)), 32)
    limbs = torch.from_numpy(np.concatenate([a, b]).view(np.int32)).cuda()
    dig = torch.zeros(cap, 2, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    rc = mgcd.load().mgcd_gcd_digits_noalloc(limbs.data_ptr(), len(a), len(b), dig.data_ptr(), cap, cnt.data_ptr(),
                                             st.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    got = [(p & 0xFFFFFFFF, w) for p, w in dig[: int(cnt.item())].tolist()]
    with mgcd.Device(0, 32) as dev:
        assert int(st.item()) == 0 and got == dev.gcd_digits(u, v)


def test_small_and_staged_uploads(mgcd):
    """Plans around 64 KB of operands, which go up in one copy or in three, results fetched in
    place (contiguous slots) and through the plan's own buffer, in turn on one context."""
    rng = random.Random(800)
    with mgcd.Device(0, 32) as dev:
        for n in (1, 3, 100, 140, 150, 160, 400, 2):
            us = [_exact(rng, 1900) * 3 for _ in range(n)] + [0, 5]
            vs = [_exact(rng, 1500) * 3 for _ in range(n)] + [7, 0]
            exp = [math.gcd(u, v) for u, v in zip(us, vs)]
            assert dev.gcd_batch(us, vs) == exp
            dev.batch_upload(*mgcd.pack_pairs(us, vs))
            for _ in range(2):
                dev.batch_run()
                g, off, glen, st = dev.batch_download()
                assert (np.asarray(st) == 0).all()
                assert [mgcd.from_limbs(g[int(o): int(o) + int(k)]) for o, k in zip(off, glen)] == exp
