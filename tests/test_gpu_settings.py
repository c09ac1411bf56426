"""What a caller sets for batches is what runs, in batches of few pairs too: the shapes of the
launches (occupancy trace: one record per CTA, phases for the K-slot CTAs), the moduli counts
and reruns, with exact gcds."""
import math
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(rng, bits):
    out = []
    for nb in bits:
        g = rng.getrandbits(nb // 4) | 1
        out.append((g * (rng.getrandbits(nb - nb // 4) | 1), g * (rng.getrandbits(nb // 2) | 1)))
    return [p[0] for p in out], [p[1] for p in out]


def _run(dev, us, vs):
    """The size class's CTA counts, the K-slot CTAs among them, and the longest kernel's CTA size."""
    dev.set_cta_trace(True)
    assert dev.gcd_batch(us, vs) == [math.gcd(u, v) for u, v in zip(us, vs)]
    rec = dev.batch_cta_trace()
    dev.set_cta_trace(False)
    ctas = [int((rec["size_class"] == c).sum()) for c in range(4)]
    kslot = [int(((rec["size_class"] == c) & (rec["iterations"] > 0)).sum()) for c in range(4)]
    return ctas, kslot, dev.batch_elapsed_ms()[2]


@pytest.mark.parametrize("threads,k", [(256, 2), (512, 4), (512, 8), (1024, 2)])
def test_class_shapes(mgcd, threads, k):
    rng = random.Random(threads + k)
    us, vs = _pairs(rng, [3000] * 16 + [12000] * 8 + [40000] * 3)
    with mgcd.Device(0, 32) as dev:
        assert dev.spread()
        assert _run(dev, us, vs)[1] == [0, 0, 0, 0]          # on clusters
        for c in (0, 1, 2):
            dev.set_size_class(c, threads, k, 1.0)
        assert not dev.spread()
        ctas, kslot, longest = _run(dev, us, vs)
        assert ctas == kslot == [-(-16 // k), -(-8 // k), -(-3 // k), 0] and longest == threads
        dev.set_spread(True)
        assert _run(dev, us, vs)[1] == [0, 0, 0, 0]
        dev.set_spread(False)
        assert _run(dev, us, vs)[1] == ctas


@pytest.mark.parametrize("threads,k,ctas", [(512, 2, 8), (512, 4, 16), (1024, 1, 4), (256, 2, 2)])
def test_cluster_class_shapes(mgcd, threads, k, ctas):
    rng = random.Random(7 * threads + k)
    us, vs = _pairs(rng, [200000] * 5 + [3000] * 6)
    with mgcd.Device(0, 32) as dev:
        dev.set_size_class(3, threads, k, 1.0)
        dev.set_cluster_size(ctas)
        n, kslot, longest = _run(dev, us, vs)
        assert n[3] == ctas * -(-5 // k) and longest == threads
        assert n[0] == kslot[0] > 0


def test_fraction_and_growth(mgcd, oracle):
    """A low fraction reruns the pairs it cannot hold; a pair's set grows from where it is set."""
    rng = random.Random(3)
    us, vs = _pairs(rng, [230000] * 3 + [20000] * 4)
    us.append(rng.getrandbits(240000) | 1)                   # (almost surely) coprime
    vs.append(rng.getrandbits(239000) | 1)
    exp = [math.gcd(u, v) for u, v in zip(us, vs)]
    with mgcd.Device(0, 32) as dev:
        dev.set_size_class(3, 512, 2, 0.6)
        dev.set_cluster_size(4)
        assert dev.gcd_batch(us, vs) == exp
        assert dev.batch_retried() > 0
    with mgcd.Device(0, 32) as dev:
        dev.set_growth(0.2, 20)
        us, vs = us[3:7], vs[3:7]
        assert dev.gcd_batch(us, vs) == exp[3:7]
        for i, (u, v) in enumerate(zip(us, vs)):
            a, b = max(u, v), min(u, v)
            ref = oracle.num_moduli_needed(a.bit_length(), 32)
            dig, n = dev.batch_pair_digits(i)
            st, odig, _, on = oracle.modgcd_grow(a, b, 32, oracle.gen_moduli(32, 4096),
                                                 oracle.grow_start_count(ref, 0.2), oracle.grow_cap(ref), 20)
            if st != 0:                                      # rerun with the reference's count
                st, odig, _, _ = oracle.modgcd(a, b, 32, oracle.gen_moduli(32, 4096), ref)
                on = ref
            assert st == 0 and (dig, n) == (odig, on)


def test_loaded_table_keeps_the_switch(mgcd):
    rng = random.Random(4)
    us, vs = _pairs(rng, [5000] * 20)
    with mgcd.Device(0, 27) as dev:
        dev.load_tuning(mgcd.default_tuning_path(dev))
        assert dev.spread() and _run(dev, us, vs)[1] == [0, 0, 0, 0]
        dev.set_spread(False)
        dev.load_tuning(mgcd.default_tuning_path(dev))
        assert not dev.spread() and sum(_run(dev, us, vs)[1]) > 0


@pytest.mark.parametrize("cls,threads,n,bits", [(0, 256, 16, 400), (0, 256, 32, 300), (1, 512, 8, 9000)])
def test_long_queues(mgcd, cls, threads, n, bits):
    """n pairs per SM, the least at which a default shape gives way to smaller CTAs: one that
    the caller has set, the same numbers even, does not."""
    torch = pytest.importorskip("torch")
    rng = random.Random(n + bits)
    us, vs = _pairs(rng, [bits] * (n * torch.cuda.get_device_properties(0).multi_processor_count))
    with mgcd.Device(0, 32) as dev:
        assert dev.get_size_class(cls)[:2] == (threads, 2)
        assert _run(dev, us, vs)[2] == threads // 2
        dev.set_size_class(cls, threads, 2, 1.0)
        assert _run(dev, us, vs)[2] == threads
        dev.load_tuning(mgcd.default_tuning_path(dev))
        assert dev.get_size_class(cls)[:2] == (threads, 2)
        assert _run(dev, us, vs)[2] == threads // 2


def test_class2_queues(mgcd):
    """By default two pairs per CTA while they fit the SMs, four beyond."""
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    us, vs = _pairs(random.Random(5), [40000] * (2 * sms + 1))
    with mgcd.Device(0, 32) as dev:
        assert _run(dev, us[:-1], vs[:-1])[0] == [0, 0, sms, 0]
        assert _run(dev, us, vs)[0] == [0, 0, -(-(2 * sms + 1) // 4), 0]
        dev.set_size_class(2, 1024, 4, 1.0)
        assert _run(dev, us[:-1], vs[:-1])[0] == [0, 0, -(-2 * sms // 4), 0]


@pytest.mark.parametrize("L", [27, 32])
def test_small_batch_of_equal_pairs(mgcd, L):
    """Half as many pairs as SMs: clusters of two CTAs, one pair each, rather than larger
    clusters with several pairs."""
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    us, vs = _pairs(random.Random(6), [40000] * (sms // 2))
    with mgcd.Device(0, L) as dev:
        assert _run(dev, us, vs)[0] == [0, 0, sms // 2 * 2, 0]


@pytest.mark.parametrize("bits", [[200000] * 30 + [16000] * 46, [200000] * 3 + [64000] * 40 + [3000] * 30,
                                  [64000] * 50 + [16000] * 20])
def test_small_batch_fits_the_sms(mgcd, bits):
    """The classes of a small batch share the SMs: no more CTAs than SMs."""
    torch = pytest.importorskip("torch")
    us, vs = _pairs(random.Random(7), bits)
    with mgcd.Device(0, 27) as dev:
        assert sum(_run(dev, us, vs)[0]) <= torch.cuda.get_device_properties(0).multi_processor_count


def test_shapes_do_not_depend_on_earlier_batches(mgcd):
    """A small batch takes the same shapes and gives the same results after many uploads of
    other sizes (the context keeps a bounded number of the runtime's answers)."""
    rng = random.Random(8)
    us, vs = _pairs(rng, [30000] * 5 + [9000] * 7 + [2000] * 9)
    with mgcd.Device(0, 32) as dev:
        first = _run(dev, us, vs)
        for nb in range(2000, 62000, 1500):
            a, b = _pairs(rng, [nb] * 3)
            dev.batch_upload(*mgcd.pack_pairs(a, b))
        assert _run(dev, us, vs) == first


@pytest.mark.parametrize("L,k", [(32, 1), (32, 2), (27, 4)])
def test_operand_alignment_several_pairs_per_cta(mgcd, L, k):
    """Operands that start at every limb of a 16-byte line, of lengths around a staging tile's
    1,024 limbs, on the kernels with k pairs per CTA."""
    rng = random.Random(9)
    us = [rng.getrandbits(32 * n) | 1 << (32 * n - 1) | 1 for n in (1, 3, 4, 5, 1023, 1024, 1025, 2049)]
    vs = [rng.getrandbits(u.bit_length() - 5) | 1 for u in us]
    with mgcd.Device(0, L) as dev:
        for c in (0, 1, 2):
            dev.set_size_class(c, 512, k, 1.0)
        dev.set_cta_trace(True)
        for shift in range(4):
            gap, parts, off, places = np.zeros(shift, dtype=np.uint32), [], 0, []
            for x in [x for p in zip(us, vs) for x in p]:
                parts += [gap, mgcd.to_limbs(x)]
                places.append((off + shift, len(parts[-1])))
                off += shift + len(parts[-1])
            o = np.array([p[0] for p in places], dtype=np.uint64)
            n = np.array([p[1] for p in places], dtype=np.uint32)
            g, g_off, g_len, st = dev.gcd_batch_packed(np.concatenate(parts).astype(np.uint32), o[0::2].copy(),
                                                       n[0::2].copy(), o[1::2].copy(), n[1::2].copy())
            assert (st == 0).all()
            assert ((dev.batch_cta_trace()["iterations"] > 0) == (k > 1)).any()
            for i, (u, v) in enumerate(zip(us, vs)):
                a = int(g_off[i])
                assert mgcd.from_limbs(g[a: a + int(g_len[i])]) == math.gcd(u, v), (shift, i)
