"""Waits of a thread-block cluster that run out: one CTA (host-set hook) never publishes its
keys to the others.  Every CTA leaves the pair, which fails with MGCD_ERR_TIMEOUT; the other
pairs of a batch are exact, and the same context then computes correctly."""
import math
import random

import pytest

pytestmark = pytest.mark.gpu


def _pair(rng, nbits, gbits):
    g = rng.getrandbits(gbits) | (1 << (gbits - 1))
    return g * (rng.getrandbits(nbits - gbits) | 1), g * (rng.getrandbits(nbits - gbits) | 1)


@pytest.mark.parametrize("cta", [0, 1, 15])
def test_single_pair(mgcd, cta):
    rng = random.Random(cta)
    u, v = _pair(rng, 60000, 9000)                   # 16 CTAs
    with mgcd.Device(0, 32) as dev:
        dev.set_wait_timeout_ms(200)
        dev.test_withhold_cta(cta)
        with pytest.raises(mgcd.GcdError) as e:
            dev.gcd(u, v)
        assert mgcd.STATUS_NAMES[e.value.status] == "MGCD_ERR_TIMEOUT"
        dev.test_withhold_cta(-1)
        assert dev.gcd(u, v) == math.gcd(u, v)


@pytest.mark.parametrize("threads,k,ctas,cta", [(512, 1, 4, 4), (512, 1, 8, 9), (256, 2, 8, 8), (512, 2, 16, 17),
                                                (1024, 4, 8, 15), (256, 4, 2, 3)])
def test_batch(mgcd, threads, k, ctas, cta):
    """Pairs of the cluster class: the second cluster's first or another CTA withholds."""
    rng = random.Random(threads + k + ctas)
    pairs = [_pair(rng, rng.randint(180000, 200000), rng.randint(1, 60000)) for _ in range(14)]
    us, vs = [u for u, _ in pairs], [v for _, v in pairs]
    exp = [math.gcd(u, v) for u, v in pairs]
    with mgcd.Device(0, 32) as dev:
        dev.set_class_cluster(0, 2)                  # (class 0 is empty)
        dev.set_size_class(3, threads, k, 1.0)
        dev.set_cluster_size(ctas)
        dev.set_wait_timeout_ms(200)
        dev.test_withhold_cta(cta)
        res, st = dev.gcd_batch(us, vs, return_status=True)
        names = [mgcd.STATUS_NAMES[int(x)] for x in st]
        assert set(names) == {"MGCD_OK", "MGCD_ERR_TIMEOUT"}
        assert all(r == e for r, e, n in zip(res, exp, names) if n == "MGCD_OK")
        dev.test_withhold_cta(-1)
        assert dev.gcd_batch(us, vs) == exp


def test_small_batch(mgcd):
    """A batch of few pairs with the default settings, each pair on a cluster of its own."""
    rng = random.Random(9)
    pairs = [_pair(rng, 20000, 5000) for _ in range(10)]
    us, vs = [u for u, _ in pairs], [v for _, v in pairs]
    exp = [math.gcd(u, v) for u, v in pairs]
    with mgcd.Device(0, 32) as dev:
        dev.set_wait_timeout_ms(200)
        dev.test_withhold_cta(1)
        res, st = dev.gcd_batch(us, vs, return_status=True)
        names = [mgcd.STATUS_NAMES[int(x)] for x in st]
        assert set(names) == {"MGCD_OK", "MGCD_ERR_TIMEOUT"}
        assert all(r == e for r, e, n in zip(res, exp, names) if n == "MGCD_OK")
        dev.test_withhold_cta(-1)
        assert dev.gcd_batch(us, vs) == exp
