"""A context is created beside other work on the GPU without waiting for all of its SMs."""
import math
import random
import threading
import time

import pytest

pytestmark = pytest.mark.gpu


def test_creation_beside_a_running_batch(mgcd):
    """All but a dozen SMs are held by a batch of one pair per CTA for some tenths of a second."""
    torch = pytest.importorskip("torch")
    n = torch.cuda.get_device_properties(0).multi_processor_count - 12
    rng = random.Random(1)
    us = [rng.getrandbits(170000) | 1 for _ in range(n)]
    vs = [rng.getrandbits(170000) | 1 for _ in range(n)]
    with mgcd.Device(0, 32) as dev:
        dev.set_growth(0)
        dev.set_size_class(2, 1024, 1, 1.0)
        dev.batch_upload(*mgcd.pack_pairs(us, vs))
        dev.batch_run()
        dev.batch_sync()                             # (the kernels are loaded)
        ms = dev.batch_elapsed_ms()[0]
        dev.batch_run()
        wait = threading.Thread(target=dev.batch_sync)
        wait.start()
        time.sleep(0.02)
        t = time.perf_counter()
        with mgcd.Device(0, 32) as other:
            t = time.perf_counter() - t
            wait.join()
            assert t < 0.5e-3 * ms, (t, ms)
            u, v = us[0] << 250000 | 1, vs[0] << 250000 | 1
            assert other.gcd(u, v) == math.gcd(u, v)       # its first pair on a grid
