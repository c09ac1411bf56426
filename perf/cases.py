"""The work that a user of this framework has it do, as cases that can be timed: single
gcds (one call each), batches end to end and in steps, the allocation-free call and the
request server, over the operand sizes, modulus widths and input mixes of the repository's
own configurations, tests and benchmark.

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what a program holds before the call (operands, context, server)
  run(state)           one pass through the public entry points; its outputs
  work(case)           bytes and integer operations one pass cannot do without
  exact(case, seed)    the outputs as Python's exact gcd gives them
"""
import importlib
import math

import numpy as np
import torch

mgcd = importlib.import_module("modgcd-onegpu_gb300")

# One context per modulus width and launch table, as a program keeps it.
_devices = {}


def _device(L, tuned):
    if (L, tuned) not in _devices:
        dev = mgcd.Device(0, L)
        if tuned:
            dev.load_tuning(mgcd.default_tuning_path(dev))
        _devices[L, tuned] = dev
    return _devices[L, tuned]


def listed():
    return [
        # The smallest call: a key-sized pair, one CTA; launches, copies and latency.
        {"name": "pair_512b", "kind": "pair", "L": 32, "ubits": 512, "vbits": 509, "gbits": 130},
        # The single-pair configuration (10,240-bit operands, 2,048-bit gcd), as the signed
        # digits that the reference's kernel returns.
        {"name": "digits_10k", "kind": "digits", "L": 32, "ubits": 10240, "vbits": 10240, "gbits": 2048},
        # An ordinary large pair on a thread-block cluster, at the width of the tuned batches.
        {"name": "pair_64k", "kind": "pair", "L": 27, "ubits": 65536, "vbits": 65536, "gbits": 16384},
        # A ragged pair on the whole GPU (cooperative grid): unequal odd lengths.
        {"name": "pair_200k", "kind": "pair", "L": 27, "ubits": 200003, "vbits": 170111, "gbits": 30011},
        # The largest single pair of the latency sweep.
        {"name": "pair_1m", "kind": "pair", "L": 32, "ubits": 1 << 20, "vbits": 1 << 20, "gbits": 1 << 18},
        # A caller that owns all device memory: the allocation-free entry point.
        {"name": "noalloc_8k", "kind": "noalloc", "L": 32, "ubits": 8191, "vbits": 7999, "gbits": 1000},
        # The benchmark's mixed batch, end to end with host buffers.
        {"name": "batch_mixed", "kind": "batch", "L": 27, "tuned": True, "pairs": 4096, "lo": 1024, "hi": 65536,
         "mix": "mixed"},
        # A few pairs of all sizes with the default settings: the GPU is not full.
        {"name": "batch_few", "kind": "steps", "L": 32, "tuned": False, "pairs": 61, "lo": 1024, "hi": 65536,
         "mix": "mixed"},
        # The small pairs of the skewed workload: many short loops, set-up and finish count.
        {"name": "batch_small", "kind": "steps", "L": 32, "tuned": True, "pairs": 16384, "lo": 512, "hi": 4096,
         "mix": "small"},
        # Pairs above one CTA (size class 3): K pairs per thread-block cluster.
        {"name": "batch_large", "kind": "steps", "L": 32, "tuned": True, "pairs": 24, "lo": 160000, "hi": 300000,
         "mix": "mixed"},
        # A resident batch replayed from a CUDA graph: device work and the results' way back.
        {"name": "graph_1000", "kind": "graph", "L": 27, "tuned": True, "pairs": 1000, "lo": 2000, "hi": 16384,
         "mix": "mixed"},
        # A burst of requests on the server's continuous lanes.
        {"name": "serve_burst", "kind": "serve", "L": 32, "tuned": True, "pairs": 700, "lo": 1024, "hi": 32768,
         "mix": "mixed"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(2 ** rng.uniform(math.log2(lo), math.log2(hi))))


def draw(rng):
    L = rng.choice([22, 27, 27, 32, 32])
    kind = rng.choice(["pair", "pair", "digits", "noalloc", "batch", "batch", "steps", "steps", "graph", "serve"])
    if kind in ("pair", "digits", "noalloc"):
        L = 32 if kind == "noalloc" else L
        bits = _log_uniform(rng, 300, 30000 if kind == "noalloc" else 1 << 20 if L == 32 else 700000)
        v = max(64, int(bits / rng.uniform(1.0, 2.0)))
        return {"kind": kind, "L": L, "ubits": bits, "vbits": v, "gbits": int(rng.uniform(0.0, 0.6) * v)}
    tuned = rng.random() < 0.7
    if rng.random() < 0.2 and kind in ("batch", "steps"):          # pairs above one CTA
        lo, hi, n = 140000, 300000, rng.randint(2, 20)
    else:
        hi = _log_uniform(rng, 3000, 65536 if kind != "serve" else 32768)
        lo = max(512, int(hi / rng.uniform(2.0, 64.0)))
        # no more work than the largest listed batch: pairs times the square of the sizes
        most = int(4096 * (65536.0 / hi) ** 1.2)
        n = _log_uniform(rng, 1, min(most, 16384 if kind != "serve" else 1500))
    return {"kind": kind, "L": L, "tuned": tuned, "pairs": n, "lo": lo, "hi": hi,
            "mix": "small" if hi <= 6000 else "mixed"}


# ------------------------------------------------------------------------- inputs ----

def _bits(rng, n):
    """Random n-bit integer with its top two bits set, so that the product of an m-bit and an
    n-bit one has m + n bits (m, for n = 1): a case's sizes are the same for every seed."""
    return (int.from_bytes(rng.bytes((n + 7) // 8), "little") & ((1 << n) - 1)) | (3 << n >> 2)


def _sizes(case):
    """[(bits of u, bits of v, bits of the planted gcd; -1: v divides u)]."""
    if case["kind"] in ("pair", "digits", "noalloc"):
        return [(case["ubits"], case["vbits"], case["gbits"])]
    rng = np.random.default_rng([case["pairs"], case["lo"], case["hi"]])
    out = []
    for _ in range(case["pairs"]):
        if case["mix"] == "small":                 # U[lo, hi] bits, gcd up to a half
            u = int(rng.integers(case["lo"], case["hi"] + 1))
            v = int(rng.integers(u // 2, u + 1))
            out.append((u, v, int(rng.integers(1, max(2, v // 2)))))
            continue
        # log-uniform sizes, v up to half as long; a quarter coprime, one in twenty v | u,
        # the others with a planted gcd of up to half of v
        u = _log_uniform(rng, case["lo"], case["hi"])
        v = max(2, int(round(u / rng.uniform(1.0, 2.0))))
        r = rng.random()
        out.append((u, v, 0 if r < 0.25 else -1 if r < 0.30 else int(rng.uniform(0.0, 0.5) * v)))
    return out


def _pairs(case, seed):
    rng = np.random.default_rng([seed, 20240611])
    us, vs = [], []
    for u, v, g in _sizes(case):
        if g < 0:
            b = _bits(rng, v)
            us.append(b * _bits(rng, max(1, u - v)))
            vs.append(b)
        elif g == 0:
            us.append(_bits(rng, u))
            vs.append(_bits(rng, v))
        else:
            d = _bits(rng, g)
            us.append(d * _bits(rng, max(1, u - g)))
            vs.append(d * _bits(rng, max(1, v - g)))
    return us, vs


def _pinned(n, dtype):
    """A pinned host array, as a program that copies to the GPU often keeps."""
    t = torch.empty(max(int(n), 1) * np.dtype(dtype).itemsize, dtype=torch.uint8, pin_memory=True)
    return t.numpy().view(dtype)[: int(n)]


# ------------------------------------------------------------------------- passes ----

def prepare(case, seed):
    us, vs = _pairs(case, seed)
    kind, L = case["kind"], case["L"]
    s = {"kind": kind}
    if kind in ("pair", "digits"):
        s.update(dev=_device(L, False), u=us[0], v=vs[0], limbs=(vs[0].bit_length() + 31) // 32,
                 cap=mgcd.moduli_needed(us[0].bit_length(), L))
    elif kind == "noalloc":
        a, b = mgcd.to_limbs(us[0]), mgcd.to_limbs(vs[0])
        cap = mgcd.moduli_needed(32 * max(len(a), len(b)), 32)
        limbs = torch.from_numpy(np.concatenate([a, b]).view(np.int32)).cuda()
        s.update(limbs=limbs, un=len(a), vn=len(b), cap=cap, lib=mgcd.load(),
                 digits=torch.zeros(cap, 2, dtype=torch.int32, device="cuda"),
                 count=torch.zeros(1, dtype=torch.int32, device="cuda"),
                 status=torch.full((1,), -1, dtype=torch.int32, device="cuda"))
    else:
        packed = list(mgcd.pack_pairs(us, vs))
        if kind in ("batch", "steps"):
            limbs = _pinned(len(packed[0]), np.uint32)
            limbs[:] = packed[0]
            packed[0] = limbs
            s.update(dev=_device(L, case["tuned"]), packed=packed)
        if kind == "batch":
            off, cap, tot = mgcd.result_layout(packed[2], packed[4])
            n = len(us)
            s["out"] = (_pinned(tot, np.uint32), off, cap, np.zeros(n, np.uint32), np.zeros(n, np.int32))
        if kind in ("graph", "serve"):
            dev = mgcd.Device(0, L)                # its own: it keeps the batch, or the server
            if case["tuned"]:
                dev.load_tuning(mgcd.default_tuning_path(dev))
            s["dev"] = dev
            if kind == "graph":
                dev.batch_use_graph(True)
                dev.batch_upload(*packed)
            else:
                s.update(packed=packed, arrival=np.zeros(len(us)), server=mgcd.Server(dev))
    return s


def _padded(a, n):
    out = np.zeros((n,) + a.shape[1:], dtype=a.dtype)
    out[: len(a)] = a
    return out


def _gcds(g, off, n):
    """The gcds taken out of their slots (a slot's limbs past its gcd are unspecified)."""
    out = np.zeros_like(g)
    for o, k in zip(off.tolist(), n.tolist()):
        out[o: o + k] = g[o: o + k]
    return out


def run(s):
    kind = s["kind"]
    if kind == "pair":
        return _padded(mgcd.to_limbs(s["dev"].gcd(s["u"], s["v"])), s["limbs"])
    if kind == "digits":
        return _padded(np.array(s["dev"].gcd_digits(s["u"], s["v"]), dtype=np.int64), s["cap"])
    if kind == "noalloc":
        rc = s["lib"].mgcd_gcd_digits_noalloc(s["limbs"].data_ptr(), s["un"], s["vn"], s["digits"].data_ptr(),
                                              s["cap"], s["count"].data_ptr(), s["status"].data_ptr(),
                                              torch.cuda.current_stream().cuda_stream)
        if rc != mgcd.MGCD_OK:
            raise mgcd.GcdError(rc, mgcd.status_string(rc))
        return s["digits"], s["count"], s["status"]
    if kind == "serve":
        g, _, g_len, st, _, _ = s["server"].replay_packed(*s["packed"], s["arrival"])
        return g, g_len, st
    dev = s["dev"]
    if kind == "batch":
        g, off, g_len, st = dev.gcd_batch_packed(*s["packed"], out=s["out"])
        return _gcds(g, off, g_len), g_len.copy(), st.copy()
    if kind == "steps":
        dev.batch_upload(*s["packed"])
    dev.batch_run()
    g, _, g_len, st = dev.batch_download()
    return g, g_len, st


# ---------------------------------------------------------------- what it cannot avoid ----

# Integer operations of one Horner step of a residue, of one reduction-loop update (a
# modular inverse and two products) and of one digit's update of a modulus in the recovery.
OPS_RESIDUE, OPS_UPDATE, OPS_RECOVERY = 9, 257, 124


def work(case):
    nbytes = flops = 0
    for u, v, g in _sizes(case):
        u, v = max(u, v), min(u, v)
        g = v if g < 0 else g
        n = mgcd.moduli_needed(u, case["L"])
        # each iteration takes about log2(moduli) + 1 bits off both operands and one modulus
        # out of the loop; v reaches 0 when u is the gcd
        it = min(n, (v - g) / (math.log2(n) + 1.0) + 2)
        dig = g / case["L"] + 1
        nbytes += (u + v + g) / 8 + 12 * n + 8 * dig
        flops += OPS_RESIDUE * n * (u + v) / 32 + OPS_UPDATE * it * (n - it / 2) + \
            OPS_RECOVERY * dig * max(1.0, n - it - dig / 2)
    return {"bytes": float(nbytes), "flops": float(flops)}


def exact(case, seed):
    if case["kind"] not in ("pair", "batch", "steps", "graph", "serve"):
        return None                                # signed digits: fixed by the moduli table
    if sum(float(u) * (v - max(g, 0)) for u, v, g in _sizes(case)) > 3e12:
        return None                                # over about 20 seconds of exact gcds
    us, vs = _pairs(case, seed)
    words = lambda x: (x.bit_length() + 31) // 32  # noqa: E731
    gs = [math.gcd(u, v) for u, v in zip(us, vs)]
    if case["kind"] == "pair":
        cap = [words(vs[0])]
    else:
        cap = [max(words(u), words(v)) + 1 for u, v in zip(us, vs)]
    g = b"".join(x.to_bytes(4 * c, "little") for x, c in zip(gs, cap))
    g = np.frombuffer(g, dtype="<u4").astype(np.uint32)
    if case["kind"] == "pair":
        return g
    return g, np.array([words(x) for x in gs], dtype=np.uint32), np.zeros(len(gs), dtype=np.int32)
