"""The calls this library's performance is judged by.

A case names a plan (version, n, k, precision), how it is called and how many
signals one call takes.  `call` is the entry point:

  execute   sfft.execute on a numpy array: the drop-in Python call of sFFT 0.1
            (host buffers, dense result)
  host      sfft_exec_many on page-locked host buffers, dense results
  device    sfft_exec_many on device buffers, dense results
  batch     sfft_exec_batch_ex: device signals, sparse device results, one
            seed per signal (plain v2 lists every comb candidate in a fixed
            order)
  voted     sfft_exec_batch_ex with a v2 plan in the voted mode; the short
            lists, whose order is free, are scattered into spectra
  mixed     MixedBatch: signals of uneven (n, k) through one captured graph,
            autotuned constants

Signals are seeded k-sparse spectra with |X| = 1 and uniform phases (the
n = 2^22, k = 100 workload: magnitudes log-uniform in [0.1, 10]); v1 and v3
run noiseless, v2 with complex Gaussian noise.  Plans are kept from one input
to the next, as a program keeps them.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from sfft_gb300 import _lib, signals
from sfft_gb300.serving import MixedBatch
from sfft_gb300.sfft import describe_plan, sfft

_libc = ctypes.CDLL(None)
_libc.srand48.argtypes = [ctypes.c_long]
_libc.srandom.argtypes = [ctypes.c_uint]


def _case(name, call, version, n, k, precision="fp64", batch=1, dtype="complex128"):
    c = {"call": call, "version": version, "n": n, "k": k, "precision": precision, "batch": batch, "dtype": dtype}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest drop-in call: latency, launches and copies
        _case("v1-8k-execute", "execute", 1, 1 << 13, 50),
        # one small request in the reduced-precision form, as a server sees it
        _case("v2-64k-f32-one", "batch", 2, 1 << 16, 50, "fp32"),
        # many ordinary v1 transforms of a program that keeps its data on the device
        _case("v1-64k-device-64", "device", 1, 1 << 16, 50, batch=64),
        # the metric workload: reduced precision, and the bit-exact form
        _case("v2-4m-f32-32", "batch", 2, 1 << 22, 100, "fp32", batch=32),
        _case("v2-4m-f64-8", "batch", 2, 1 << 22, 100, "fp64", batch=8),
        # complex64 signals, an odd number of them
        _case("v2-1m-f32-c64-13", "batch", 2, 1 << 20, 50, "fp32", batch=13, dtype="complex64"),
        # requests with many tones, only the voted candidates wanted, as a server runs them
        _case("v2-4m-k500-voted-4", "voted", 2, 1 << 22, 500, "fp32", batch=4),
        # exactly sparse signals: the large single transform, and a batch of small ones
        _case("v3-16m-device", "device", 3, 1 << 24, 1000),
        _case("v3-256k-device-16", "device", 3, 1 << 18, 100, batch=16),
        # the longest v1 signal: buckets beyond one block's shared memory
        _case("v1-16m-device", "device", 1, 1 << 24, 50),
        # the drop-in batch call on host buffers
        _case("v2-1m-host-8", "host", 2, 1 << 20, 50, batch=8),
        # uneven shapes of one service in one call
        {"name": "mixed-24", "call": "mixed", "count": 24, "shapes": 0, "log2n": 22},
    ]


def draw(rng):
    call = rng.choice(["execute", "host", "device", "device", "batch", "batch", "batch", "voted", "mixed"])
    if call == "mixed":
        return {"call": "mixed", "count": rng.randint(5, 24), "shapes": rng.randint(1, 9999), "log2n": rng.randint(19, 22)}
    if call == "device" and rng.random() < 0.5:
        n = 1 << rng.randint(17, 24)
        k = int(round(math.exp(rng.uniform(math.log(100), math.log(max(101, min(1000, n // 1024)))))))
        return _case("", call, 3, n, k, batch=_count(rng, n, 1 << 24, 32))
    version = 2 if call in ("batch", "voted") else rng.choice([1, 2])
    # the reference's tables hold k = 50 for every n, and more tones at 2^22
    lo, hi = {"execute": (13, 18), "host": (14, 20), "device": (13, 22), "batch": (14, 23), "voted": (16, 23)}[call]
    n = 1 << rng.randint(lo, hi)
    k = rng.choice([50, 100, 200, 500]) if n == 1 << 22 else 50
    precision = rng.choice(["fp32", "fp64"]) if call == "batch" else "fp32" if call == "voted" else "fp64"
    dtype = rng.choice(["complex128", "complex64"]) if call == "batch" else "complex128"
    batch = 1 if call == "execute" else _count(rng, n, {"host": 1 << 23, "voted": 1 << 24}.get(call, 1 << 25), 64)
    return _case("", call, version, n, k, precision, batch, dtype)


def _count(rng, n, most, limit):
    top = max(1, min(limit, most // n))
    return int(math.exp(rng.uniform(0, math.log(top + 0.99))))


# ------------------------------------------------------------------ plans --

@functools.lru_cache(maxsize=None)
def _plan(n, k, version, precision, batch, voted):
    import warnings
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return sfft(n, k, version, precision=precision, max_batch=batch, voted=voted)


def _shapes(case):
    rng = np.random.default_rng(case["shapes"])
    return [(1 << int(rng.integers(16, case["log2n"] + 1)), int(rng.integers(10, 501))) for _ in range(case["count"])]


class _View:
    """A device buffer of the library, for torch.as_tensor."""

    def __init__(self, ptr, count, kind):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": kind, "data": (ptr, False), "version": 2}


@functools.lru_cache(maxsize=None)
def _mixed(shapes):
    m = MixedBatch([(n, k, 2, "fp32") for n, k in shapes], tune=2)
    views = []
    for s in range(len(shapes)):
        idx, val, vb, cap = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_int(), ctypes.c_long()
        if m._L.sfft_mixed_result(m._m, s, ctypes.byref(idx), ctypes.byref(val), ctypes.byref(vb), ctypes.byref(cap)) < 0:
            raise RuntimeError(_lib.last_error())
        views.append((torch.as_tensor(_View(idx.value, cap.value, "<i4"), device="cuda"),
                      torch.as_tensor(_View(val.value, cap.value, "<c8"), device="cuda")))
    return m, views


# ----------------------------------------------------------------- states --

def _signal(case, n, k, version, seed):
    mag = (0.1, 10.0) if (n, k) == (1 << 22, 100) else None
    snr = None if version != 2 else 20.0 if mag else 40.0
    return signals.make_signal_torch(n, k, seed, mag=mag, snr_db=snr)


def _seeds(case, seed):
    return [(int(seed) * 1009 + 7 * i + 1) & 0x3fffffff for i in range(case.get("batch", case.get("count")))]


def prepare(case, seed):
    s = dict(case, seeds=_seeds(case, seed))
    call = case["call"]
    if call == "mixed":
        shapes = tuple(_shapes(case))
        s["mixed"], s["out"] = _mixed(shapes)
        s["x"] = [_signal(case, n, k, 2, sd)[0] for (n, k), sd in zip(shapes, s["seeds"])]
        return s
    n, k, version, batch = case["n"], case["k"], case["version"], case["batch"]
    p = s["plan"] = _plan(n, k, version, case["precision"], batch, call == "voted")
    xs = [_signal(case, n, k, version, sd)[0] for sd in s["seeds"]]
    if call == "execute":
        s["x"] = xs[0].cpu().numpy()
    elif call == "host":
        s["x"] = torch.stack(xs).cpu().pin_memory()
        s["out"] = torch.empty((batch, n), dtype=torch.complex128).pin_memory()
    elif call == "device":
        s["x"] = torch.stack(xs)
        s["out"] = torch.empty((batch, n), dtype=torch.complex128, device="cuda")
    else:
        s["x"] = torch.stack(xs).to(getattr(torch, case["dtype"]))
        val = torch.complex64 if case["precision"] == "fp32" else torch.complex128
        # the spectra have one more place, for the unused ends of the voted lists
        s["idx"] = torch.full((batch, p.capacity), n if call == "voted" else 0, dtype=torch.int32, device="cuda")
        s["val"] = torch.zeros((batch, p.capacity), dtype=val, device="cuda")
        s["count"] = torch.zeros(batch, dtype=torch.int32, device="cuda")
        s["stream"] = torch.cuda.Stream()
        s["cseeds"] = (ctypes.c_uint * batch)(*s["seeds"])
    if call != "execute":
        s["pin"] = (ctypes.c_void_p * batch)(*[x.data_ptr() for x in s["x"]])
    if call in ("host", "device"):
        s["pout"] = (ctypes.c_void_p * batch)(*[o.data_ptr() for o in s["out"]])
    torch.cuda.synchronize()
    return s


def run(s):
    call = s["call"]
    if call == "mixed":
        s["mixed"].run(s["x"], s["seeds"])
        return s["out"]
    p = s["plan"]
    if call in ("batch", "voted"):
        if p._L.sfft_exec_batch_ex(p.sfft_plan, s["batch"], s["pin"], 1 if s["dtype"] == "complex64" else 0, s["cseeds"],
                                   s["idx"].data_ptr(), s["val"].data_ptr(), s["count"].data_ptr(), p.capacity,
                                   s["stream"].cuda_stream) != 0:
            raise RuntimeError(_lib.last_error())
        if call == "batch":
            return s["idx"], s["val"], s["count"]
        with torch.cuda.stream(s["stream"]):
            out = torch.zeros((s["batch"], s["n"] + 1), dtype=s["val"].dtype, device="cuda")
            return out.scatter_(1, s["idx"].long(), s["val"])[:, :s["n"]], s["count"]
    # the drop-in calls draw from glibc's streams, which the program seeds
    _libc.srandom(s["seeds"][0])
    _libc.srand48(s["seeds"][0])
    if call == "execute":
        return p.execute(s["x"])
    p._L.sfft_exec_many(p.sfft_plan, s["batch"], s["pin"], s["pout"])
    if _lib.last_error():
        raise RuntimeError(_lib.last_error())
    return s["out"]


def exact(case, seed):
    """The spectrum for dense results: the FP64 FFT of the input, conjugated
    for v1/v2 as sFFT 0.1 returns it.  (Entries it does not recover are zero:
    on v2's noisy signals they are the noise floor.)  The sparse lists hold
    estimates of randomly chosen frequencies through random permutations; no
    closed value belongs to them."""
    if case["call"] not in ("execute", "host", "device"):
        return None
    out = []
    for sd in _seeds(case, seed):
        x = _signal(case, case["n"], case["k"], case["version"], sd)[0]
        X = torch.fft.fft(x) / case["n"]
        out.append(X if case["version"] == 3 else torch.conj(X).resolve_conj())
    return out[0].cpu().numpy() if case["call"] == "execute" else torch.stack(out)


# ------------------------------------------------------------------- work --

def _v12_work(f, n, item, out_item, voted, dense):
    """Bytes and operations of one v1/v2 transform with parameters f."""
    B, num, Be, W, cl, Ll, _, Le, wl, we, xs = f
    comb = W * cl if cl and W else 0
    samples = min(n, Ll * wl + Le * we + comb)
    cands = 0 if voted else min(W, cl * num) * (n // W)
    bytes_ = samples * item + (16 * n if dense else cands * out_item)
    fft = 5.0 * (Ll * B * math.log2(B) + Le * Be * math.log2(Be) + (comb * math.log2(W) if comb else 0))
    flops = 8.0 * (Ll * wl + Le * we) + fft + cands * 6.0 * (Ll + Le)
    return bytes_, flops


def work(case):
    if case["call"] == "mixed":
        L, total = _lib.load(), [0.0, 0.0]
        for n, k in _shapes(case):
            kk, prm, f = L.sfft_tuned_k(k), _lib.Params(), (ctypes.c_long * 11)()
            ok = L.sfft_tuned_params(n, kk, 1, ctypes.byref(prm)) >= 0
            if not ok or L.sfft_describe_plan_params(n, kk, 1, ctypes.byref(prm), f, 11) < 0:
                raise ValueError(_lib.last_error())
            b, o = _v12_work(list(f), n, 16, 12, False, False)
            total = [total[0] + b, total[1] + o]
        return {"bytes": total[0], "flops": total[1]}
    n, k, version = case["n"], case["k"], case["version"]
    dense = case["call"] in ("execute", "host", "device")
    d = describe_plan(n, k, version)
    if version == 3:
        W, B1, w1, B2, w2 = d["W_Man"], d["B_g1"], d["w_g1"], d["B_g2"], d["w_g2"]
        b = 16 * min(n, 2 * W + w1 + 1 + w2 + 1) + 16 * n
        o = sum(10.0 * m * math.log2(m) for m in (W, B1, B2)) + 16.0 * (w1 + w2) + 60.0 * k
    else:
        f = list(d.values())
        if version == 1:
            f[3], f[4] = 1, 0  # v1 has no comb
        item = 8 if case["dtype"] == "complex64" else 16
        b, o = _v12_work(f, n, item, 12 if case["precision"] == "fp32" else 20, case["call"] == "voted" or version == 1, dense)
        if case["call"] == "host":
            b = 32.0 * n  # the whole signal goes in over the link
    return {"bytes": float(b * case["batch"]), "flops": float(o * case["batch"])}
