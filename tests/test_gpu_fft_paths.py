"""Bucket and comb FFTs in one CTA and over many CTAs, and the selection that
follows them, at the sizes where their shapes change.

Every shape performs the same stages with the same roundings, so a plan
whose FFTs are forced over many CTAs (SFFT_GB300_MAX_SMEM_FFT) must give the
bucket values, selected buckets and comb residues of the plan that keeps
them in one CTA, bit for bit.  The selected buckets are also compared with
find_largest_indices (src/utils.cc:130-158) restated on the bucket values.
"""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sfft_gb300 import _lib, build
    build.build()
    return torch, _lib, _lib.load()


def _largest(power, num):
    """Ascending indices of the num largest, ties at the cutoff in order."""
    cut = np.sort(power)[len(power) - num - 1]
    above = np.nonzero(power > cut)[0]
    equal = np.nonzero(power == cut)[0][:max(0, num - above.size)]
    return np.sort(np.concatenate([above, equal]))[:num]


def _fetch(L, plan, what, count, dtype):
    buf = np.empty(count, dtype=dtype)
    c = L.sfft_debug_fetch(plan, what, buf.ctypes.data, count)
    assert c >= 0
    return buf[:c]


# (n, k, B_loc, B_est, W, comb samplings)
SHAPES = [
    (1 << 10, 1, 16, 32, 64, 1),
    (1 << 12, 3, 128, 64, 512, 3),
    (1 << 14, 7, 256, 512, 1024, 8),
    (1 << 16, 50, 1024, 2048, 4096, 2),
    (1 << 16, 50, 4096, 128, 16384, 1),
    (1 << 18, 100, 8192, 4096, 32768, 2),
    (1 << 20, 100, 16384, 8192, 8192, 1),
    (1 << 20, 30, 32768, 1024, 131072, 1),
]


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("signal", ["noise", "zero"])
def test_many_cta_ffts_equal_one_cta(env, monkeypatch, shape, prec, signal):
    torch, _lib, L = env
    from sfft_gb300 import signals
    n, k, Bl, Be, W, cl = shape
    root = math.sqrt(n * k / math.log2(n))
    prm = _lib.Params((Bl + 0.5) * 1.001 / root, (Be + 0.5) * 1.001 / root, W * Bl / n * 1.0001, 3, 5, 2, cl, 1e-6, 1e-6)
    f = (ctypes.c_long * 11)()
    assert L.sfft_describe_plan_params(n, k, 1, ctypes.byref(prm), f, 11) == 11, _lib.last_error()
    assert (f[0], f[2], f[3], f[4]) == (Bl, Be, W, cl)
    x = (signals.make_signal_torch(n, k, 3, snr_db=20.0)[0] if signal == "noise"
         else torch.zeros(n, dtype=torch.complex128, device="cuda"))
    got = []
    for limit in (None, "16"):
        if limit:
            monkeypatch.setenv("SFFT_GB300_MAX_SMEM_FFT", limit)
        opt = _lib.Options(_lib.SFFT_PREC_FP32 if prec == "fp32" else _lib.SFFT_PREC_FP64, -1, 1)
        plan = L.sfft_make_plan_params(n, k, 1, ctypes.byref(prm), ctypes.byref(opt))
        assert plan, _lib.last_error()
        cap = L.sfft_output_capacity(plan)
        idx = torch.empty(cap, dtype=torch.int32, device="cuda")
        val = torch.empty(cap, dtype=torch.complex64 if prec == "fp32" else torch.complex128, device="cuda")
        cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
        pin, seed = (ctypes.c_void_p * 1)(x.data_ptr()), (ctypes.c_uint * 1)(9)
        torch.cuda.synchronize()
        for _ in range(2):   # the second run finds the first one's workspace
            assert L.sfft_exec_batch_ex(plan, 1, pin, 0, seed, idx.data_ptr(), val.data_ptr(), cnt.data_ptr(), cap,
                                        None) == 0, _lib.last_error()
            assert L.sfft_sync(plan) == 0, _lib.last_error()
        xs = _fetch(L, plan, 3, f[10], np.complex64 if prec == "fp32" else np.complex128)
        J = _fetch(L, plan, 1, 8 * 2 * k, np.int32).reshape(8, -1)
        got.append((xs, J, _fetch(L, plan, 4, W, np.int32), int(cnt[0])))
        L.sfft_free_plan(plan)
    for a, b in zip(got[0], got[1]):
        np.testing.assert_array_equal(a, b)
    xs, J, comb, count = got[0]
    assert np.all(np.diff(comb) > 0) and 2 * k <= comb.size <= min(W, 2 * k * cl) and count == comb.size * (n // W)
    at = 0
    for j in range(8):
        v = xs[at:at + (Bl if j < 3 else Be)]
        at += v.size
        if prec == "fp64":   # the same rounded products and sum
            np.testing.assert_array_equal(J[j], _largest(v.real * v.real + v.imag * v.imag, 2 * k))
    if signal == "zero":
        np.testing.assert_array_equal(J, np.tile(np.arange(2 * k, dtype=np.int32), (8, 1)))
