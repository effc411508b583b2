"""Estimation by comb residue class with 32, 128 (one group a CTA), 256 and
512 candidates per residue and the largest loop count: values equal the
restated estimates of the run's own buckets, bit for bit in FP64, and a
residue's candidates come in steps of max(R / 256, 1) repetitions."""
import ctypes
import math

import numpy as np
import pytest

from test_gpu_estimation import env  # noqa: F401
from test_gpu_estimation import test_estimation_matches_restatement as check

pytestmark = pytest.mark.gpu
N, K, B = 1 << 18, 40, 1024


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("est_loops", [5, 28])
@pytest.mark.parametrize("W", [8192, 2048, 1024, 512])
def test_groups(env, W, est_loops, prec):  # noqa: F811
    c = (B + 0.5) * 1.001 / math.sqrt(N * K / math.log2(N))
    check(env, N, K, (c, c, W * B / N * 1.0001, 4, est_loops, 3, 1, 1e-8, 1e-8), prec)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("W", [8192, 2048, 1024, 512, 256])
def test_output_order(env, W, prec):  # noqa: F811
    torch, _lib, L = env
    from sfft_gb300 import signals
    c = (B + 0.5) * 1.001 / math.sqrt(N * K / math.log2(N))
    prm = _lib.Params(c, c, W * B / N * 1.0001, 4, 5, 3, 1, 1e-8, 1e-8)
    opt = _lib.Options(_lib.SFFT_PREC_FP32 if prec == "fp32" else _lib.SFFT_PREC_FP64, -1, 1)
    plan = L.sfft_make_plan_params(N, K, 1, ctypes.byref(prm), ctypes.byref(opt))
    assert plan, _lib.last_error()
    cap = L.sfft_output_capacity(plan)
    x = signals.make_signal_torch(N, K, 3, snr_db=30.0)[0]
    idx = torch.empty(cap, dtype=torch.int32, device="cuda")
    val = torch.empty(cap, dtype=torch.complex64 if prec == "fp32" else torch.complex128, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert L.sfft_exec_batch_ex(plan, 1, (ctypes.c_void_p * 1)(x.data_ptr()), 0, (ctypes.c_uint * 1)(5), idx.data_ptr(),
                                val.data_ptr(), cnt.data_ptr(), cap, None) == 0, _lib.last_error()
    assert L.sfft_sync(plan) == 0, _lib.last_error()
    comb = np.empty(W, np.int32)
    comb = comb[:L.sfft_debug_fetch(plan, 4, comb.ctypes.data, W)]
    R = N // W
    S = max(R // 256, 1)
    rep = (np.arange(S)[:, None] + S * np.arange(R // S)[None, :]).ravel()
    want = (comb[:, None] + W * rep[None, :]).ravel()
    np.testing.assert_array_equal(idx[:int(cnt[0])].cpu().numpy(), want)
    L.sfft_free_plan(plan)
