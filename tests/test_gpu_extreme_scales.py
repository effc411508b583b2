"""Signals so large that an intermediate overflows before the values do."""
import ctypes

import numpy as np
import pytest

from test_gpu_estimation import restated_estimates
from test_gpu_estimation_values import K, N, _run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sfft_gb300 import _lib, build
    build.build()
    return torch, _lib, _lib.load()


@pytest.mark.parametrize("scale", [1.5 * 2.0 ** 126, 1.25 * 2.0 ** 127, 1.75 * 2.0 ** 127, 2.0 ** 128])
def test_fp64_medians_where_the_fp32_scale_overflows(env, scale):
    """Around 2^127 the FP32 copies of the bucket values are finite and the sums
    of their magnitudes are not: the error bound is infinite and proves no
    median.  A clean signal: its loops agree to more digits than FP32 has."""
    from sfft_gb300 import signals
    x, _, _ = signals.make_signal(N, K, 17)
    gi, gv, (pp, xs, ai, comb, wl, we) = _run(env, x * scale, True)
    rf, rv = restated_estimates(N, pp, xs, ai, comb, wl, we)
    o = np.argsort(rf)
    np.testing.assert_array_equal(gi, rf[o])
    np.testing.assert_array_equal(gv, rv[o])


@pytest.mark.parametrize("exponent", [0, 200, 300, 400, 500])
@pytest.mark.parametrize("n,k", [(1 << 16, 50), (1 << 18, 100)])
def test_v3_tones_of_any_size(env, oracle_lib, n, k, exponent):
    """|value|^2 fits up to 2^511: the oracle's values of the signal, scaled,
    within the 1e-10 of the parity tests, and nothing else that size.  (What is
    left of large tones passes v3's absolute thresholds and is listed too.)"""
    torch, _lib, L = env
    from sfft_gb300 import signals
    x, _, _ = signals.make_signal(n, k, 60)
    oi, ov = oracle_lib.OraclePlan(n, k, 2).exec(x, seed=3)
    scale = 2.0 ** exponent
    plan = L.sfft_make_plan_ex(n, k, 2, 0, ctypes.byref(_lib.Options(0, -1, 1)))
    assert plan, _lib.last_error()
    cap = L.sfft_output_capacity(plan)
    idx = torch.empty(cap, dtype=torch.int32, device="cuda")
    val = torch.empty(cap, dtype=torch.complex128, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    xd = torch.from_numpy(x * scale).cuda()
    torch.cuda.synchronize()
    assert L.sfft_exec_batch_ex(plan, 1, (ctypes.c_void_p * 1)(xd.data_ptr()), 0, (ctypes.c_uint * 1)(3), idx.data_ptr(),
                                val.data_ptr(), cnt.data_ptr(), cap, None) == 0, _lib.last_error()
    torch.cuda.synchronize()
    c = int(cnt[0])
    got = np.zeros(n, dtype=np.complex128)
    got[idx[:c].cpu().numpy()] = val[:c].cpu().numpy() / scale
    L.sfft_free_plan(plan)
    want = np.zeros(n, dtype=np.complex128)
    want[oi] = ov
    assert np.max(np.abs(got - want)) <= 1e-10
