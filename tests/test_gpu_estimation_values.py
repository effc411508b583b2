"""FP64 estimation on values at the ends of the number range and on values that
are none.  The corrected quotient that replaces the IEEE division is used only
for exponents where it cannot over- or underflow, and the FP32 selection must
not claim a median it cannot see: a signal scaled by 1e-300 .. 1e290 gives the
restated estimates bit for bit, and infinities, NaNs and zeros give the same
through the residue-class kernel as through random lookups."""
import ctypes

import numpy as np
import pytest

from test_gpu_estimation import _fetch, restated_estimates

pytestmark = pytest.mark.gpu
N, K, PRM = 1 << 18, 40, (2.0, 2.0, 16.0, 4, 12, 3, 2, 1e-8, 1e-8)


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sfft_gb300 import _lib, build
    build.build()
    return torch, _lib, _lib.load()


def _run(env, x, want_state):
    torch, _lib, L = env
    prm = _lib.Params(*PRM)
    plan = L.sfft_make_plan_params(N, K, 1, ctypes.byref(prm), ctypes.byref(_lib.Options(0, -1, 1)))
    assert plan, _lib.last_error()
    cap = L.sfft_output_capacity(plan)
    idx = torch.empty(cap, dtype=torch.int32, device="cuda")
    val = torch.empty(cap, dtype=torch.complex128, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    xd = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    assert L.sfft_exec_batch_ex(plan, 1, (ctypes.c_void_p * 1)(xd.data_ptr()), 0, (ctypes.c_uint * 1)(3), idx.data_ptr(),
                                val.data_ptr(), cnt.data_ptr(), cap, None) == 0, _lib.last_error()
    assert L.sfft_sync(plan) == 0, _lib.last_error()
    c = int(cnt[0])
    gi, gv = idx[:c].cpu().numpy(), val[:c].cpu().numpy()
    o = np.argsort(gi)
    state = None
    if want_state:
        f = (ctypes.c_long * 11)()
        L.sfft_describe_plan_params(N, K, 1, ctypes.byref(prm), f, 11)
        pp = dict(zip(["B_loc", "B_thresh", "B_est", "W_Comb", "Comb_loops", "loops_loc", "loops_thresh", "loops_est",
                       "w_loc", "w_est", "x_samp_size"], (int(v) for v in f)))
        Lr = pp["loops_loc"] + pp["loops_est"]
        state = (pp, _fetch(L, plan, 3, pp["x_samp_size"], np.complex128), _fetch(L, plan, 0, 2 * Lr, np.int32)[Lr:],
                 _fetch(L, plan, 4, pp["W_Comb"], np.int32).astype(np.int64),
                 _fetch(L, plan, 8, 4 * N // pp["B_loc"], np.float64), _fetch(L, plan, 9, 4 * N // pp["B_est"], np.float64))
        assert not state[4].reshape(-1, 4)[:, 3].any() and not state[5].reshape(-1, 4)[:, 3].any()
    L.sfft_free_plan(plan)
    return gi[o], gv[o], state


@pytest.mark.parametrize("scale", [1.0, 1e-300, 1e-250, 1e-40, 1e30, 1e250])
def test_scaled_signals_match_restatement(env, scale):
    from sfft_gb300 import signals
    x, _, _ = signals.make_signal(N, K, 17, snr_db=30.0)
    gi, gv, (pp, xs, ai, comb, wl, we) = _run(env, x * scale, True)
    rf, rv = restated_estimates(N, pp, xs, ai, comb, wl, we)
    o = np.argsort(rf)
    np.testing.assert_array_equal(gi, rf[o])
    np.testing.assert_array_equal(gv, rv[o])


@pytest.mark.parametrize("kind", ["inf", "nan", "zeros", "one tone", "tiny"])
def test_odd_values_as_by_random_lookups(env, monkeypatch, kind):
    from sfft_gb300 import signals
    x, _, _ = signals.make_signal(N, K, 18, snr_db=30.0)
    if kind in ("inf", "nan"):
        x[12345] = complex(float(kind), 1.0)
    elif kind == "zeros":
        x[::2] = 0
    elif kind == "one tone":
        x = np.exp(2j * np.pi * 777 * np.arange(N) / N)
    else:
        x = x * 5e-324 ** 0.99
    a = _run(env, x, False)
    monkeypatch.setenv("SFFT_GB300_MAX_SMEM_FFT", "256")   # bucket FFTs beyond it: no grouped layout
    b = _run(env, x, False)
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1].view(np.float64), b[1].view(np.float64))
