"""Estimation of few and of many candidates (v1 and voted v2): one warp per
candidate up to a number that depends on the batch, one thread beyond.  The
same signal alone and among others must give the same values, and both must
be the reference's on the run's own bucket values
(computefourier-1.0-2.0.cc:340-419), noiseless signals (all values near zero
or tied) among them."""
import ctypes

import numpy as np
import pytest

from test_gpu_estimation import _fetch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sfft_gb300 import _lib, build
    build.build()
    return torch, _lib, _lib.load()


def restated(n, pp, xs, ai, f, win):
    Ll, L = pp["loops_loc"], pp["loops_loc"] + pp["loops_est"]
    re, im = np.empty((L, f.size)), np.empty((L, f.size))
    for j in range(L):
        B = pp["B_loc"] if j < Ll else pp["B_est"]
        off = min(j, Ll) * pp["B_loc"] + max(0, j - Ll) * pp["B_est"]
        q = n // B
        w = win[0 if j < Ll else 1].reshape(-1, 4)
        p = (f * int(ai[j])) % n
        hashed, dist = p // q, p % q
        up = dist > q // 2
        hashed = np.where(up, (hashed + 1) % B, hashed)
        m = np.where(up, dist - q, dist) + (q - 1) // 2
        v = xs[off + hashed]
        c, d, den = w[m, 0], w[m, 1], w[m, 2]
        re[j] = (v.real * c + v.imag * d) / den
        im[j] = (v.real * d - v.imag * c) / den
    k = (L - 1) // 2
    return np.sort(re, axis=0)[k] + 1j * np.sort(im, axis=0)[k]


# (n, k, constants, version, batch): loop counts 2, 20, 30 and 32; few candidates, more than the warps take, a large batch
CASES = [
    (1 << 14, 5, (1.0, 1.0, 2.0, 1, 1, 1, 1, 1e-8, 1e-8), 1, 1),
    (1 << 16, 50, (1.0, 1.0, 2.0, 4, 16, 3, 1, 1e-8, 1e-8), 1, 1),
    (1 << 16, 50, (1.0, 1.0, 2.0, 4, 16, 3, 1, 1e-8, 1e-8), 1, 40),
    (1 << 20, 500, (1.0, 1.0, 2.0, 6, 24, 1, 1, 1e-8, 1e-8), 1, 2),
    (1 << 18, 50, (1.0, 1.0, 2.0, 4, 28, 2, 1, 1e-8, 1e-8), 2, 3),
]


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("snr", [30.0, None])
@pytest.mark.parametrize("n,k,prm,version,batch", CASES)
def test_listed_candidates_match_restatement(env, n, k, prm, version, batch, snr, prec):
    torch, _lib, L = env
    from sfft_gb300 import signals
    pr = _lib.Params(*prm)
    opt = _lib.Options(_lib.SFFT_PREC_FP32 if prec == "fp32" else _lib.SFFT_PREC_FP64, -1, batch)
    plan = L.sfft_make_plan_params(n, k, version - 1, ctypes.byref(pr), ctypes.byref(opt))
    assert plan, _lib.last_error()
    f = (ctypes.c_long * 11)()
    assert L.sfft_describe_plan_params(n, k, version - 1, ctypes.byref(pr), f, 11) == 11
    pp = dict(zip(["B_loc", "B_thresh", "B_est", "W_Comb", "Comb_loops", "loops_loc", "loops_thresh", "loops_est", "w_loc",
                   "w_est", "x_samp_size"], (int(v) for v in f)))
    if version == 2:
        assert L.sfft_plan_v2_voted(plan, 1) == 0, _lib.last_error()
    x = signals.make_signal_torch(n, k, 17, snr_db=snr)[0]
    cap = L.sfft_output_capacity(plan)
    Lr = pp["loops_loc"] + pp["loops_est"]
    got = []
    for m in {1, batch}:
        idx = torch.empty((m, cap), dtype=torch.int32, device="cuda")
        val = torch.empty((m, cap), dtype=torch.complex64 if prec == "fp32" else torch.complex128, device="cuda")
        cnt = torch.zeros(m, dtype=torch.int32, device="cuda")
        pin, seeds = (ctypes.c_void_p * m)(*[x.data_ptr()] * m), (ctypes.c_uint * m)(*[23] * m)
        torch.cuda.synchronize()
        assert L.sfft_exec_batch_ex(plan, m, pin, 0, seeds, idx.data_ptr(), val.data_ptr(), cnt.data_ptr(), cap, None) == 0
        assert L.sfft_sync(plan) == 0, _lib.last_error()
        for s in range(m):
            c = int(cnt[s])
            gi, gv = idx[s, :c].cpu().numpy().astype(np.int64), val[s, :c].cpu().numpy()
            o = np.argsort(gi)
            got.append((gi[o], gv[o]))
    for gi, gv in got[1:]:
        np.testing.assert_array_equal(gi, got[0][0])
        np.testing.assert_array_equal(gv, got[0][1])
    if prec == "fp64":
        xs = _fetch(L, plan, 3, pp["x_samp_size"], np.complex128)
        ai = _fetch(L, plan, 0, 2 * Lr, np.int32)[Lr:]
        win = [_fetch(L, plan, 8 + e, 4 * n // pp[b], np.float64) for e, b in enumerate(("B_loc", "B_est"))]
        np.testing.assert_array_equal(got[0][1], restated(n, pp, xs, ai, got[0][0], win))
    L.sfft_free_plan(plan)
