"""FP64 fold: the block size follows the number of bucket samples in the
launch, so a signal's samples and outputs must not depend on how many
signals are transformed with it.  Allocation-free entry point: several comb
loops keep their planes in the static scratch."""
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


def _run(env, plan, xs, cap):
    torch, _lib, L = env
    S = len(xs)
    idx = torch.empty(S, cap, dtype=torch.int32, device="cuda")
    val = torch.empty(S, cap, dtype=torch.complex128, device="cuda")
    cnt = torch.zeros(S, dtype=torch.int32, device="cuda")
    pin = (ctypes.c_void_p * S)(*[x.data_ptr() for x in xs])
    seed = (ctypes.c_uint * S)(*([9] * S))
    torch.cuda.synchronize()
    assert L.sfft_exec_batch_ex(plan, S, pin, 0, seed, idx.data_ptr(), val.data_ptr(), cnt.data_ptr(), cap, None) == 0, \
        _lib.last_error()
    assert L.sfft_sync(plan) == 0, _lib.last_error()
    out = []
    for i in range(S):
        c = int(cnt[i])
        gi, gv = idx[i, :c].cpu().numpy(), val[i, :c].cpu().numpy()
        o = np.argsort(gi)
        out.append((gi[o], gv[o]))
    return out


@pytest.mark.parametrize("n,k,version", [(1 << 10, 3, 0), (1 << 13, 20, 0), (1 << 16, 50, 1), (1 << 20, 100, 0)])
def test_outputs_do_not_depend_on_the_batch(env, n, k, version):
    torch, _lib, L = env
    from sfft_gb300 import signals
    opt = _lib.Options(_lib.SFFT_PREC_FP64, -1, 64)
    plan = L.sfft_make_plan_ex(n, k, version, 64, ctypes.byref(opt))
    assert plan, _lib.last_error()
    cap = L.sfft_output_capacity(plan)
    x = signals.make_signal_torch(n, k, 5)[0]
    (i1, v1), = _run(env, plan, [x], cap)
    assert i1.size
    for S in (2, 7, 40):
        for gi, gv in _run(env, plan, [x] * S, cap):
            np.testing.assert_array_equal(gi, i1)
            np.testing.assert_array_equal(gv, v1)
    L.sfft_free_plan(plan)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_noalloc_with_several_comb_loops(env, oracle_lib, prec):
    torch, _lib, L = env
    from sfft_gb300 import signals
    n, k, Bl, Be, W, cl = 1 << 14, 7, 256, 512, 1024, 8
    root = math.sqrt(n * k / math.log2(n))
    prm = _lib.Params((Bl + 0.5) * 1.001 / root, (Be + 0.5) * 1.001 / root, W * Bl / n * 1.0001, 3, 5, 2, cl, 1e-6, 1e-6)
    opt = _lib.Options(_lib.SFFT_PREC_FP32 if prec == "fp32" else _lib.SFFT_PREC_FP64, -1, 1)
    plan = L.sfft_make_plan_params(n, k, 1, ctypes.byref(prm), ctypes.byref(opt))
    assert plan, _lib.last_error()
    cap = L.sfft_output_capacity(plan)
    cdt, vdt = (np.complex64, torch.complex64) if prec == "fp32" else (np.complex128, torch.complex128)
    x = signals.make_signal_torch(n, k, 3, snr_db=20.0)[0]
    hi, hv = np.empty(cap, np.int32), np.empty(cap, np.complex128)
    idx = torch.empty(cap, dtype=torch.int32, device="cuda")
    val = torch.empty(cap, dtype=vdt, device="cuda")
    status = torch.zeros(2, dtype=torch.int32, device="cuda")
    xh = x.cpu().numpy()
    for seed in (21, 22):
        oracle_lib.seed_libc(seed)
        c = L.sfft_exec_sparse(plan, xh.ctypes.data, hi.ctypes.data, hv.ctypes.data, cap)
        assert c > 0, _lib.last_error()
        torch.cuda.synchronize()
        oracle_lib.seed_libc(seed)
        assert L.sfft_exec_noalloc(plan, x.data_ptr(), _lib.SFFT_IN_C128, idx.data_ptr(), val.data_ptr(), cap,
                                   status.data_ptr(), None) == 0, _lib.last_error()
        torch.cuda.synchronize()
        assert status.tolist() == [c, 0]
        o, g = np.argsort(hi[:c]), np.argsort(idx[:c].cpu().numpy())
        np.testing.assert_array_equal(idx[:c].cpu().numpy()[g], hi[:c][o])
        np.testing.assert_array_equal(val[:c].cpu().numpy()[g], hv[:c][o].astype(cdt))
    L.sfft_free_plan(plan)
