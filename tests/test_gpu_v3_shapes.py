"""v3 alone and in batches: few signals run on clusters of 16 CTAs, many on
clusters of 8, and every size has its own split of the comb FFT and the
filter folds.  Slot 0 against the oracle (support equal, values within the
1e-10 of the parity tests), every other slot against the same signal alone:
the same support, values within 1e-11 of the largest (subtractions by FP64
atomics come in any order; each moves a bucket by half a unit in the last
place, some 10^2 of them by 10^-14 of it)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(oracle_lib):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sfft_gb300 import _lib, build
    build.build()
    return torch, _lib, _lib.load(), oracle_lib


@pytest.mark.parametrize("n,k,batch,c64", [
    (1 << 14, 8, 20, False),      # the smallest: 2 permuted buckets, comb of 64
    (1 << 15, 31, 5, False),
    (1 << 17, 127, 40, False),    # k no power of two
    (1 << 19, 400, 3, True),      # complex64 signals
    (1 << 21, 2047, 2, False),    # comb of 16384, 1024 and 256 buckets
    (1 << 21, 1023, 1, False),
])
def test_v3_alone_and_in_batches(env, n, k, batch, c64):
    torch, _lib, L, O = env
    from sfft_gb300 import signals
    sig = [signals.make_signal(n, k, 60 + s)[0] for s in range(min(batch, 3))]
    if c64:
        sig = [x.astype(np.complex64) for x in sig]
    dev = [torch.from_numpy(x).cuda() for x in sig]
    plan = L.sfft_make_plan_ex(n, k, 2, 0, ctypes.byref(_lib.Options(0, -1, batch)))
    assert plan, _lib.last_error()
    cap = L.sfft_output_capacity(plan)

    def run(which):
        m = len(which)
        idx = torch.empty((m, cap), dtype=torch.int32, device="cuda")
        val = torch.empty((m, cap), dtype=torch.complex128, device="cuda")
        cnt = torch.zeros(m, dtype=torch.int32, device="cuda")
        pin = (ctypes.c_void_p * m)(*[dev[w].data_ptr() for w in which])
        seeds = (ctypes.c_uint * m)(*[100 + w for w in which])
        torch.cuda.synchronize()
        assert L.sfft_exec_batch_ex(plan, m, pin, int(c64), seeds, idx.data_ptr(), val.data_ptr(), cnt.data_ptr(), cap,
                                    None) == 0, _lib.last_error()
        assert L.sfft_sync(plan) == 0, _lib.last_error()
        out = []
        for s in range(m):
            c = int(cnt[s])
            gi, gv = idx[s, :c].cpu().numpy(), val[s, :c].cpu().numpy()
            o = np.argsort(gi)
            out.append((gi[o], gv[o]))
        return out

    order = [s % len(sig) for s in range(batch)]
    many = run(order)
    alone = [run([w])[0] for w in range(len(sig))]
    L.sfft_free_plan(plan)
    for s, w in enumerate(order):
        np.testing.assert_array_equal(many[s][0], alone[w][0])
        scale = max(1.0, float(np.max(np.abs(alone[w][1]), initial=0.0)))
        assert float(np.max(np.abs(many[s][1] - alone[w][1]), initial=0.0)) <= 1e-11 * scale
    op = O.OraclePlan(n, k, 2)
    oi, ov = op.exec(sig[0].astype(np.complex128), seed=100)
    np.testing.assert_array_equal(many[0][0], oi)
    scale = max(1.0, float(np.max(np.abs(ov), initial=0.0)))
    assert float(np.max(np.abs(many[0][1] - ov), initial=0.0)) <= 1e-10 * scale
