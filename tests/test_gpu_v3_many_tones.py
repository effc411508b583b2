"""v3 with thousands of tones: combs of 2^15 to 2^17 (several passes of an
estimate over the buckets, tiles of one column), 8192 Gaussian buckets, and
more than 1024 tones in one block of the peeling clusters (8 blocks for a
batch, 16 alone), whose rest goes through global memory.  Every slot against
the oracle's spectrum, with the 1e-10 of the parity tests (entries below that
come from the rounding of large ones)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 1 << 22


@pytest.mark.parametrize("k,batch", [(4100, 1), (4100, 6), (12000, 1), (12000, 6), (16383, 1), (16383, 6)])
def test_v3_many_tones(oracle_lib, k, batch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sfft_gb300 import _lib, build, signals
    build.build()
    L = _lib.load()
    x, _, _ = signals.make_signal(N, k, 60)
    oi, ov = oracle_lib.OraclePlan(N, k, 2).exec(x, seed=100)
    plan = L.sfft_make_plan_ex(N, k, 2, 0, ctypes.byref(_lib.Options(0, -1, batch)))
    assert plan, _lib.last_error()
    cap = L.sfft_output_capacity(plan)
    xd = torch.from_numpy(x).cuda()
    idx = torch.empty((batch, cap), dtype=torch.int32, device="cuda")
    val = torch.empty((batch, cap), dtype=torch.complex128, device="cuda")
    cnt = torch.zeros(batch, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert L.sfft_exec_batch_ex(plan, batch, (ctypes.c_void_p * batch)(*[xd.data_ptr()] * batch), 0,
                                (ctypes.c_uint * batch)(*[100] * batch), idx.data_ptr(), val.data_ptr(), cnt.data_ptr(),
                                cap, None) == 0, _lib.last_error()
    assert L.sfft_sync(plan) == 0, _lib.last_error()
    L.sfft_free_plan(plan)
    want = np.zeros(N, dtype=np.complex128)
    want[oi] = ov
    scale = max(1.0, float(np.max(np.abs(ov))))
    for s in range(batch):
        c = int(cnt[s])
        gi, gv = idx[s, :c].cpu().numpy(), val[s, :c].cpu().numpy()
        assert len(np.unique(gi)) == c
        got = np.zeros(N, dtype=np.complex128)
        got[gi] = gv
        assert np.max(np.abs(got - want)) <= 1e-10 * scale
