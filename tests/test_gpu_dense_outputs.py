"""Dense outputs cleared beside the transform: device outputs that hold other
data before, in-place calls and outputs that overlap another signal's input
(cleared after the transform), and mixtures of host and device buffers give
what separate host buffers give."""
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


@pytest.mark.parametrize("version,n,k", [(1, 1 << 13, 50), (2, 1 << 16, 50), (3, 1 << 17, 100), (3, 1 << 14, 9)])
def test_dense_outputs_in_any_buffer(env, version, n, k):
    torch, _lib, L, O = env
    from sfft_gb300 import signals
    m = 5
    sig = [signals.make_signal(n, k, 70 + s, snr_db=40.0 if version == 2 else None)[0] for s in range(m)]
    plan = L.sfft_make_plan_ex(n, k, version - 1, 0, ctypes.byref(_lib.Options(0, -1, 4)))   # two launches: 4 + 1
    assert plan, _lib.last_error()

    def call(ins, outs):
        O.seed_libc(31)
        torch.cuda.synchronize()
        L.sfft_exec_many(plan, m, (ctypes.c_void_p * m)(*ins), (ctypes.c_void_p * m)(*outs))
        assert _lib.last_error() == ""

    want = np.full((m, n), 7 + 7j)
    call([x.ctypes.data for x in sig], [w.ctypes.data for w in want])

    def close(got):
        if version < 3:
            np.testing.assert_array_equal(got, want)
        else:
            np.testing.assert_array_equal(got != 0, want != 0)
            assert np.max(np.abs(got - want)) <= 1e-11

    xd = torch.from_numpy(np.stack(sig)).cuda()
    od = torch.full((m, n), 3 + 4j, dtype=torch.complex128, device="cuda")
    call([x.data_ptr() for x in xd], [o.data_ptr() for o in od])
    close(od.cpu().numpy())
    both = xd.clone()                                     # in place
    call([x.data_ptr() for x in both], [x.data_ptr() for x in both])
    close(both.cpu().numpy())
    # one buffer, each output half a signal before its own input: within one launch an output also
    # covers the end of the input before it, which is read by then
    buf = torch.zeros(2 * m * n + n, dtype=torch.complex128, device="cuda")
    at = [(2 * s + 1) * n for s in range(m)]
    for a, x in zip(at, xd):
        buf[a:a + n] = x
    call([buf[a:].data_ptr() for a in at], [buf[a - n // 2:].data_ptr() for a in at])
    close(np.stack([buf[a - n // 2:a + n - n // 2].cpu().numpy() for a in at]))
    host = np.full((m, n), 1 - 1j)                        # mixed
    od.fill_(5)
    call([sig[s].ctypes.data if s & 1 else xd[s].data_ptr() for s in range(m)],
         [host[s].ctypes.data if s < 3 else od[s].data_ptr() for s in range(m)])
    close(np.concatenate([host[:3], od[3:].cpu().numpy()]))
    L.sfft_free_plan(plan)
