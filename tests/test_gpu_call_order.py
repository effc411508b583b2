"""Calls that follow one another without a wait in between: what a batch still
reads or writes is not touched by the next call.  Every result equals that of
the same calls with the device idle in between."""
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


class Calls:
    def __init__(self, env, version, n, k, batch):
        torch, _lib, self.L, self.O = env
        from sfft_gb300 import signals
        self.torch, self.last_error, self.version, self.n, self.m = torch, _lib.last_error, version, n, batch
        self.plan = self.L.sfft_make_plan_ex(n, k, version - 1, 0, ctypes.byref(_lib.Options(0, -1, batch)))
        assert self.plan, _lib.last_error()
        self.cap = self.L.sfft_output_capacity(self.plan)
        sig = [signals.make_signal(n, k, 40 + s, snr_db=40.0 if version == 2 else None)[0] for s in range(batch + 1)]
        self.x = torch.from_numpy(np.stack(sig[:batch])).cuda()
        self.y = torch.from_numpy(sig[batch][None]).cuda()
        self.idx = torch.empty((batch, self.cap), dtype=torch.int32, device="cuda")
        self.val = torch.empty((batch, self.cap), dtype=torch.complex128, device="cuda")
        self.cnt = torch.zeros(batch, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()

    def batch(self, x, stream=None):
        pin = (ctypes.c_void_p * self.m)(*[v.data_ptr() for v in x])
        seeds = (ctypes.c_uint * self.m)(*range(5, 5 + self.m))
        assert self.L.sfft_exec_batch_ex(self.plan, self.m, pin, 0, seeds, self.idx.data_ptr(), self.val.data_ptr(),
                                         self.cnt.data_ptr(), self.cap, stream) == 0, self.last_error()

    def dense(self, y, out):
        self.O.seed_libc(9)
        self.L.sfft_exec_many(self.plan, 1, (ctypes.c_void_p * 1)(y.data_ptr()), (ctypes.c_void_p * 1)(out.data_ptr()))
        assert self.last_error() == ""
        return out.cpu().numpy().copy()

    def lists(self):
        self.torch.cuda.synchronize()
        out = []
        for s in range(self.m):
            c = int(self.cnt[s])
            i, v = self.idx[s, :c].cpu().numpy(), self.val[s, :c].cpu().numpy()
            o = np.argsort(i, kind="stable")
            out.append((i[o], v[o]))
        return out

    def same(self, a, b):
        assert len(a) == len(b)
        for (i, v), (j, w) in zip(a, b):
            np.testing.assert_array_equal(i, j)
            self.close(v, w)

    def close(self, v, w):
        if self.version < 3:
            np.testing.assert_array_equal(v, w)
        else:  # FP64 atomics in any order
            np.testing.assert_allclose(v, w, rtol=0, atol=1e-11)


SHAPES = [(1, 1 << 18, 50, 16), (2, 1 << 20, 50, 16), (3, 1 << 18, 100, 16)]


@pytest.mark.parametrize("version,n,k,batch", SHAPES)
def test_dense_output_over_a_queued_batchs_input(env, version, n, k, batch):
    """The dense call writes the buffer that the batch, queued on the plan's
    stream, reads last."""
    c = Calls(env, version, n, k, batch)
    c.batch(c.x)
    want = c.lists()
    out = c.torch.full_like(c.y[0], 3)
    dense = c.dense(c.y[0], out)
    for s in (batch - 1, 0):
        x = c.x.clone()
        c.torch.cuda.synchronize()
        c.batch(x)
        c.close(c.dense(c.y[0], x[s]), dense)
        c.same(c.lists(), want)
    c.L.sfft_free_plan(c.plan)


@pytest.mark.parametrize("version,n,k,batch", SHAPES)
def test_calls_after_a_batch_on_another_stream(env, version, n, k, batch):
    """The plan's workspace is the batch's until it ran."""
    c = Calls(env, version, n, k, batch)
    c.batch(c.x)
    want = c.lists()
    dense = c.dense(c.y[0], c.torch.full_like(c.y[0], 3))
    host = c.y[0].cpu().numpy()
    st = c.torch.cuda.Stream()
    hi, hv = np.empty(c.cap, np.int32), np.empty(c.cap, np.complex128)
    for sparse in (False, True):
        c.cnt.zero_()
        c.torch.cuda.synchronize()
        c.batch(c.x, st.cuda_stream)
        if sparse:
            c.O.seed_libc(9)
            m = c.L.sfft_exec_sparse(c.plan, host.ctypes.data, hi.ctypes.data, hv.ctypes.data, c.cap)
            assert m >= 0, c.last_error()
            got = np.zeros_like(dense)
            got[hi[:m]] = hv[:m]
            c.close(got, dense)
        else:
            c.close(c.dense(c.y[0], c.torch.full_like(c.y[0], 3)), dense)
        c.same(c.lists(), want)
    c.L.sfft_free_plan(c.plan)
