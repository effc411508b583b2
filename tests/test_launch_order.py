"""What the library's host code launches, on the CPU: its sources run over a
CUDA runtime that keeps, for every operation, what is ordered before it
(fake_cuda/runtime.cc).  Work that a program queued on the plan's stream, or
an asynchronous batch on a stream of its own, comes before what a later call
does to the same buffers; a transform never runs with a buffer missing."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from sfft_gb300 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))
SHAPES = [(0, 1 << 13, 50), (1, 1 << 14, 50), (2, 1 << 13, 16)]   # version, n, k


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    src = [os.path.join(HERE, "fake_cuda", "runtime.cc")]
    src += [os.path.join(build.CSRC, f) for f in ("api.cc", "host_plan.cc", "tune.cc", "serve.cc")]
    subprocess.check_call(["g++", "-O1", "-fPIC", "-std=c++17", "-fopenmp", "-shared", "-Wl,-Bsymbolic", "-o", so] + src +
                          ["-I" + os.path.join(build._cuda_home(), "include"), "-I" + os.path.join(build.ROOT, "include"),
                           "-I" + build.CSRC])
    L = ctypes.CDLL(so)
    vp, cl = ctypes.c_void_p, ctypes.c_long
    for f in (L.sfft_make_plan_ex, L.sfft_plan_stream):
        f.restype = vp
    for f in (L.sfft_output_capacity, L.sfft_exec_sparse, L.sfft_plan_footprint, L.sfft_server_plan_bytes):
        f.restype = cl
    L.sfft_last_error.restype = L.fake_name.restype = ctypes.c_char_p
    return L


class Plan:
    def __init__(self, L, version, n, k, max_batch=4, prec=0):
        self.L, self.n = L, n
        self.p = vp(L.sfft_make_plan_ex(n, k, version, 0, ctypes.byref(_lib.Options(prec, -1, max_batch))))
        assert self.p, L.sfft_last_error()
        self.cap = L.sfft_output_capacity(self.p)
        self.bufs = []

    def device(self, nbytes):
        p = ctypes.c_void_p()
        assert self.L.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(nbytes)) == 0
        ctypes.memset(p, 0, nbytes)
        self.bufs.append(p)
        return p

    def signals(self, m=1):
        return (ctypes.c_void_p * m)(*[self.device(16 * self.n).value for _ in range(m)])

    def batch(self, m=2, stream=None):
        """An asynchronous batch; its transforms in the log."""
        at = self.L.fake_ops()
        r = self.L.sfft_exec_batch_ex(self.p, m, self.signals(m), 0, None, self.device(4 * m * self.cap),
                                      self.device(16 * m * self.cap), self.device(4 * m), ctypes.c_long(self.cap),
                                      ctypes.c_void_p(stream))
        return r, self.ops(at, "transform")

    def ops(self, at, *names):
        return [i for i in range(at, self.L.fake_ops()) if self.L.fake_name(i).decode() in names]

    def free(self):
        self.L.sfft_free_plan(self.p)
        for b in self.bufs:
            self.L.cudaFree(b)


vp = ctypes.c_void_p


@pytest.fixture(params=SHAPES, ids=["v1", "v2", "v3"])
def plan(fake, request):
    p = Plan(fake, *request.param)
    yield p
    p.free()


@pytest.mark.parametrize("m", [1, 5])   # one launch, and two
def test_outputs_are_cleared_after_work_on_the_plans_stream(fake, plan, m):
    """A batch with a NULL stream, or a copy queued on sfft_plan_stream, may
    still read the buffers that a dense call then writes."""
    before = plan.batch()[1]
    before.append(fake.fake_ops())
    fake.fake_work(vp(fake.sfft_plan_stream(plan.p)))
    at = fake.fake_ops()
    ins, outs = plan.signals(m), plan.signals(m)
    fake.sfft_exec_many(plan.p, m, ins, outs)
    assert fake.sfft_last_error() == b""
    assert plan.ops(at, "clear")
    for c in plan.ops(at, "clear", "setup", "transform", "scatter"):
        assert all(fake.fake_before(b, c) for b in before)


def test_only_the_transforms_of_dense_calls_go_first(fake, plan):
    """The plan's stream, on which batches run, has no priority over the
    streams of the program; a dense call's transform has one over the clearing
    of its outputs."""
    assert fake.fake_priority(vp(fake.sfft_plan_stream(plan.p))) == 0
    at = fake.fake_ops()
    plan.batch(2)
    assert all(fake.fake_op_priority(i) == 0 for i in range(at, fake.fake_ops()))
    fake.cudaDeviceSynchronize()
    at = fake.fake_ops()
    fake.sfft_exec_many(plan.p, 1, plan.signals(1), plan.signals(1))
    assert all(fake.fake_op_priority(i) < 0 for i in plan.ops(at, "transform"))
    assert all(fake.fake_op_priority(i) == 0 for i in plan.ops(at, "clear"))


def test_clearing_does_not_wait_for_the_calls_own_input_copies(fake, plan):
    """On an idle plan the outputs are cleared beside the copies of host inputs
    (v1 / v2; v3 clears after its filters)."""
    x = np.zeros(plan.n, dtype=np.complex128)
    at = fake.fake_ops()
    fake.sfft_exec_many(plan.p, 1, (vp * 1)(x.ctypes.data), plan.signals(1))
    copy, clear = plan.ops(at, "to device")[0], plan.ops(at, "clear")[0]
    if plan.p and ctypes.cast(plan.p, ctypes.POINTER(_lib.Plan)).contents.version != 2:
        assert not fake.fake_before(copy, clear)


def test_nothing_is_written_after_a_failed_call_returned(fake, plan):
    at = fake.fake_ops()
    fake.fake_fail(b"scatter")
    fake.sfft_exec_many(plan.p, 1, plan.signals(1), plan.signals(1))
    fake.fake_fail(b"")
    assert fake.sfft_last_error() != b""
    clears = plan.ops(at, "clear")
    assert clears and all(fake.fake_waited(c) for c in clears)


def _dense(p):
    p.L.sfft_exec_many(p.p, 1, p.signals(1), p.signals(1))


def _dense_host(p):
    x = np.zeros((3, p.n), dtype=np.complex128)
    a = (vp * 3)(*[v.ctypes.data for v in x])
    p.L.sfft_exec_many(p.p, 3, a, a)


def _sparse(p):
    assert p.L.sfft_exec_sparse(p.p, p.device(16 * p.n), p.device(4 * p.cap), p.device(16 * p.cap),
                                ctypes.c_long(p.cap)) == 0


def _many_sparse(p):
    cnt = (ctypes.c_int * 2)()
    assert p.L.sfft_exec_many_sparse(p.p, 2, p.signals(2), p.device(8 * p.cap), p.device(32 * p.cap), cnt,
                                     ctypes.c_long(p.cap)) == 0


@pytest.mark.parametrize("call", [_dense, _dense_host, _sparse, _many_sparse])
def test_calls_come_after_batches_on_other_streams(fake, plan, call):
    """The plan's draws, buckets and lists belong to the batch until it ran."""
    st = vp()
    assert fake.cudaStreamCreateWithFlags(ctypes.byref(st), 1) == 0
    plan.batch(4)                                   # the workspace has its size: nothing below waits for an allocation
    fake.cudaDeviceSynchronize()
    r, batch = plan.batch(2, st.value)
    assert r == 0 and batch
    at = fake.fake_ops()
    call(plan)
    assert fake.sfft_last_error() == b""
    later = plan.ops(at, "setup", "transform")
    assert later
    for i in later:
        assert all(fake.fake_before(b, i) for b in batch)


def test_calls_come_after_the_part_of_a_failed_batch(fake, plan):
    st = vp()
    assert fake.cudaStreamCreateWithFlags(ctypes.byref(st), 1) == 0
    plan.batch(4)
    fake.cudaDeviceSynchronize()
    fake.fake_fail_after(b"transform", 1)           # five signals are two launches of at most four
    r, batch = plan.batch(5, st.value)
    fake.fake_fail(b"")
    assert r == -1 and len(batch) == 1
    at = fake.fake_ops()
    _dense(plan)
    assert fake.fake_before(batch[0], plan.ops(at, "setup")[0])


@pytest.mark.parametrize("call", [_dense, _dense_host, _sparse, _many_sparse])
@pytest.mark.parametrize("limit", [1 << 14, 1 << 18, 1 << 20, 1 << 22])
def test_buffers_are_whole_after_a_batch_that_did_not_fit(fake, plan, call, limit):
    """Growing the workspace for a large batch fails at one of its buffers; the
    calls after that have all of them again (or say that they have not)."""
    fake.fake_limit(ctypes.c_size_t(limit))
    at = fake.fake_ops()
    ins, room = plan.signals(1)[0] if limit >= 16 * plan.n else None, vp(64)
    big = (vp * 4)(ins, ins, ins, ins)
    fake.sfft_exec_batch_ex(plan.p, 4, big, 0, None, room, room, room, ctypes.c_long(plan.cap), None)
    failed = not plan.ops(at, "transform")
    fake.fake_limit(ctypes.c_size_t(-1))
    at = fake.fake_ops()
    call(plan)
    done = plan.ops(at, "transform")
    assert done and all(fake.fake_whole(i) for i in done)
    assert failed or limit > 1 << 14   # the smallest limit is below every workspace


@pytest.mark.parametrize("version,n,k,prec", [
    (2, 1 << 14, 8, 0), (2, 1 << 14, 9, 0), (2, 1 << 15, 31, 0), (2, 1 << 16, 50, 0), (2, 1 << 14, 127, 0),
    (2, 1 << 16, 1000, 0), (0, 1 << 13, 50, 0), (0, 1 << 16, 50, 1), (1, 1 << 14, 50, 0), (1, 1 << 16, 50, 0),
    (1, 1 << 16, 50, 1)])
@pytest.mark.parametrize("m", [1, 32])
def test_the_servers_estimate_covers_a_plans_workspace(fake, version, n, k, prec, m):
    """A server admits a plan by its estimate for max_batch signals: it is no
    less than what such a batch makes the plan hold, but for a twentieth, and
    not several times more."""
    p = Plan(fake, version, n, k, m, prec)
    r, done = p.batch(m)
    assert r == 0 and done
    held, estimate = fake.sfft_plan_footprint(p.p), fake.sfft_server_plan_bytes(n, k, version, prec, m)
    p.free()
    print(version, n, k, prec, m, held, estimate, estimate / held)
    assert 0.95 * held <= estimate <= 4 * held


@pytest.mark.parametrize("call", [_dense, _dense_host, _sparse, _many_sparse])
def test_every_copy_comes_after_work_on_the_plans_stream(fake, plan, call):
    """That work may still write a call's inputs or read its outputs."""
    call(plan)                                      # the staging has its size
    fake.cudaDeviceSynchronize()
    work = fake.fake_ops()
    fake.fake_work(vp(fake.sfft_plan_stream(plan.p)))
    call(plan)
    assert fake.sfft_last_error() == b""
    for i in range(work + 1, fake.fake_ops()):
        assert fake.fake_before(work, i), fake.fake_name(i)
