"""Vote counts and hits of the location loops (computefourier-1.0-2.0.cc:91-184)
restated on the run's own selected buckets, permutations and comb residues,
at shapes on both sides of the voting kernels' rules: counting by comb
residue or by candidate, ranges wider and narrower than the comb width,
bitmaps in and beyond shared memory."""
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


# (version, n, k, B_loc, W, comb samplings, location loops, threshold)
SHAPES = [
    (1, 1 << 16, 50, 1024, 64, 1, 5, 4),
    (1, 1 << 14, 3, 16, 64, 1, 2, 1),          # ranges of 1024 positions, threshold 1
    (1, 1 << 22, 100, 131072, 64, 1, 3, 2),    # bitmaps beyond shared memory
    (2, 1 << 16, 50, 1024, 8192, 6, 4, 2),     # 8 repetitions a residue: by candidate
    (2, 1 << 18, 20, 512, 128, 1, 4, 3),       # by residue, ranges of 512 positions: four per residue
    (2, 1 << 20, 10, 2048, 1024, 2, 7, 3),     # by residue, ranges narrower than the comb width
    (2, 1 << 10, 1, 16, 512, 1, 3, 2),         # two repetitions a residue
    (2, 1 << 20, 500, 8192, 2048, 1, 4, 3),    # 1000 selected buckets
]


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_votes_match_restatement(env, shape, prec):
    torch, _lib, L = env
    from sfft_gb300 import signals
    version, n, k, B, W, cl, loops, thresh = shape
    root = math.sqrt(n * k / math.log2(n))
    prm = _lib.Params((B + 0.5) * 1.001 / root, (B + 0.5) * 1.001 / root, W * B / n * 1.0001, loops, 2, thresh, cl, 1e-6, 1e-6)
    f = (ctypes.c_long * 11)()
    assert L.sfft_describe_plan_params(n, k, version - 1, ctypes.byref(prm), f, 11) == 11, _lib.last_error()
    assert f[0] == B and (version == 1 or (f[3], f[4]) == (W, cl))
    opt = _lib.Options(_lib.SFFT_PREC_FP32 if prec == "fp32" else _lib.SFFT_PREC_FP64, -1, 2)
    plan = L.sfft_make_plan_params(n, k, version - 1, ctypes.byref(prm), ctypes.byref(opt))
    assert plan, _lib.last_error()
    xs = [signals.make_signal_torch(n, k, 5 + s, snr_db=20.0)[0] for s in range(2)]
    for voted in ((False,) if version == 1 else (False, True)):
        if version == 2:
            assert L.sfft_plan_v2_voted(plan, int(voted)) == 0, _lib.last_error()
        cap = L.sfft_output_capacity(plan)
        idx = torch.empty((2, cap), dtype=torch.int32, device="cuda")
        val = torch.empty((2, cap), dtype=torch.complex64 if prec == "fp32" else torch.complex128, device="cuda")
        cnt = torch.zeros(2, dtype=torch.int32, device="cuda")
        seeds = (ctypes.c_uint * 2)(4, 5)
        torch.cuda.synchronize()
        for order in ((0, 1), (1, 0)):  # slot 0 sees one signal after the other: earlier counts must not show
            pin = (ctypes.c_void_p * 2)(*[xs[o].data_ptr() for o in order])
            assert L.sfft_exec_batch_ex(plan, 2, pin, 0, seeds, idx.data_ptr(), val.data_ptr(), cnt.data_ptr(), cap,
                                        None) == 0, _lib.last_error()
            assert L.sfft_sync(plan) == 0, _lib.last_error()

        def fetch(what, count):
            buf = np.empty(count, dtype=np.int32)
            c = L.sfft_debug_fetch(plan, what, buf.ctypes.data, count)
            assert c >= 0
            return buf[:c].astype(np.int64)

        a = fetch(0, 2 * (loops + 2))[:loops]
        J = fetch(1, (loops + 2) * 2 * k).reshape(loops + 2, -1)[:loops]
        q = n // B
        want = np.zeros(n, dtype=np.int64)
        for j in range(loops):
            p = (J[j][:, None] * q - q // 2 + np.arange(q)[None, :]) % n
            want[(p * a[j]) % n] += 1
        if version == 2:
            comb = np.zeros(W, dtype=bool)
            comb[fetch(4, W)] = True
            want[~comb[np.arange(n) % W]] = 0
        np.testing.assert_array_equal(fetch(2, n), want)
        if version == 1 or voted:
            hits = np.nonzero(want >= thresh)[0]
            assert int(cnt[0]) == hits.size
            np.testing.assert_array_equal(np.sort(idx[0, :hits.size].cpu().numpy()), hits)
    L.sfft_free_plan(plan)
