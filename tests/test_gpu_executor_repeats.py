"""The persistent executor's estimation copies bucket values that other blocks
of the same launch stored.  Runs on two sets of signals in turn, so that values
of the run before would show, equal the graph's bit for bit every time."""
import numpy as np
import pytest

from test_gpu_mixed import FP32, V2, _create_tuned, _result, _run, _uneven_shapes

pytestmark = pytest.mark.gpu


def test_executor_in_turn_on_two_sets_of_signals():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sfft_gb300 import _lib, build, signals
    build.build()
    L = _lib.load()
    sigs = [(n, k, V2, FP32) for n, k in _uneven_shapes(16, seed0=40)]
    sets = [[signals.make_signal_torch(n, k, base + i, snr_db=40.0)[0] for i, (n, k, _, _) in enumerate(sigs)]
            for base in (300, 600)]
    seeds = [[s + i for i in range(len(sigs))] for s in (5, 50)]
    torch.cuda.synchronize()
    mg = _create_tuned(L, _lib, sigs, False)
    want = []
    for xs, sd in zip(sets, seeds):
        _run(L, _lib, mg, xs, sd)
        want.append([_result(torch, _lib, L, mg, s) for s in range(len(sigs))])
    L.sfft_mixed_destroy(mg)
    mp = _create_tuned(L, _lib, sigs, True)
    for turn in range(20):
        a = turn & 1
        _run(L, _lib, mp, sets[a], seeds[a])
        for s in range(len(sigs)):
            i, v = _result(torch, _lib, L, mp, s)
            np.testing.assert_array_equal(i, want[a][s][0])
            np.testing.assert_array_equal(v, want[a][s][1])
    L.sfft_mixed_destroy(mp)
