"""Signals so large that an intermediate overflows before the values do."""
import ctypes

import numpy as np
import pytest

from test_gpu_estimation import restated_estimates
from test_gpu_estimation_values import K, N, _run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sfft_gb300 import _lib, build
    build.build()
    return torch, _lib, _lib.load()


@pytest.mark.parametrize("scale", [1.5 * 2.0 ** 126, 1.25 * 2.0 ** 127, 1.75 * 2.0 ** 127, 2.0 ** 128])
def test_fp64_medians_where_the_fp32_scale_overflows(env, scale):
    """Around 2^127 the FP32 copies of the bucket values are finite and the sums
    of their magnitudes are not: the error bound is infinite and proves no
    median.  A clean signal: its loops agree to more digits than FP32 has."""
    from sfft_gb300 import signals
    x, _, _ = signals.make_signal(N, K, 17)
    gi, gv, (pp, xs, ai, comb, wl, we) = _run(env, x * scale, True)
    rf, rv = restated_estimates(N, pp, xs, ai, comb, wl, we)
    o = np.argsort(rf)
    np.testing.assert_array_equal(gi, rf[o])
    np.testing.assert_array_equal(gv, rv[o])
