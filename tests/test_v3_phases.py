"""v3's phases, angles, square roots and reciprocals (csrc/phase.cuh), compiled
for the host, against 113-bit arithmetic.

Bounds, with u = 2^-53 = 1.11e-16.  cis: the table's value and the last sum are
rounded to u / 2 each for components up to 1, and a correction below 0.0031
adds three roundings of that: 1.02 u.  cis_step: the same, and half a unit of
2^-64 turn more for each of three fractions: within 0.01 u.  angle_of: the last
sum, up to pi, is rounded to 2 u; the turned vector carries the rounding of the
table and of two products, at most 2 u; 4.1 u in all.  sqrt_of, recip_of: the
last sum is the only rounding, u of the value, after an exact remainder."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from sfft_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))
U = 2.0 ** -53
COUNT = 100000


@pytest.fixture(scope="module")
def phase(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("phase") / "libphase.so")
    import platform
    quad = ["-lquadmath"] if platform.machine() == "x86_64" else []
    subprocess.check_call(["g++", "-O2", "-fPIC", "-std=gnu++17", "-ffp-contract=off", "-shared", "-I" + build.CSRC, "-o", so,
                           os.path.join(HERE, "phase_host.cc")] + quad)
    L = ctypes.CDLL(so)
    d, i = ctypes.c_double, ctypes.c_int
    for f, args in ((L.phase_cis, [d]), (L.phase_step, [d, i, d]), (L.phase_angle, [d, d]), (L.phase_sqrt, [d]),
                    (L.phase_recip, [d])):
        f.restype, f.argtypes = d, args
    L.phase_step_value.argtypes = [d, i, d, ctypes.POINTER(d), ctypes.POINTER(d)]
    L.phase_table()
    return L


def _sizes(rng, lo, hi):
    return np.exp(rng.uniform(np.log(lo), np.log(hi), COUNT)) * rng.choice([-1.0, 1.0], COUNT)


def test_phases(phase):
    rng = np.random.default_rng(1)
    special = [0.0, -0.0, 1e-300, np.pi, -np.pi / 2, 2.0 ** 53, 2.0 ** 63, np.pi * 2.0 ** 40]
    assert max(phase.phase_cis(a) for a in [*special, *_sizes(rng, 1e-3, 1e19)]) <= 1.02 * U


def test_phases_of_steps(phase):
    rng = np.random.default_rng(2)
    a, b, k = _sizes(rng, 1.0, 1e10), _sizes(rng, 1.0, 1e10), rng.integers(0, 60000, COUNT)
    assert max(phase.phase_step(x, int(i), y) for x, i, y in zip(a, k, b)) <= 1.03 * U


def test_angles(phase):
    rng = np.random.default_rng(3)
    y, x = _sizes(rng, 1e-9, 1e9), _sizes(rng, 1e-9, 1e9)
    axes = [(0.0, 1.0), (0.0, -1.0), (1.0, 0.0), (-1.0, 0.0), (1.0, 1.0), (-1e-5, -1.0), (1e-200, 1e-300), (0.0, 0.0)]
    assert max(phase.phase_angle(p, q) for p, q in [*axes, *zip(y, x)]) <= 4.1 * U


def test_square_roots_and_reciprocals(phase):
    rng = np.random.default_rng(4)
    a = np.abs(_sizes(rng, 1e-18, 1e18))
    assert max(phase.phase_sqrt(v) for v in [1e-200, 1e200, 4.0, *a]) <= 1.001 * U
    assert max(phase.phase_recip(v) for v in [1e-200, 1e200, 4.0, *a]) <= 1.001 * U


def test_steps_follow_the_reference_s_running_product(phase):
    """The permuted filter's phases (computefourier-3.0.cc:66-87 multiplies them
    up one by one): at n = 2^24, k = 1000 the product's own rounding drifts by
    less than 1e-12 from the phases formed directly."""
    n, count = 1 << 24, 2945
    ig, ai, b = 9876543, 7654321, 1234567
    a0, a1 = 2 * np.pi * ig * b / n, 2 * np.pi * ai * b / n
    sh, st = complex(np.cos(a0), np.sin(a0)), complex(np.cos(a1), np.sin(a1))
    re, im = ctypes.c_double(), ctypes.c_double()
    worst = 0.0
    for i in range(count):
        phase.phase_step_value(a0, i, a1, ctypes.byref(re), ctypes.byref(im))
        worst = max(worst, abs(sh - complex(re.value, im.value)))
        sh *= st
    assert worst < 1e-12
