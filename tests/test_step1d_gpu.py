"""1D solves run several whole RK4 steps per launch, the points in registers
(overlapping windows of 32, 64 or 128 points).  The same bits as the gather
kernels, and in FP64 / FP32 as the oracle, for both methods and every
boundary code: on grids of one window, of one window and one point, with the
end point first or last in a window, on both sides of every line of the
dispatch rule, for step counts that leave a remainder launch; and when the
state has been left in the other buffer and the knob then changes the form."""
import numpy as np
import pytest

import oracle
from nlsemagic_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# windows store 128 - 8 m (CD) or 128 - 16 m points in FP32 and mixed (m = 10
# and 6 here), 8, 16 and 56 or 16 and 48 in FP64
SMALL = [4, 5, 8, 16, 17, 31, 32, 33, 34, 48, 49, 50, 65, 97, 127, 128, 129, 161, 193]
LINES = [1216, 1217, 8192, 8193, 32768, 32769, 65536, 65537, 98305, 524289]


def _case(n):
    h = 0.1
    x = -n * h / 2 + h * np.arange(n)
    U = (np.exp(-x * x / 40.0) * np.exp(0.4j * x) + 0.3 * np.cos(0.9 * x)).astype(complex)
    return U, 0.2 * np.cos(0.3 * x), h


def bits_equal(a, b):  # NaNs alike whatever their payload (the CPU's differs)
    a = np.ascontiguousarray(a, dtype=np.complex128).view(np.float64)
    b = np.ascontiguousarray(b, dtype=np.complex128).view(np.float64)
    return np.array_equal(a, b, equal_nan=True)


def _run(n, BC, method, prec, steps, gather=False):
    import nlsemagic_gb300 as ng
    U, V, h = _case(n)
    k = 0.5 * W.linear_stability_k(1, method, h, 1.0)
    flags = ng.FLAG_MSD_GUARD | (ng.FLAG_GATHER if gather else 0)
    from nlsemagic_gb300 import autotune
    old = autotune.get_knob("small1d.max_points")
    try:
        autotune.set_knob("small1d.max_points", 0)
        return ng.take_steps(U, V, -1.0, 1.0, h * h, BC, steps, k, method=method, precision=prec,
                             flags=flags)
    finally:
        autotune.set_knob("small1d.max_points", old)


@pytest.mark.parametrize("prec", [1, 2, 3])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3, 4])
def test_step1d_same_bits_small(gpu_lib, BC, method, prec):
    for n in SMALL + ([3] if BC != 4 else []):
        got = _run(n, BC, method, prec, 13)
        assert bits_equal(got, _run(n, BC, method, prec, 13, gather=True)), n
        if prec != 3:
            U, V, h = _case(n)
            k = 0.5 * W.linear_stability_k(1, method, h, 1.0)
            want = oracle.take_steps(U, V, -1.0, 1.0, h * h, BC, 13, k, method=method,
                                     precision=prec, flags=oracle.MSD_GUARD)
            assert bits_equal(got, want), n


@pytest.mark.parametrize("prec", [1, 2, 3])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [2, 4])
def test_step1d_same_bits_at_the_lines(gpu_lib, BC, method, prec):
    for n in LINES:
        got = _run(n, BC, method, prec, 11)
        assert bits_equal(got, _run(n, BC, method, prec, 11, gather=True)), n


@pytest.mark.parametrize("prec", [1, 2, 3])
def test_step1d_then_other_forms(gpu_lib, prec):
    # odd numbers of launches between runs in the gather form, whose graphs
    # hold the addresses of the buffer the state is in
    import nlsemagic_gb300 as ng
    from nlsemagic_gb300 import autotune
    n = 700
    U, V, h = _case(n)
    k = 0.5 * W.linear_stability_k(1, 2, h, 1.0)
    old = {key: autotune.get_knob(key) for key in ("seg1d", "small1d.max_points")}

    def run(forms):
        with ng.Solver((n,), method=2, precision=prec, BC=2, s=-1.0, a=1.0, h2=h * h, k=k) as sv:
            sv.upload(U, V)
            for seg, small, steps in forms:
                autotune.set_knob("seg1d", seg)
                autotune.set_knob("small1d.max_points", small)
                sv.run(steps)
            return sv.download()

    try:
        steps = (17, 3, 9, 1, 16, 2)
        a = run([(0, 0, m) for m in steps])
        b = run([(t % 2, 2048 * (t // 2 % 2), m) for t, m in enumerate(steps)])
    finally:
        for key, v in old.items():
            autotune.set_knob(key, v)
    assert bits_equal(a, b)
