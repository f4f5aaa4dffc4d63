"""2D and 3D stages by point: every point with two cells to each face in one
numbering, every point next to a face in a thread that also does the face
points it is the MSD neighbour of.  FP64, and FP32 in 3D: the oracle's bits, for
both methods and boundary codes 1-3, on grids with no deep point, one, one layer
of shell points per axis (3 cells) or two.  Contracted FP64 (the wide form): within
1e-12 of the oracle.  Mixed 3D: the bits of the streaming kernels."""
import numpy as np
import pytest

import oracle
from nlsemagic_gb300 import workloads as W

pytestmark = pytest.mark.gpu

GRIDS2 = [(3, 3), (3, 9), (9, 3), (4, 4), (5, 5), (6, 5), (13, 41), (66, 35), (130, 67)]
GRIDS3 = [(3, 3, 3), (3, 5, 4), (5, 3, 6), (6, 5, 3), (4, 4, 4), (5, 5, 5), (5, 6, 7), (9, 4, 13),
          (17, 12, 11), (33, 21, 18)]
TOL_FMA = 1e-12  # relative L2, the contracted class's contract


def bits_equal(a, b):
    a = np.ascontiguousarray(a, dtype=np.complex128).view(np.float64)
    b = np.ascontiguousarray(b, dtype=np.complex128).view(np.float64)
    return np.array_equal(a, b, equal_nan=True)


def _case(shape, method):
    h = 0.25
    X = np.meshgrid(*[-n * h / 2 + h * np.arange(n) for n in shape], indexing="ij")
    U = (0.8 + 0.2 * np.cos(0.7 * X[0]) * np.cos(0.5 * X[1])) * np.exp(0.3j * X[0] - 0.2j * X[-1])
    V = 0.1 * np.cos(0.4 * X[0] + 0.3 * X[1])
    return U, V, h, 0.5 * W.linear_stability_k(len(shape), method, h, 1.0)


def _gpu(shape, method, prec, BC, steps, flags=1):
    import nlsemagic_gb300 as ng
    U, V, h, k = _case(shape, method)
    return ng.take_steps(U, V, -1.0, 1.0, h * h, BC, steps, k, method=method, precision=prec,
                         flags=flags)


def _oracle(shape, method, prec, BC, steps):
    U, V, h, k = _case(shape, method)
    return oracle.take_steps(U, V, -1.0, 1.0, h * h, BC, steps, k, method=method, precision=prec,
                             flags=oracle.MSD_GUARD)


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3])
def test_point_exact_bits(gpu_lib, BC, method, prec):
    for shape in (GRIDS2 if prec == 2 else []) + GRIDS3:
        got = _gpu(shape, method, prec, BC, 9)
        assert bits_equal(got, _oracle(shape, method, prec, BC, 9)), shape


@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3])
def test_point_contracted(gpu_lib, BC, method):
    import nlsemagic_gb300 as ng
    for shape in GRIDS2 + GRIDS3:
        got = _gpu(shape, method, 2, BC, 9, flags=ng.FLAG_MSD_GUARD | ng.FLAG_FMA)
        assert W.rel_l2(got, _oracle(shape, method, 2, BC, 9)) <= TOL_FMA, shape


# FP32 CD: both sides of 2^20 points, even and odd rows; larger blocks above
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2])
def test_point_fp32_at_the_lines(gpu_lib, BC, method):
    import nlsemagic_gb300 as ng
    for shape in ((128, 100, 81), (128, 101, 82), (129, 101, 82)):
        got = _gpu(shape, method, 1, BC, 2)
        want = _gpu(shape, method, 1, BC, 2, flags=ng.FLAG_MSD_GUARD | ng.FLAG_GATHER)
        assert bits_equal(got, want), shape


def _mixed(shape, method, BC, z2s, steps=7):
    """One solve, run with the knob wide.z2 at each of z2s in turn."""
    import nlsemagic_gb300 as ng
    from nlsemagic_gb300 import autotune
    U, V, h, k = _case(shape, method)
    old = autotune.get_knob("wide.z2")
    try:
        with ng.Solver(shape, method=method, precision=ng.PREC_MIXED, BC=BC, s=-1.0, a=1.0,
                       h2=h * h, k=k) as sv:
            sv.upload(U, V)
            for z2 in z2s:
                autotune.set_knob("wide.z2", z2)
                sv.set_graph_steps(0)
                sv.run(steps)
            return sv.download()
    finally:
        autotune.set_knob("wide.z2", old)


@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3])
def test_point_mixed_same_bits(gpu_lib, BC, method):
    for shape in GRIDS3 + [(92, 92, 93), (92, 92, 94), (128, 100, 81), (128, 101, 82),
                           (129, 101, 82)]:
        got = _mixed(shape, method, BC, (1,))
        assert np.all(np.isfinite(got))
        assert bits_equal(got, _mixed(shape, method, BC, (0,))), shape


@pytest.mark.parametrize("method", [1, 2])
def test_point_mixed_changes_of_form(gpu_lib, method):
    # the streaming kernels keep x-face strips of lo, K and V: refilled after
    # steps by point
    shape = (22, 17, 19)
    want = _mixed(shape, method, 2, (0,) * 4)
    assert bits_equal(_mixed(shape, method, 2, (1, 0, 1, 0)), want)
    assert bits_equal(_mixed(shape, method, 2, (0, 1, 1, 0)), want)
