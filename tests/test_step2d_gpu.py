"""2D solves of the mixed class, and of FP32 with CD, run a whole RK4 step per
launch: every tile computes its four stages with the halo they need.  The same
bits as the launch-per-stage kernels (and in FP32 as the oracle), for both
methods and boundary codes 1-3: on grids of one tile, of one tile and one cell
along either axis, with faces in every position of a tile, on both sides of
every line of the dispatch rule; for odd step counts, odd graphs, and when the
form changes between runs of one solve."""
import numpy as np
import pytest

import oracle
from nlsemagic_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# tiles hold up to 20 x 20, 52 x 20 (2SHOC), 26 x 26 or 58 x 26 (CD) points
SHAPES = [(16, 16), (20, 21), (26, 27), (27, 26), (52, 40), (53, 41), (58, 78), (59, 53),
          (105, 61), (16, 161), (161, 16), (300, 19)]
LINES = [(256, 128), (257, 128), (256, 257), (512, 256), (513, 257), (512, 513), (725, 724),
         (1024, 1025)]


def bits_equal(a, b):
    a = np.ascontiguousarray(a, dtype=np.complex128).view(np.float64)
    b = np.ascontiguousarray(b, dtype=np.complex128).view(np.float64)
    return np.array_equal(a, b, equal_nan=True)


def _case(shape, method):
    h = 0.25
    X, Y = np.meshgrid(*[-n * h / 2 + h * np.arange(n) for n in shape], indexing="ij")
    U = (0.8 + 0.2 * np.cos(0.7 * X) * np.cos(0.5 * Y)) * np.exp(0.3j * X - 0.2j * Y)
    return U, 0.1 * np.cos(0.4 * X + 0.3 * Y), h, 0.5 * W.linear_stability_k(2, method, h, 1.0)


def _run(shape, BC, method, prec, runs, graph=8):
    """runs: (steps, wide2d.ty) one after the other on one solver."""
    import nlsemagic_gb300 as ng
    from nlsemagic_gb300 import autotune
    U, V, h, k = _case(shape, method)
    old = autotune.get_knob("wide2d.ty")
    try:
        with ng.Solver(shape, method=method, precision=prec, BC=BC, s=-1.0, a=1.0, h2=h * h,
                       k=k) as sv:
            sv.set_graph_steps(graph)
            sv.upload(U, V)
            for steps, ty in runs:
                autotune.set_knob("wide2d.ty", ty)
                sv.run(steps)
            return sv.download()
    finally:
        autotune.set_knob("wide2d.ty", old)


@pytest.mark.parametrize("prec,method", [(3, 1), (3, 2), (1, 1)])
@pytest.mark.parametrize("BC", [1, 2, 3])
def test_step2d_same_bits(gpu_lib, BC, prec, method):
    for shape in SHAPES:
        got = _run(shape, BC, method, prec, [(11, 0)])
        assert np.all(np.isfinite(got))
        assert bits_equal(got, _run(shape, BC, method, prec, [(11, 8)])), shape
        if prec == 1:
            U, V, h, k = _case(shape, method)
            want = oracle.take_steps(U, V, -1.0, 1.0, h * h, BC, 11, k, method=method,
                                     precision=1, flags=oracle.MSD_GUARD)
            assert bits_equal(got, want), shape


@pytest.mark.parametrize("prec,method", [(3, 1), (3, 2), (1, 1)])
@pytest.mark.parametrize("BC", [1, 2])
def test_step2d_same_bits_at_the_lines(gpu_lib, BC, prec, method):
    for shape in LINES:
        assert bits_equal(_run(shape, BC, method, prec, [(5, 0)]),
                          _run(shape, BC, method, prec, [(5, 16)])), shape


@pytest.mark.parametrize("prec", [1, 3])
def test_step2d_odd_graphs_and_changes_of_form(gpu_lib, prec):
    shape, runs = (70, 45), [(7, 0), (8, 8), (3, 0), (10, 0), (5, 8), (5, 0), (6, 8)]
    want = _run(shape, 3, 1, prec, [(sum(n for n, _ in runs), 8)], graph=0)
    for graph in (0, 1, 5, 8):
        assert bits_equal(_run(shape, 3, 1, prec, runs, graph), want), graph
