"""Batched mixed 1D and 2D solves in whole RK4 steps: tasks of a tile's step (2D) or
of several steps (1D), ordered per solve by counters.  The single solver's bits
for every boundary code (1D one-sided ends included), uneven step counts and
runs cut at any step; and when a 3D solve joins and leaves, which puts the whole
class through the launch-per-stage kernel in between."""
import numpy as np
import pytest

from nlsemagic_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# (shape, method, BC, steps): one tile, several, sides one cell beyond a tile
SOLVES = [((5,), 1, 1, 9), ((128,), 2, 2, 31), ((1537,), 1, 2, 23), ((1025,), 2, 3, 40),
          ((3000,), 2, 4, 17), ((9000,), 1, 4, 12), ((58, 26), 1, 1, 30), ((59, 27), 1, 2, 21),
          ((53, 21), 2, 2, 25), ((120, 90), 2, 1, 8), ((3, 40), 2, 3, 33), ((200, 61), 1, 3, 1)]


def bits_equal(a, b):
    a = np.ascontiguousarray(a, dtype=np.complex128).view(np.float64)
    b = np.ascontiguousarray(b, dtype=np.complex128).view(np.float64)
    return np.array_equal(a, b, equal_nan=True)


def _field(shape, method):
    h = 0.2
    X = np.meshgrid(*[-n * h / 2 + h * np.arange(n) for n in shape], indexing="ij")
    U = (0.8 + 0.2 * np.cos(0.7 * X[0]) * np.cos(0.5 * X[-1])) * np.exp(0.3j * X[0] - 0.2j * X[-1])
    return U, 0.1 * np.cos(0.4 * X[0]), h, 0.5 * W.linear_stability_k(len(shape), method, h, 1.0)


@pytest.mark.parametrize("cuts", [(100,), (1, 1, 100), (5, 7, 2, 100), (24, 3, 100)])
@pytest.mark.parametrize("join", [False, True])
def test_batch_steps_same_bits(gpu_lib, cuts, join):
    import nlsemagic_gb300 as ng
    b = ng.Batch(1 << 28)
    want, slots = [], []
    for shape, method, BC, steps in SOLVES:
        U, V, h, k = _field(shape, method)
        slots.append(b.add(U, V, -1.0, 1.0, h * h, BC, steps, k, method, ng.PREC_MIXED))
        want.append(ng.take_steps(U, V, -1.0, 1.0, h * h, BC, steps, k, method=method,
                                  precision=ng.PREC_MIXED))
    for t, steps in enumerate(cuts):
        third = None
        if join and t % 2 == 1:
            U, V, h, k = _field((9, 8, 7), 2)
            third = b.add(U, V, -1.0, 1.0, h * h, 1, 50, k, 2, ng.PREC_MIXED)
        b.run(steps)
        b.sync()
        assert b.last_launches == 1
        if third is not None:
            b.remove(third)
    for (shape, *_), sl, w in zip(SOLVES, slots, want):
        assert b.remaining(sl) == 0
        assert bits_equal(b.download(sl), w), shape
    b.close()
