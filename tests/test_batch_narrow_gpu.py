"""Batches whose work is mostly on narrow 2D grids run by stage passes, and by whole
steps once those have finished: the single solver's bits throughout, with and
without a solve that neither segments nor rectangles take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (shape, method, BC, steps); the narrow ones' whole steps are over the line
NARROW = [((3, 27000), 2, 2, 13), ((8, 26000), 2, 2, 21), ((5, 27001), 2, 2, 17)]
OTHERS = [((700,), 1, 2, 30), ((129,), 2, 3, 40), ((40, 60), 1, 1, 25), ((61, 33), 2, 2, 31)]
LINEAR = [((300,), 2, 4, 26)]


def _field(shape):
    X = np.meshgrid(*[0.2 * np.arange(n) for n in shape], indexing="ij")
    U = (0.8 + 0.2 * np.cos(0.7 * X[0]) * np.cos(0.5 * X[-1])) * np.exp(0.3j * X[0] - 0.2j * X[-1])
    return U, 0.1 * np.cos(0.4 * X[0])


@pytest.mark.parametrize("cuts", [(60,), (5, 9, 60), (14, 1, 8, 60)])
@pytest.mark.parametrize("extra", [[], LINEAR])
def test_batch_of_narrow_grids(gpu_lib, cuts, extra):
    import nlsemagic_gb300 as ng
    solves = NARROW + OTHERS + extra
    b = ng.Batch(1 << 26)
    want, slots = [], []
    for shape, method, BC, steps in solves:
        U, V = _field(shape)
        args = (U, V, -1.0, 1.0, 0.04, BC, steps, 0.004)
        slots.append(b.add(*args, method, ng.PREC_MIXED))
        want.append(ng.take_steps(*args, method=method, precision=ng.PREC_MIXED))
    for n in cuts:
        b.run(n)
        b.sync()
        assert b.last_launches == 1
    for sl, w, (shape, *_) in zip(slots, want, solves):
        assert b.remaining(sl) == 0 and np.all(np.isfinite(w))
        assert np.array_equal(np.ascontiguousarray(b.download(sl)).view(np.float64),
                              np.ascontiguousarray(w).view(np.float64)), shape
    b.close()
