"""A knob that changes the form of the kernels, set while a solver holds
captured graphs: the results are those of one form throughout.  3D mixed 2SHOC:
the streaming kernels keep x-face strips of lo, which a graph of steps by
point, or of a run without strips, does not write."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (34, 17, 19)


def _state(phase):
    x, y, z = np.meshgrid(*[np.linspace(0.0, 1.0, n) for n in SHAPE], indexing="ij")
    U = (0.8 + 0.2 * np.cos(2.1 * x + 0.3 + phase) * np.cos(1.7 * y) * np.cos(1.3 * z + 0.5)
         + 0.15j * np.sin(1.9 * x + 1.1 * y + 0.7 * z))
    return U, 0.5 + 0.5 * (x - 0.5) ** 2 + 0.3 * (y - 0.4) ** 2 + 0.2 * z


def _run(script, BC, graph_steps):
    """script: ("run", steps), ("load", phase) or (knob, value), in order."""
    import nlsemagic_gb300 as ng
    from nlsemagic_gb300 import autotune
    old = {k: autotune.get_knob(k) for k in ("wide.z2", "wide.pdl", "wide.tile_order",
                                             "wide.strips")}
    try:
        with ng.Solver(SHAPE, method=2, precision=ng.PREC_MIXED, BC=BC, s=-1.0, a=1.0, h2=0.09,
                       k=0.004) as sv:
            sv.set_graph_steps(graph_steps)
            for what, value in script:
                if what == "run":
                    sv.run(value)
                elif what == "load":
                    sv.upload(*_state(value))
                else:
                    autotune.set_knob(what, value)
            return np.ascontiguousarray(sv.download()).view(np.float64)
    finally:
        for k, v in old.items():
            autotune.set_knob(k, v)


def _scripts(knob):
    yield [("load", 0.0), ("run", 8), (knob, 0), ("run", 9), (knob, 1), ("run", 9)]
    yield [("load", 0.0), (knob, 0), ("run", 9), (knob, 1), ("run", 9), (knob, 0), ("run", 9)]
    # streaming with strips, then a new state and no strips
    yield [("wide.z2", 0), ("load", 0.0), ("run", 9), ("load", 0.7), (knob, 0),
           ("wide.strips", 0), ("run", 9)]


@pytest.mark.parametrize("BC", [2, 3])
@pytest.mark.parametrize("knob", ["wide.z2", "wide.pdl", "wide.tile_order", "wide.strips"])
def test_knob_changes_with_captured_graphs(gpu_lib, knob, BC):
    for script in _scripts(knob):
        want = _run([x for x in script if x[0] in ("run", "load")], BC, 0)
        assert np.all(np.isfinite(want))
        for graph_steps in (4, 8, 3):
            assert np.array_equal(_run(script, BC, graph_steps), want), (script, graph_steps)
