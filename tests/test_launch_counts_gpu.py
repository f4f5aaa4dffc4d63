"""Launches a step, as the solver reports them: one per stage, two where a
stage forms D and then F, three and two for the streaming mixed 3D kernels."""
import pytest

pytestmark = pytest.mark.gpu


def test_launches_per_step(gpu_lib):
    import nlsemagic_gb300 as ng
    g, f, s = ng.FLAG_GATHER, ng.FLAG_FMA, ng.FLAG_STREAM
    three, two = (20, 17, 19), (40, 33)
    # shape, precision, method, BC, flags, launches
    for case in [(three, 2, 2, 2, f, 4), (two, 2, 2, 1, f, 4), (three, 2, 1, 2, f, 4),
                 (three, 2, 2, 2, f | g, 8), (three, 2, 2, 2, 0, 8), (two, 2, 2, 2, 0, 8),
                 (three, 1, 2, 2, 0, 8), (three, 2, 2, 2, s, 4), (three, 1, 2, 2, s, 4),
                 (three, 1, 1, 1, s, 4), (three, 3, 2, 2, 0, 4), (three, 3, 2, 2, s, 12),
                 (three, 3, 1, 2, s, 8), ((70000,), 2, 2, 2, 0, 4), ((70000,), 2, 2, 4, 0, 8),
                 ((5000,), 1, 2, 4, 0, 4), ((5000,), 3, 2, 2, g, 8)]:
        shape, prec, method, BC, flags, want = case
        with ng.Solver(shape, method=method, precision=prec, BC=BC,
                       flags=ng.FLAG_MSD_GUARD | flags) as sv:
            assert sv.launches_per_step == want, case
