"""The tests of the streaming 3D kernels, and of the 1D forms that the knob
"seg1d" 0 leaves, on those kernels: at their sizes a solve goes by point, or in
whole steps, unless asked otherwise (NLSE_FLAG_STREAM; the knob).  Each keeps its
comparisons; both sides run the forms named in it."""
import functools

import numpy as np
import pytest
import test_autotune_gpu
import test_parity_gpu
import test_pdl_gpu
import test_small1d_gpu
import test_strips_gpu
import test_z2_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture
def stream(gpu_lib, monkeypatch):
    """Solvers and one-shot calls with NLSE_FLAG_STREAM added."""
    import nlsemagic_gb300 as ng
    default = ng.FLAG_MSD_GUARD

    def streaming(f):
        @functools.wraps(f)
        def g(*args, flags=default, **kw):
            return f(*args, flags=flags | ng.FLAG_STREAM, **kw)
        return g

    monkeypatch.setattr(ng, "Solver", streaming(ng.Solver))
    monkeypatch.setattr(ng, "take_steps", streaming(ng.take_steps))
    with ng.Solver((20, 17, 19), precision=ng.PREC_MIXED) as sv:
        assert sv.launches_per_step == 12  # ghosts, interior, faces
    return gpu_lib


@pytest.fixture
def stages1d(gpu_lib):
    from nlsemagic_gb300 import autotune
    old = autotune.get_knob("seg1d")
    autotune.set_knob("seg1d", 0)
    yield gpu_lib
    autotune.set_knob("seg1d", old)


@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3])
@pytest.mark.parametrize("shape,zc", test_z2_gpu.CASES)
def test_two_planes_match_one(stream, shape, zc, BC, method):
    test_z2_gpu.test_two_planes_match_one(stream, shape, zc, BC, method)


@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3])
@pytest.mark.parametrize("shape,zc", [((20, 17, 20), 0), ((38, 33, 66), 5), ((38, 33, 66), 7),
                                      ((70, 45, 100), 0), ((36, 9, 12), 0)])
def test_tile_heights(stream, shape, zc, BC, method):
    test_z2_gpu.test_tile_heights_give_the_same_bits(stream, shape, zc, BC, method)


@pytest.mark.parametrize("BC", [1, 2, 3])
@pytest.mark.parametrize("shape", test_pdl_gpu.SHAPES)
def test_pdl(stream, shape, BC):
    test_pdl_gpu.test_pdl_matches_stream_order(stream, shape, BC)


@pytest.mark.parametrize("BC", [1, 2, 3])
@pytest.mark.parametrize("shape", test_strips_gpu.SHAPES)
def test_strips(stream, shape, BC):
    test_strips_gpu.test_strips_match_full_arrays(stream, shape, BC)


@pytest.mark.parametrize("BC", [2, 3])
@pytest.mark.parametrize("shape", [(40, 40, 40), (96, 64, 130)])
def test_strips_graphs(stream, shape, BC):
    test_strips_gpu.test_strips_graphs_and_split_runs(stream, shape, BC)


def test_strips_refilled(stream):
    test_strips_gpu.test_strips_refilled_after_upload_and_knob_changes(stream)


@pytest.mark.parametrize("BC", [1, 2, 3])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("shape", [(33, 5, 5), (4, 4, 30), (3, 40, 3), (36, 17, 9), (64, 40, 21),
                                   (5, 6, 7), (70, 9, 33)])
def test_mixed_edge_shapes(stream, shape, method, BC):
    test_parity_gpu.test_mixed_3d_edge_shapes(stream, shape, method, BC)


@pytest.mark.parametrize("BC", [1, 2, 3])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("shape", [(33, 5, 5), (65, 66, 4), (129, 3, 7), (31, 33, 34), (64, 64, 9),
                                   (130, 17, 3), (4, 4, 130), (3, 200, 3)])
def test_exact_edge_shapes(stream, shape, method, BC):
    test_parity_gpu.test_exact_edge_shapes_3d(stream, shape, method, BC)


def test_tuned_knobs_same_bits(stream, tmp_path, monkeypatch):
    from nlsemagic_gb300 import autotune
    import nlsemagic_gb300 as ng
    monkeypatch.setattr(autotune, "Solver", ng.Solver)
    test_autotune_gpu.test_tune_cache_apply_and_same_results(stream, tmp_path, monkeypatch)


@pytest.mark.parametrize("prec", [1, 3])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3, 4])
@pytest.mark.parametrize("n,steps", [(64, 7), (1024, 20), (4096, 9)])
def test_small1d(stages1d, n, steps, BC, method, prec):
    test_small1d_gpu.test_small1d_matches_stage_launches(stages1d, n, steps, BC, method, prec)


# FP64 above the step kernel's limit: segments of 256 points, shifted by one
# where n = 256 m + 1
@pytest.mark.parametrize("flags", ["exact", "contracted"])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3])
@pytest.mark.parametrize("n", [65792, 65793, 65794, 65795, 66047])
def test_staged_segments(gpu_lib, n, BC, method, flags):
    import nlsemagic_gb300 as ng
    x = 0.1 * (np.arange(n) - n / 2)
    U = np.exp(0.4j * x) * (0.6 + 0.3 * np.cos(0.05 * x))
    V = 0.2 * np.cos(0.3 * x)
    f = ng.FLAG_MSD_GUARD | (ng.FLAG_FMA if flags == "contracted" else 0)

    def run(f):
        return ng.take_steps(U, V, -1.0, 1.0, 0.01, BC, 7, 0.002, method=method,
                             precision=ng.PREC_DOUBLE, flags=f).view(np.float64)

    got, want = run(f), run(f | ng.FLAG_GATHER)
    assert np.all(np.isfinite(want))
    if flags == "exact":
        assert np.array_equal(got, want)
    else:
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
