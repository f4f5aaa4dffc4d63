"""On both sides of the sizes where a solve changes its kernels: the bits of the
gather kernels (contracted FP64: its rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(shape):
    X = np.meshgrid(*[0.2 * np.arange(n) for n in shape], indexing="ij")
    U = (0.8 + 0.2 * np.cos(0.7 * X[0]) * np.cos(0.5 * X[-1])) * np.exp(0.3j * X[0] - 0.2j * X[-1])
    return U, 0.1 * np.cos(0.4 * X[0] + 0.3 * X[-1])


def _run(shape, method, prec, BC, flags=0, runs=(11,)):
    import nlsemagic_gb300 as ng
    U, V = _state(shape)
    with ng.Solver(shape, method=method, precision=prec, BC=BC, s=-1.0, a=1.0, h2=0.04, k=0.004,
                   flags=ng.FLAG_MSD_GUARD | flags) as sv:
        sv.upload(U, V)
        for n in runs:
            sv.run(n)
        return np.ascontiguousarray(sv.download()).view(np.float64)


@pytest.mark.parametrize("prec", [1, 3])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3, 4])
def test_small_1d(gpu_lib, BC, method, prec):
    # single-block launches up to 128 or 256 points, the step kernel above
    import nlsemagic_gb300 as ng
    for n in (4, 127, 128, 129, 255, 256, 257):
        want = _run((n,), method, prec, BC, ng.FLAG_GATHER)
        assert np.all(np.isfinite(want))
        assert np.array_equal(_run((n,), method, prec, BC), want), n
        assert np.array_equal(_run((n,), method, prec, BC, runs=(1, 3, 7)), want), n


@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3])
def test_fp32_2d_few_blocks(gpu_lib, BC, method):
    # the next launch triggered early up to 8 blocks (32 x 8 tiles): races would
    # show in repeated runs
    import nlsemagic_gb300 as ng
    for shape in [(3, 3), (9, 8), (15, 15), (32, 64), (33, 64), (64, 33), (15, 130), (300, 9)]:
        want = _run(shape, method, 1, BC, ng.FLAG_GATHER, (41,))
        for _ in range(3):
            assert np.array_equal(_run(shape, method, 1, BC, runs=(41,)), want), shape


@pytest.mark.parametrize("flags", ["fp32", "fp64", "contracted"])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3])
def test_small_grids_by_gather(gpu_lib, BC, method, flags):
    # 2D FP64: 128 points (MSD), 3072 (CD) or 320 and 240 (2SHOC); 3D: 64
    import nlsemagic_gb300 as ng
    prec, f = {"fp32": (1, 0), "fp64": (2, 0), "contracted": (2, ng.FLAG_FMA)}[flags]
    shapes = [(3, 3, 3), (4, 4, 4), (3, 3, 8), (5, 13, 3), (4, 4, 5)]
    if prec == 2:
        shapes += [(3, 3), (16, 8), (43, 3), (15, 16), (16, 20), (107, 3), (48, 64), (439, 7), (3, 1200)]
    for shape in shapes:
        got = _run(shape, method, prec, BC, f, (9, 1))
        want = _run(shape, method, prec, BC, f | ng.FLAG_GATHER, (10,))
        assert np.all(np.isfinite(want))
        if f:
            assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want), shape
        else:
            assert np.array_equal(got, want), shape


@pytest.mark.parametrize("prec,method", [(3, 1), (3, 2), (1, 1)])
@pytest.mark.parametrize("BC", [1, 2, 3])
def test_narrow_2d(gpu_lib, BC, prec, method):
    # whole steps or stage launches by the share of tiles at a face: the bits of
    # the stage launches ("wide2d.ty" 16)
    from nlsemagic_gb300 import autotune
    old = autotune.get_knob("wide2d.ty")
    for shape in [(16, 9000), (9000, 17), (64, 3000), (3001, 63), (128, 1600), (27, 5400), (24, 24),
                  (45, 45), (46, 45), (530, 531)]:
        got = _run(shape, method, prec, BC, runs=(9, 2))
        try:
            autotune.set_knob("wide2d.ty", 16)
            want = _run(shape, method, prec, BC, runs=(11,))
        finally:
            autotune.set_knob("wide2d.ty", old)
        assert np.all(np.isfinite(want))
        assert np.array_equal(got, want), shape
