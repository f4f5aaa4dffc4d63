"""3D 2SHOC in FP64 and FP32 without D scratch (NLSE_FLAG_STREAM, and solves
whose scratch does not fit beside what they hold): the oracle's bits, and the
grids that fit are those that fitted before there was a scratch."""
import numpy as np
import pytest

import oracle
from nlsemagic_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# edges of the 32 x 8 tile and of z chunks; odd rows (no TMA); 3 cells thin
GRIDS = [(3, 3, 3), (5, 6, 7), (33, 5, 5), (65, 66, 4), (31, 33, 34), (64, 64, 9), (130, 17, 3),
         (4, 4, 130), (3, 40, 3), (36, 17, 9), (66, 9, 33)]


def bits_equal(a, b):
    a = np.ascontiguousarray(a, dtype=np.complex128).view(np.float64)
    b = np.ascontiguousarray(b, dtype=np.complex128).view(np.float64)
    return np.array_equal(a, b, equal_nan=True)


def _case(shape):
    X = np.meshgrid(*[0.25 * np.arange(n) for n in shape], indexing="ij")
    U = (0.8 + 0.2 * np.cos(0.7 * X[0]) * np.cos(0.5 * X[1])) * np.exp(0.3j * X[0] - 0.2j * X[2])
    return U, 0.1 * np.cos(0.4 * X[0] + 0.3 * X[1])


def _want(U, V, method, prec, BC, steps):
    return oracle.take_steps(U, V, -1.0, 1.0, 0.0625, BC, steps, 0.004, method=method,
                             precision=prec, flags=oracle.MSD_GUARD)


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("BC", [1, 2, 3])
def test_stream_form_bits(gpu_lib, BC, method, prec):
    import nlsemagic_gb300 as ng
    for shape in GRIDS:
        U, V = _case(shape)
        got = ng.take_steps(U, V, -1.0, 1.0, 0.0625, BC, 9, 0.004, method=method, precision=prec,
                            flags=ng.FLAG_MSD_GUARD | ng.FLAG_STREAM)
        assert bits_equal(got, _want(U, V, method, prec, BC, 9)), shape


def test_server_admits_what_fits_without_scratch(gpu_lib):
    import nlsemagic_gb300 as ng
    from nlsemagic_gb300.serve import Server
    reqs = W.serving_requests(count=1, rate=100.0, n3=(40, 41), steps=(20, 21), ratio=(0, 0, 1))
    i = reqs[0].inst
    i.precision, i.method = ng.PREC_DOUBLE, 2
    lean = ng.Solver.bytes_for(i.U.shape, 2, ng.PREC_DOUBLE, i.BC,
                               ng.FLAG_MSD_GUARD | ng.FLAG_STREAM)
    srv = Server(pool_bytes=1 << 24, solo_points=1, solo_bytes=lean, fp64_fma=False,
                 keep_snapshots=True)
    summary, done = srv.serve(reqs)
    srv.close()
    assert summary["rejected"] == 0 and len(done) == 1
    want = oracle.take_steps(i.U, i.V, i.s, i.a, i.h * i.h, i.BC, i.steps, i.k, method=2,
                             precision=2, flags=oracle.MSD_GUARD)
    assert bits_equal(done[0].snapshot, want)


def test_scratch_that_does_not_fit(gpu_lib):
    """Device memory filled so that the solver fits and its scratch does not: at
    creation, and when the staging buffers of an upload need its room."""
    import torch

    import nlsemagic_gb300 as ng
    shape = (160, 150, 140)
    n = int(np.prod(shape))
    base, scratch, stage = 72 * n, 16 * n, 24 * n
    U, V = _case(shape)

    def solver(flags=ng.FLAG_MSD_GUARD):
        return ng.Solver(shape, method=2, precision=ng.PREC_DOUBLE, BC=1, s=-1.0, a=1.0,
                         h2=0.0625, k=0.004, flags=flags)

    def result(sv):
        sv.upload(U, V)
        sv.run(10)  # a captured graph and single steps
        return sv.download()

    with solver(ng.FLAG_MSD_GUARD | ng.FLAG_STREAM) as sv:  # its kernels are loaded, too
        lean = sv.device_bytes
        want = result(sv)

    def fill(leave):
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        return torch.empty(free - leave, dtype=torch.uint8, device="cuda")

    room = 24 << 20  # for the allocator's and graphs' own use
    assert room < scratch / 2
    block = fill(base + stage + room)
    try:
        with solver() as sv:  # base fits; the scratch too, until the upload
            assert sv.device_bytes == lean + scratch
            assert bits_equal(result(sv), want)
            assert sv.device_bytes == lean + stage
    finally:
        del block
        torch.cuda.empty_cache()
    block = fill(base + room)
    try:
        with solver() as sv:
            assert sv.device_bytes == lean
    finally:
        del block
        torch.cuda.empty_cache()
    with solver() as sv:
        assert bits_equal(result(sv), want)
        assert sv.device_bytes == lean + scratch + stage
