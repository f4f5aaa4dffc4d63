"""Host calls with interleaved complex arrays against the planar entry points:
the same bits, whatever the order, stride and values of the input."""
import ctypes

import numpy as np
import pytest

from nlsemagic_gb300 import api
from nlsemagic_gb300._lib import load

pytestmark = pytest.mark.gpu

SPECIAL = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e300]


def field(shape, special=False, seed=3):
    rng = np.random.default_rng(seed)
    U = np.empty(shape, dtype=np.complex128, order="F")
    U.real = rng.uniform(-1, 1, shape)
    U.imag = rng.uniform(-1, 1, shape)
    if special:
        flat = U.reshape(-1, order="F")
        assert np.shares_memory(flat, U)
        for t, (x, y) in enumerate((x, y) for x in SPECIAL for y in SPECIAL):
            flat[(7 * t) % flat.size] = complex(x, y)
    V = np.asfortranarray(rng.uniform(0, 1, shape))
    return U, V


def forms(U):
    """U in Fortran order, in C order and as every second point of a larger array."""
    wide = np.zeros(tuple(2 * m for m in U.shape), dtype=np.complex128)
    view = wide[tuple(slice(None, None, 2) for _ in U.shape)]
    view[...] = U
    return U, np.ascontiguousarray(U), view


def same(a, b):
    for x, y in ((a.real, b.real), (a.imag, b.imag)):
        ok = ~np.isnan(x)
        assert np.array_equal(x, y, equal_nan=True)
        assert np.array_equal(np.signbit(x[ok]), np.signbit(y[ok]))


def planar_take_steps(U, V, prob, steps):
    re, im = api.planar(U)
    vv = np.ascontiguousarray(V.ravel(order="F"))
    out_r, out_i = np.empty_like(re), np.empty_like(im)
    api.check(load().nlse_take_steps(ctypes.byref(prob), api._ptr(re), api._ptr(im), api._ptr(vv),
                                     api._ptr(out_r), api._ptr(out_i), steps))
    with np.errstate(all="ignore"):
        return (out_r + 1j * out_i).reshape(U.shape, order="F")


@pytest.mark.parametrize("prec", [1, 2, 3])
@pytest.mark.parametrize("shape,steps,special", [
    ((3,), 2, False), ((1, 257), 1, False), ((257, 1), 0, True), ((19, 23), 3, False),
    ((19, 23), 0, True), ((7, 9, 11), 2, False), ((7, 9, 11), 0, True)])
def test_take_steps(shape, steps, special, prec):
    U, V = field(shape, special)
    args = (1.0, 0.7, 1.0, 1, steps, 0.01)  # s, a, h2, BC, chunk, k
    ndim, dims = api.grid_dims(shape)
    prob = api.make_problem(ndim, dims, 1, prec, 1, 1.0, 0.7, 1.0, 0.01, api.FLAG_MSD_GUARD)
    want = planar_take_steps(U, V, prob, steps)
    keep = U.copy(order="F")
    for form in forms(U):
        same(api.take_steps(form, V, *args, method=1, precision=prec), want)
    same(U, keep)  # the input is only read


@pytest.mark.parametrize("prec", [2, 3])
@pytest.mark.parametrize("shape,steps,special", [((5,), 3, False), ((33, 17), 2, False),
                                                 ((33, 17), 0, True), ((6, 7, 8), 1, False)])
def test_batch(shape, steps, special, prec):
    U, V = field(shape, special)
    b = api.Batch(1 << 24, 4)
    slots = [b.add(f, V, 1.0, 0.7, 1.0, 1, steps, 0.01, precision=prec) for f in forms(U)]
    b.run(max(steps, 1))
    n = U.size
    for t in slots:
        re, im = np.empty(n), np.empty(n)
        api.check(load().nlse_batch_download(b._h, t, api._ptr(re), api._ptr(im)))
        with np.errstate(all="ignore"):
            want = (re + 1j * im).reshape(shape, order="F")
        same(b.download(t), want)
        same(b.download(t), b.download(slots[1]))


def test_real_and_narrow_inputs():
    """Types other than complex128 keep the planar route."""
    U, V = field((12, 10))
    args = (1.0, 0.7, 1.0, 1, 2, 0.01)
    r = np.asfortranarray(U.real)
    same(api.take_steps(r, V, *args), api.take_steps(r.astype(np.complex128), V, *args))
    c = U.astype(np.complex64)
    same(api.take_steps(c, V, *args), api.take_steps(c.astype(np.complex128), V, *args))
    same(api.take_steps(U.astype(">c16"), V, *args), api.take_steps(U, V, *args))
