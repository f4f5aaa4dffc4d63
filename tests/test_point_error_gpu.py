"""Rounding of the contracted FP64 class's 2SHOC (NLSE_FLAG_FMA): the wide form
that 2D and 3D solves take is no further from the scheme's values in extended
precision than the compact form of the gather kernels."""
import numpy as np
import pytest

from nlsemagic_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _moved(U, offsets):
    return U[tuple(slice(1 + d, n - 1 + d) for d, n in zip(offsets, U.shape))]


def _rhs(U, V, h2):
    """F of the compact scheme, s = -1, a = 1, Dirichlet."""
    d = U.ndim
    unit = [tuple(e if t == u else 0 for u in range(d)) for t in range(d) for e in (1, -1)]
    edge = [tuple(e if x == t else f if x == u else 0 for x in range(d))
            for t in range(d) for u in range(t) for e in (1, -1) for f in (1, -1)]
    inner = (slice(1, -1),) * d
    N = -(U.real ** 2 + U.imag ** 2) - V
    U0 = U[inner]
    D = -N * U
    D[inner] = sum(_moved(U, o) - U0 for o in unit) / h2
    lap = ((12 if d == 2 else 10) * D[inner] - sum(_moved(D, o) for o in unit)
           + 2 * sum(_moved(U, o) - U0 for o in edge) / h2) / 12
    F = np.zeros_like(U)
    F[inner] = 1j * (lap + N[inner] * U0)
    return F


def _extended(U, V, h2, k, steps):
    U, V, h2, k = U.astype(np.clongdouble), V.astype(np.longdouble), np.longdouble(h2), \
        np.longdouble(k)
    for _ in range(steps):
        F = _rhs(U, V, h2)
        S = F
        for w, c in ((2, k / 2), (2, k / 2), (1, k)):
            F = _rhs(U + c * F, V, h2)
            S = S + w * F
        U = U + k / 6 * S
    return U


@pytest.mark.parametrize("shape", [(61, 53), (130, 67), (24, 21, 19)])
def test_wide_form_error(gpu_lib, shape):
    import nlsemagic_gb300 as ng
    h, steps = 0.25, 20
    X = np.meshgrid(*[-n * h / 2 + h * np.arange(n) for n in shape], indexing="ij")
    U = (0.8 + 0.2 * np.cos(0.7 * X[0]) * np.cos(0.5 * X[1])) * np.exp(0.3j * X[0] - 0.2j * X[-1])
    V = 0.1 * np.cos(0.4 * X[0] + 0.3 * X[1])
    k = 0.8 * W.linear_stability_k(len(shape), 2, h, 1.0)
    want = _extended(U, V, h * h, k, steps)

    def error(flags):
        got = ng.take_steps(U, V, -1.0, 1.0, h * h, 1, steps, k, method=2,
                            precision=ng.PREC_DOUBLE, flags=flags)
        return float(np.linalg.norm((got - want).ravel().astype(complex)) /
                     np.linalg.norm(U.ravel()))

    flags = ng.FLAG_MSD_GUARD | ng.FLAG_FMA
    wide, compact = error(flags), error(flags | ng.FLAG_GATHER)
    assert compact < 1e-14  # the reference is of the same scheme
    assert wide <= compact, (wide, compact)
