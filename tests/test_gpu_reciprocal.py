"""The reciprocals of the flip-symmetric passes: the iteration's error over the
whole exponent range against the exact value and CUDA's division, its guard's
edges, and solves whose divisors leave the guard."""
import numpy as np
import pytest

import duct_b200 as D
from duct_b200 import synth

pytestmark = pytest.mark.gpu


def reciprocals(ctx, x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.empty((3, x.size))
    ctx._check(D.lib().ductgpu_selftest_reciprocal(ctx.h, D._ptr(x), D._ptr(y), x.size))
    return y[0], y[1] == 1.0, y[2]


def test_every_exponent(gpu_ctx):
    """Within 0.51 ulp, and within one ulp of the rounded division, at 400 mantissas of each
    binary exponent, both signs: where the iteration serves it is r (1 + e +
    e^2) with |e| <= 2^-20, 2^-60 off before its one rounding (2^-53), and the
    check in 64-bit mantissas adds 2^-62."""
    rng = np.random.default_rng(1)
    mant = np.concatenate([[1.0, np.nextafter(1.0, 2.0), 1.5, np.nextafter(2.0, 1.0)], 1.0 + rng.random(396)])
    e = np.arange(-1022, 1024)
    x = np.ldexp(mant[None, :], e[:, None]) * np.where(rng.random((e.size, mant.size)) < 0.5, -1.0, 1.0)
    r, served, q = (a.reshape(x.shape) for a in reciprocals(gpu_ctx, x.ravel()))
    assert np.array_equal(served, np.broadcast_to(((e >= -1000) & (e <= 1000))[:, None], x.shape))
    with np.errstate(under="ignore"):
        assert np.array_equal(q, 1.0 / x)               # CUDA's division is the correctly rounded one
        assert np.array_equal(r[~served], q[~served])
    assert np.all(np.abs(r - q) <= np.spacing(np.abs(q)))
    err = np.abs(r[served].astype(np.longdouble) * x[served].astype(np.longdouble) - 1)
    assert err.max() <= 2.0 ** -53 + 2.0 ** -60 + 2.0 ** -62


def test_edges_of_the_guard(gpu_ctx):
    tiny, big = 2.0 ** -1000, np.ldexp(1.0, 1001)
    x = np.array([tiny, np.nextafter(tiny, 0.0), np.nextafter(big, 0.0), big, 0.0, -0.0, np.inf, -np.inf, np.nan,
                  2.0 ** -1074, -2.0 ** -1060, np.finfo(float).max, np.finfo(float).tiny])
    r, served, q = reciprocals(gpu_ctx, x)
    assert served.tolist() == [True, False, True] + [False] * 10
    assert np.array_equal(r[~served], q[~served], equal_nan=True)
    assert np.array_equal(np.signbit(r), np.signbit(q)) and np.isnan(r[8])
    assert r[4] == np.inf and r[5] == -np.inf and r[6] == 0.0
    assert np.all(np.abs(r[served] - q[served]) <= np.spacing(q[served]))


@pytest.mark.parametrize("m", [33, 34, 65, 98, 129, 193])
def test_divisors_outside_the_guard(gpu_ctx, m):
    """Planes of one field with lambda on both sides of 2^1001: beyond it every
    divisor is -lambda to rounding, so the solution is -rhs / lambda to the rounding
    of four products (5e-12, as for Dirichlet fields elsewhere); the others are
    what they are by themselves, bit for bit; on chip equals the passes."""
    xalp = np.array([1.0, 2.0 ** 501, 3.0, 2.0 ** 499, 2.0 ** 500.75])
    huge = xalp ** 2 >= 2.0 ** 1001
    rhs = np.asfortranarray(2.0 ** 60 * synth.chebyshev_rhs(m, m, xalp.size, seed=m, ib=1))
    gpu_ctx.pseudomat(m)
    sols = []
    try:
        for kernel in (D.PASS_PARITY, D.PASS_PARITY_QUEUE):
            gpu_ctx.set_pass_kernel(kernel)
            sols.append(gpu_ctx.helm3d(rhs.copy(order="F"), "d", 0.0, xalp, ib=1))
        alone = [gpu_ctx.helm3d(np.asfortranarray(rhs[:, :, k:k + 1]), "d", 0.0, xalp[k:k + 1], ib=1)
                 for k in range(xalp.size)]
    finally:
        gpu_ctx.set_pass_kernel(-1)
    assert huge.tolist() == [False, True, False, False, True]
    assert np.array_equal(sols[0], sols[1]) and np.all(np.isfinite(sols[0]))
    for k in range(xalp.size):
        assert np.array_equal(sols[0][:, :, k], alone[k][:, :, 0])
        if huge[k]:
            inner = (slice(1, -1), slice(1, -1), k)
            want, got = rhs[inner], -(sols[0][inner] * 2.0 ** 600) * (xalp[k] ** 2 * 2.0 ** -600)
            assert np.linalg.norm(got - want) <= 5e-12 * np.linalg.norm(want)
