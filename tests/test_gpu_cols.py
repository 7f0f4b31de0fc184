"""The flip-symmetric pass kernel (k_pass_cols) where it can go wrong: interior
points below, at and above its row tiles (16) and half blocks (32, 64, 96), odd
and even, with and without a middle point, and line counts that leave a last
unit of 4 partial, against the oracle.  The two are different
FP64 decompositions of one operator: 5e-12 for Dirichlet fields, 2e-10 for
Neumann ones, the bounds of test_gpu_parity.py.  A field's planes must
not depend on the batch they are in: bit for bit."""
import numpy as np
import pytest

import duct_b200 as D
from duct_b200 import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel())


@pytest.mark.parametrize("m", [5, 18, 34, 35, 65, 66, 67, 98, 99, 129, 130, 131, 146, 161, 192, 193])
def test_half_blocks_and_remainders(gpu_ctx, oracle, m):
    ops = oracle.Ops(m)
    gpu_ctx.pseudomat(m)
    gpu_ctx.set_pass_kernel(D.PASS_PARITY)
    try:
        for bound, lam, tol in (("d", 3.0e3, 5e-12), ("n", 3.0e3, 2e-10)):
            rhs = synth.chebyshev_rhs(m, m, 3, seed=m, ib=0)
            xalp = np.array([0.0, 1.5, 7.0])
            ref, _ = oracle.helm3d(rhs, ops, bound, lam, xalp)
            sol = gpu_ctx.helm3d(rhs.copy(order="F"), bound, lam, xalp, ipro=0)
            assert rel(sol, ref) < tol
            one = gpu_ctx.helm3d(np.asfortranarray(rhs[:, :, 1:2]), bound, lam, xalp[1:2], ib=1)
            assert np.array_equal(one[:, :, 0], sol[:, :, 1])
    finally:
        gpu_ctx.set_pass_kernel(-1)
