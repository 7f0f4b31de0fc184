"""The solve of a plane on chip (k_plane, at most 63 interior points a side)
against the four passes, whose arithmetic and order it keeps: bit for bit, for
odd and even sizes up to its half blocks, Dirichlet and Neumann fields (a
singular plane among them), solutions in place of their right-hand sides, the
adjoint, rectangles, and the calls that go back to the passes (arrays that
overlap, many small planes)."""
import numpy as np
import pytest

import duct_b200 as D
from duct_b200 import synth

pytestmark = pytest.mark.gpu


def fields_of(ctx, m, counts, inplace):
    out = []
    for k, (bound, lam, nm) in enumerate(counts):
        f = synth.chebyshev_rhs(m, m, nm, seed=70 + k, ib=0)
        r = ctx.device_array(f.shape)
        r.upload(f)
        out.append(dict(rhs=r, sol=r if inplace else ctx.device_array(f.shape), xalp=0.5 * np.arange(nm), alambda=lam, ib=0,
                        bound=bound))
    return out


def solved(ctx, m, kernel, counts, inplace=False, adjoint=False):
    """Solutions, right-hand sides after the call, and its pass launches."""
    ctx.set_pass_kernel(kernel)
    try:
        fields = fields_of(ctx, m, counts, inplace)
        ctx.profile(True)
        ctx.profile_reset()
        if adjoint:
            ctx.solve_adjoint_fields_dev(fields)
        else:
            ctx.solve_fields_dev(fields, precision=D.PREC_FP64)
        ctx.synchronize()
        launches = ctx.profile_read(D.K_PASS_FP64)[1]
        ctx.profile(False)
        got = [f["sol"].download() for f in fields] + [f["rhs"].download() for f in fields]
        for f in fields:
            f["rhs"].free()
            if not inplace:
                f["sol"].free()
        return got, launches
    finally:
        ctx.set_pass_kernel(-1)


@pytest.mark.parametrize("m", [5, 6, 18, 33, 34, 35, 56, 57, 64, 65])
@pytest.mark.parametrize("inplace", [False, True])
def test_equal_to_the_passes(gpu_ctx, m, inplace):
    gpu_ctx.pseudomat(m)
    counts = [("d", 4.0e3, 3), ("n", 0.0, 2), ("d", 1.0, 1)]
    a, na = solved(gpu_ctx, m, D.PASS_PARITY, counts, inplace)
    b, nb = solved(gpu_ctx, m, D.PASS_PARITY_QUEUE, counts, inplace)
    assert (na, nb) == (4, 1)
    for x, y in zip(a, b):
        assert np.all(np.isfinite(x)) and np.array_equal(x, y)


@pytest.mark.parametrize("m", [6, 33, 65])
def test_adjoint_equal_to_the_passes(gpu_ctx, m):
    gpu_ctx.pseudomat(m)
    counts = [("d", 4.0e3, 3), ("n", 0.0, 2)]
    a, na = solved(gpu_ctx, m, D.PASS_PARITY, counts, adjoint=True)
    b, nb = solved(gpu_ctx, m, D.PASS_PARITY_QUEUE, counts, adjoint=True)
    assert (na, nb) == (4, 1)
    for x, y in zip(a, b):
        assert np.all(np.isfinite(x)) and np.array_equal(x, y)


@pytest.mark.parametrize("m,planes,launches", [(33, 120, 1), (41, 255, 4), (33, 255, 4), (57, 255, 1)])
def test_many_small_planes_go_by_the_passes(gpu_ctx, m, planes, launches):
    """Both sides of the rule's lines on a GPU of 120 to 190 SMs, equal bit for bit."""
    gpu_ctx.pseudomat(m)
    counts = [("d", 4.0e3, planes)]
    a, na = solved(gpu_ctx, m, D.PASS_PARITY, counts)
    b, nb = solved(gpu_ctx, m, D.PASS_PARITY_QUEUE, counts)
    assert (na, nb) == (4, launches)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


def test_overlapping_arrays_go_by_the_passes(gpu_ctx):
    """A field that is solved into another's right-hand side: the passes read
    every right-hand side before they write a solution."""
    m, nm = 65, 3
    gpu_ctx.pseudomat(m)
    out = {}
    for kernel in (D.PASS_PARITY, D.PASS_PARITY_QUEUE):
        gpu_ctx.set_pass_kernel(kernel)
        try:
            f = fields_of(gpu_ctx, m, [("d", 4.0e3, nm), ("d", 1.0, nm)], False)
            mine = f[0]["sol"]
            f[0]["sol"] = f[1]["rhs"]
            gpu_ctx.solve_fields_dev(f, precision=D.PREC_FP64)
            gpu_ctx.synchronize()
            out[kernel] = [x["sol"].download() for x in f]
            for x in (f[0]["rhs"], f[1]["rhs"], f[1]["sol"], mine):
                x.free()
        finally:
            gpu_ctx.set_pass_kernel(-1)
    for x, y in zip(out[D.PASS_PARITY], out[D.PASS_PARITY_QUEUE]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("my,mz", [(19, 34), (65, 33), (64, 65)])
def test_rectangles(oracle, my, mz):
    nm, aspect, xalp = 3, 1.5, np.array([0.0, 1.0, 4.0])
    rhs = synth.chebyshev_rhs(my, mz, nm, seed=my, ib=0)
    ref = oracle.helm3d_temp(rhs, oracle.Dir(my, 1.0), oracle.Dir(mz, aspect), 3.0e3, xalp)
    out = []
    for fold in (None, 1):
        with D.Context(0) as ctx:
            ctx.pseudomat_temp(0, my, mz, 1.0, aspect)
            if fold is not None:
                ctx.set_rect_fold(fold)
            r, s = ctx.device_array(rhs.shape), ctx.device_array(rhs.shape)
            r.upload(rhs)
            ctx.profile(True)
            ctx.profile_reset()
            ctx.solve_rect_fields_dev([dict(rhs=r, sol=s, xalp=xalp, alambda=3.0e3, ib=0, slot=0)])
            ctx.synchronize()
            out.append((s.download(), ctx.profile_read(D.K_PASS_FP64)[1]))
            r.free()
            s.free()
    assert (out[0][1], out[1][1]) == (1, 4)
    assert np.array_equal(out[0][0], out[1][0])
    assert np.linalg.norm(out[0][0] - ref) < 5e-12 * np.linalg.norm(ref)
