"""Line products on the resident-operator core (k_dcols, k_mode_lines) at line
lengths below, at and above their 16-row tiles, line counts that leave a last
unit of 4 partial, against the forms they
replace: the derivative kernel of line kernel 2 (the same operators, another
order of sums) and the FFT transforms of line kernel 0.

Tolerances: a sum of N products in any order is within N eps sum |a| |x| of the
exact one (to first order), so two forms differ by at most twice that: with R the
largest absolute row sum of the operator, 2 N eps R max|x|; the FFT forms stay
within the same bound."""
import ctypes as C

import numpy as np
import pytest

import duct_b200 as D
from duct_b200 import synth

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52
LENGTHS = [17, 25, 33, 49, 65, 97, 129, 145, 193]


def field(rng, shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


def row_sum(n, order):
    return np.abs(D.cheb_deriv_matrix(n, order)).sum(axis=1).max()


def run(ctx, kernel, f, call, outs):
    ctx.set_line_kernel(kernel)
    try:
        src = ctx.device_array(f.shape)
        src.upload(f)
        dst = [ctx.device_array(f.shape) for _ in range(outs)]
        call(src, *dst)
        ctx.synchronize()
        got = [d.download() for d in (dst or [src])]
        for d in [src] + dst:
            d.free()
        return got
    finally:
        ctx.set_line_kernel(1)


@pytest.mark.parametrize("n", LENGTHS + [19, 37, 109, 163])
@pytest.mark.parametrize("sign", [-1, 1])
def test_transforms(gpu_ctx, n, sign):
    nm = 3
    for my, mz, d in ((n, 33, "y"), (33, n, "z")):
        f = field(np.random.default_rng(n), (my, mz, nm))

        def call(src):
            gpu_ctx._check(D.lib().ductgpu_transyz_dev(gpu_ctx.h, C.c_void_p(src.ptr), my, mz, nm, d.encode(), sign))

        a, = run(gpu_ctx, 1, f, call, 0)
        b, = run(gpu_ctx, 0, f, call, 0)
        # rows of the forward matrix sum to at most 2, of the inverse to n
        assert np.abs(a - b).max() <= 2 * n * EPS * (2.0 if sign < 0 else n) * np.abs(f).max()


@pytest.mark.parametrize("n", [65, 97, 109, 129, 145, 163, 193])
def test_transforms_do_not_depend_on_the_batch(gpu_ctx, n):
    """Bit for bit, a field's first modes by themselves."""
    nm, few = 150, 3                        # 4950 lines: 32 and more for every SM
    for my, mz, d in ((n, 33, "y"), (33, n, "z")):
        f = field(np.random.default_rng(n), (my, mz, nm))
        got = []
        for k in (nm, few):
            def call(src):
                gpu_ctx._check(D.lib().ductgpu_transyz_dev(gpu_ctx.h, C.c_void_p(src.ptr), my, mz, k, d.encode(), -1))

            got += run(gpu_ctx, 1, np.asfortranarray(f[:, :, :k]), call, 0)
        assert np.array_equal(got[0][:, :, :few], got[1])


def test_every_length_in_one_context(gpu_ctx):
    """A context keeps operators for all the lengths that transyz takes."""
    for n in (17, 19, 25, 33, 37, 49, 55, 65, 73, 97, 109, 129, 145, 163, 193):
        f = field(np.random.default_rng(n), (n, n, 2))
        for d in (b"y", b"z"):
            def call(src):
                for sign in (-1, 1):
                    gpu_ctx._check(D.lib().ductgpu_transyz_dev(gpu_ctx.h, C.c_void_p(src.ptr), n, n, 2, d, sign))

            there_and_back, = run(gpu_ctx, 1, f, call, 0)
            # two products with row sums of at most 2 and n, n terms each
            assert np.abs(there_and_back - f).max() <= 2 * n * EPS * 2 * n * np.abs(f).max()


@pytest.mark.parametrize("n", [33, 163])
def test_transform_first_used_inside_a_capture(n):
    """The operators of a length are built on first use, also while the
    context's stream is being captured: the replay equals later direct calls."""
    torch = pytest.importorskip("torch")
    f = field(np.random.default_rng(n), (n, n, 3))
    with D.Context(0) as ctx:
        a, b = ctx.device_array(f.shape), ctx.device_array(f.shape)
        side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        x = torch.zeros(8, device="cuda")
        ctx._check(D.lib().ductgpu_set_stream(ctx.h, C.c_void_p(side.cuda_stream)))
        for arr in (a, b):
            arr.upload(f)
        ctx.synchronize()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            x += 1.0
            ctx._check(D.lib().ductgpu_transyz_dev(ctx.h, C.c_void_p(a.ptr), n, n, 3, b"y", -1))
        graph.replay()
        torch.cuda.synchronize()
        ctx._check(D.lib().ductgpu_transyz_dev(ctx.h, C.c_void_p(b.ptr), n, n, 3, b"y", -1))
        ctx.synchronize()
        assert np.array_equal(a.download(), b.download()) and np.all(np.isfinite(b.download()))
        assert not np.array_equal(b.download(), f)
        del graph
        a.free()
        b.free()
        ctx._check(D.lib().ductgpu_set_stream(ctx.h, None))


@pytest.mark.parametrize("n", LENGTHS)
def test_derivatives(gpu_ctx, n):
    nm = 75 if n >= 145 else 3
    xalp = 0.5 * np.arange(nm)
    for my, mz in ((n, 33), (33, n)):
        f = field(np.random.default_rng(n), (my, mz, nm))
        top = np.abs(f).max()
        one = 2 * max(my, mz) * EPS * max(row_sum(my, 1), row_sum(mz, 1)) * top
        two = 2 * max(my, mz) * EPS * (row_sum(my, 2) + row_sum(mz, 2) + xalp[-1] ** 2) * top
        for outs, tol, call in ((3, one, lambda s, x, y, z: gpu_ctx.grad3d_dev(s, x, y, z, xalp, 1.0)),
                                (1, two, lambda s, o: gpu_ctx.laplacian3d_dev(s, o, xalp, 1.0))):
            for a, b in zip(run(gpu_ctx, 1, f, call, outs), run(gpu_ctx, 2, f, call, outs)):
                assert np.all(np.isfinite(a)) and np.abs(a - b).max() <= tol


@pytest.mark.parametrize("n", LENGTHS + [257])
def test_derivatives_do_not_depend_on_the_batch(gpu_ctx, n):
    """Bit for bit, a field's first modes by themselves: one to three outputs a
    job, x-terms, accumulated outputs and mode 0, from a few lines to 16 and more
    for every SM."""
    nm, few = 75, 3
    xalp = 0.5 * np.arange(nm)
    for my, mz in ((n, 33), (33, n)):
        rng = np.random.default_rng(n)
        f = [field(rng, (my, mz, nm)) for _ in range(5)]

        def results(k):
            dev = []
            try:
                for a in f + [f[0]] * 9:
                    dev.append(gpu_ctx.device_array((my, mz, k)))
                    dev[-1].upload(np.asfortranarray(a[:, :, :k]))
                u, v, w, p, phi, gx, gy, gz, lap, div, *vort = dev
                x = xalp[:k]
                gpu_ctx.grad3d_dev(u, gx, gy, gz, x, 1.5)
                gpu_ctx.laplacian3d_dev(v, lap, x, 0.5, what="a")
                gpu_ctx.div3d_dev(u, v, w, div, x, 1.0)
                gpu_ctx._check(D.lib().ductgpu_vorticity_dev(gpu_ctx.h, *(C.c_void_p(a.ptr) for a in (u, v, w, vort[0])), my, mz, k,
                                                             x.ctypes.data_as(C.c_void_p), 1.0, 1))
                gpu_ctx.update_uvwp_dev(u, v, w, p, phi, x, 0.4, 0.3, 1.0e-3, 5.0e-4)
                gpu_ctx.synchronize()
                return [a.download() for a in dev]
            finally:
                for a in dev:
                    a.free()

        for a, b in zip(results(nm), results(few)):
            assert np.all(np.isfinite(a)) and np.array_equal(a[:, :, :few], b)


@pytest.mark.parametrize("m", [13, 25, 37, 73, 97, 145])
def test_shen_by_parity(gpu_ctx, oracle, m):
    """Chebyshev <-> Legendre products by parity, at the row tiles that
    test_gpu_shen.py leaves out, Dirichlet and Neumann fields in one call; its tolerance."""
    xalp = np.array([0.0, 0.5, 7.0])
    gpu_ctx.preshen(m, "d")
    gpu_ctx.preshen(m, "n")
    fields, refs = [], []
    for k, (bound, lam) in enumerate((("d", 2.5), ("n", 0.0))):
        f = synth.chebyshev_rhs(m, m, 3, seed=m + k, ib=0)
        refs.append(oracle.helm3d_shen(f, oracle.Shen(m, bound), lam, xalp, ib=0)[0])
        r, s = gpu_ctx.device_array(f.shape), gpu_ctx.device_array(f.shape)
        r.upload(f)
        fields.append(dict(rhs=r, sol=s, xalp=xalp, alambda=lam, ib=0, bound=bound))
    gpu_ctx.solve_shen_fields_dev(fields)
    gpu_ctx.synchronize()
    for f, ref in zip(fields, refs):
        assert np.linalg.norm(f["sol"].download() - ref) < 1e-12 * np.linalg.norm(ref)
        f["rhs"].free()
        f["sol"].free()
