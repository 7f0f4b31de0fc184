"""Captured graphs against buffers that grow later: a call of the same context
that needs a larger workspace must leave a graph's own alone.  Results equal
those of the same calls without graphs, bit for bit, and arrays allocated after
the growth (of the sizes a wrongly freed workspace would hand out again) keep
their values over a replay."""
import ctypes as C

import numpy as np
import pytest

import duct_b200 as D
from duct_b200 import synth

pytestmark = pytest.mark.gpu


def partial_sums(m, planes):
    """Complex elements of the Neumann fill's partial sums."""
    return 2 * planes * ((m - 2 + 31) // 32) * m * 4 // 2


class Watched:
    """Arrays that nobody may write."""

    def __init__(self, ctx, sizes):
        self.a = [ctx.device_array((n,)) for n in sizes for _ in range(3)]
        for a in self.a:
            a.upload(np.full(a.shape, 7.5 - 2.5j))
        ctx.synchronize()

    def check(self):
        for a in self.a:
            assert np.all(a.download() == 7.5 - 2.5j)
            a.free()


@pytest.mark.parametrize("m", [33, 65])
def test_stepper_graphs_survive_the_gradient(m):
    """ductgpu_dns_grad_wallstress solves its adjoints in a workspace larger
    than the captured substeps' (whose solves up to 65 points a side run on chip)."""
    mg, alp = 64, 1.0
    M = mg // 3
    state = synth.dns_initial(mg, m, alp, 0.05, seed=3)[:4]
    out = []
    for graphs in (True, False):
        with D.Context(0) as ctx:
            ctx.pseudomat(m)
            with D.Dns(ctx, mg, alp, 1.0 / 2000.0, 1.0e-3) as d:
                d.set_fields(*state)
                d.set_graphs(graphs)
                d.steps(3)                 # sized, captured, replayed
                g = d.grad_wallstress()
                watched = Watched(ctx, [partial_sums(m, M), partial_sums(m, 3 * M)])
                d.steps(2)
                ctx.synchronize()
                out.append((g, d.fields()))
                watched.check()
    assert out[0][0][0] == out[1][0][0] and np.array_equal(out[0][0][1], out[1][0][1])
    for a, b in zip(out[0][1], out[1][1]):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


def test_stepper_graphs_survive_another_stepper():
    """A second stepper on the context sets up its own mass-flow coefficients;
    the first one's captured substeps keep theirs."""
    m, mg, nu, dt = 33, 64, 1.0 / 2000.0, 1.0e-3
    state = synth.dns_initial(mg, m, 1.0, 0.05, seed=3)[:4]
    out = []
    for second in (True, False):
        with D.Context(0) as ctx:
            ctx.pseudomat(m)
            with D.Dns(ctx, mg, 1.0, nu, dt) as d:
                d.set_fields(*state)
                d.steps(3)
                if second:
                    with D.Dns(ctx, mg, 1.0, 2.0 * nu, 0.5 * dt) as e:
                        e.set_fields(*state)
                        e.steps(3)
                watched = Watched(ctx, [3 * m * m // 2, 3 * m * m, 128])
                d.steps(3)
                ctx.synchronize()
                out.append(d.fields())
                watched.check()
    for a, b in zip(*out):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


@pytest.mark.parametrize("m,kernel", [(65, -1), (129, -1), (129, D.PASS_PARITY_QUEUE)])
def test_solve_graph_survives_a_larger_solve(m, kernel):
    """A graph of three Dirichlet fields and a Neumann one, then a direct
    Neumann solve with more partial sums, then the graph again, after another
    graph was created and destroyed on the larger workspace."""
    nm = 21 if kernel < 0 else 5
    with D.Context(0) as ctx:
        ctx.pseudomat(m)
        ctx.set_pass_kernel(kernel)

        def field(bound, lam, n, seed):
            f = synth.chebyshev_rhs(m, m, n, seed=seed, ib=0)
            r, s = ctx.device_array(f.shape), ctx.device_array(f.shape)
            r.upload(f)
            return dict(rhs=r, sol=s, xalp=0.5 * np.arange(n), alambda=lam, ib=0, bound=bound)

        fields = [field(b, x, nm, k) for k, (b, x) in enumerate((("d", 4e3), ("d", 1.0), ("d", 9.0), ("n", 0.0)))]
        ctx.solve_fields_dev(fields)
        ctx.synchronize()
        ref = [f["sol"].download() for f in fields]
        gid = ctx.graph_create(fields)
        larger = [field("n", 0.0, 4 * nm + 40, 9)]
        ctx.solve_fields_dev(larger)
        other = ctx.graph_create(larger)
        ctx.graph_launch(other)
        ctx.graph_destroy(other)
        watched = Watched(ctx, [partial_sums(m, nm), 4 * nm * m * m * 2])
        for f in fields:
            f["sol"].upload(np.zeros(f["sol"].shape, dtype=complex, order="F"))
        for _ in range(2):
            ctx.graph_launch(gid)
        ctx.synchronize()
        for f, a in zip(fields, ref):
            assert np.array_equal(f["sol"].download(), a)
        watched.check()
        ctx.graph_destroy(gid)
        ctx.solve_fields_dev(fields)
        ctx.synchronize()
        for f, a in zip(fields, ref):
            assert np.array_equal(f["sol"].download(), a)


@pytest.mark.parametrize("kind", ["square", "rect", "shen"])
def test_solve_refused_inside_a_callers_capture(kind):
    """lambda and the workspaces move as later calls grow them, so a solve may
    not go into a graph that the library does not know; the capture and the
    context stay usable."""
    torch = pytest.importorskip("torch")
    m, nm = 33, 3
    with D.Context(0) as ctx:
        ctx.pseudomat(m)
        ctx.pseudomat_temp(0, m, m)
        ctx.preshen(m, "d")
        f = synth.chebyshev_rhs(m, m, nm, seed=1, ib=0)
        r, s = ctx.device_array(f.shape), ctx.device_array(f.shape)
        r.upload(f)
        fields = [dict(rhs=r, sol=s, xalp=0.5 * np.arange(nm), alambda=3.0, ib=0, bound="d", slot=0)]
        solve = dict(square=ctx.solve_fields_dev, rect=ctx.solve_rect_fields_dev, shen=ctx.solve_shen_fields_dev)[kind]
        side, graph, x = torch.cuda.Stream(), torch.cuda.CUDAGraph(), torch.zeros(8, device="cuda")
        ctx._check(D.lib().ductgpu_set_stream(ctx.h, C.c_void_p(side.cuda_stream)))
        ctx.synchronize()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            x += 1.0
            with pytest.raises(D.DuctGPUError):
                solve(fields)
            x += 1.0
        graph.replay()
        torch.cuda.synchronize()
        assert float(x[0]) == 2.0
        solve(fields)
        ctx.synchronize()
        assert np.all(np.isfinite(s.download()))
        del graph
        ctx._check(D.lib().ductgpu_set_stream(ctx.h, None))
        r.free()
        s.free()
