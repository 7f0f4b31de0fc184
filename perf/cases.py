"""What a user of this library has it do, as timed cases.

Each case is a dict of plain values; `listed` gives the named ones, `draw`
more of the same ranges.  `prepare` makes what a program holds before the
call (fields in device memory, a context with its operators, a captured
graph or a stepper), `run` is one call of the public entry points, `exact`
the same result from dense 64-bit linear algebra, written from the
discrete equations without this library.

Fields are complex (my, mz, nmodes), y fastest: a torch tensor of shape
(nmodes, mz, my).
"""
import ctypes as C
import math

import numpy as np
import torch

import duct_b200 as D

DEV = "cuda"
NU, DT = 1.0 / 2000.0, 1.0e-3            # the solve batches: lambda = kx^2 + 2 / (nu dt)


# ---- the cases -----------------------------------------------------------
def listed():
    return [
        # one Dirichlet field of a small duct in a direct call: all latency
        dict(name="solve_33", kind="solve", my=33, modes=17, fields="d", graph=False),
        # u, v, w and the pressure of a substep at a small size, direct calls
        dict(name="solve_65", kind="solve", my=65, modes=21, fields="dddn", graph=False),
        # the same at the benchmark's size, replayed from a captured graph
        dict(name="solve_129", kind="solve", my=129, modes=64, fields="dddn", graph=True),
        # the largest square grid with the modes of a 256-point streamwise DNS
        dict(name="solve_193", kind="solve", my=193, modes=85, fields="dddn", graph=False),
        # four ducts of different aspect ratios in one batch (uneven sizes)
        dict(name="rect_4ducts", kind="rect", ducts="65x65x32,65x129x48,49x145x64,33x129x96", graph=True),
        # the backward (adjoint) solve of u, v, w, p: the gradient of a step
        dict(name="adjoint_65", kind="adjoint", my=65, modes=21, fields="dddn"),
        # the Shen-Legendre solver on the benchmark's batch
        dict(name="shen_129", kind="shen", my=129, modes=64, fields="dddn"),
        # transforms, derivatives and pencil transposes called one by one
        dict(name="transforms_193", kind="transforms", my=193, mz=193, modes=85),
        # the operators of a host-driven time step: advection, laplacian, gradient, divergence
        dict(name="operators_97", kind="operators", my=97, mz=97, mgalx=144),
        # the drop-in for the Fortran code: fields in pinned host memory
        dict(name="host_129", kind="host", my=129, modes=64, fields="dddn"),
        # one RK3/CN time step of a small DNS, and of the large one with statistics
        dict(name="dns_65", kind="dns", my=65, mgalx=64, stats=0),
        dict(name="dns_193", kind="dns", my=193, mgalx=256, stats=1),
    ]


LINES = [17, 25, 33, 49, 65, 97, 129, 145, 193]     # my - 1 the transforms take: 16 .. 192


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "rect", "adjoint", "shen", "transforms", "operators", "host", "dns"])
    if kind in ("solve", "adjoint", "host"):
        my = _log(rng, 17, 193)                          # odd and even sizes
        modes = _log(rng, 3, 85)
        c = dict(kind=kind, my=my, modes=modes, fields=rng.choice(["d", "n", "ddd", "dddn"]))
        if kind == "solve":
            c["graph"] = rng.random() < 0.5
        return c
    if kind == "rect":
        n = rng.randint(1, 4)
        return dict(kind=kind, graph=rng.random() < 0.5,
                    ducts=",".join("%dx%dx%d" % (_log(rng, 17, 145), _log(rng, 17, 145), _log(rng, 4, 64)) for _ in range(n)))
    if kind == "shen":
        return dict(kind=kind, my=rng.choice([m for m in LINES if 25 <= m < 190]), modes=_log(rng, 3, 64),
                    fields=rng.choice(["d", "n", "dddn"]))
    if kind == "transforms":
        return dict(kind=kind, my=rng.choice(LINES), mz=rng.choice(LINES), modes=_log(rng, 4, 85))
    if kind == "operators":
        return dict(kind=kind, my=rng.choice(LINES), mz=rng.choice(LINES), mgalx=rng.choice([64, 144, 256]))
    return dict(kind=kind, my=rng.choice([33, 49, 65, 97, 129, 145]), mgalx=rng.choice([64, 144, 256]),
                stats=rng.choice([0, 1]))


# ---- common pieces -------------------------------------------------------
class Field(D.DeviceArray):
    """A torch tensor as the library's device array."""

    def __init__(self, ctx, t):
        self.ctx, self.t, self.ptr = ctx, t, t.data_ptr()
        self.shape, self.dtype = tuple(reversed(t.shape)), np.dtype(np.complex128)
        self.nbytes = t.numel() * 16


class State(dict):
    """What a program holds; a captured graph goes back when it goes."""

    def __del__(self):
        if self.get("gid") is not None:
            self["ctx"].graph_destroy(self["gid"])


class Stepper(D.Dns):
    """A time stepper that goes back when nothing refers to it any more (its
    own context and the tensors that view its fields refer to it)."""

    def __del__(self):
        self.close()


class Context(D.Context):
    def __del__(self):
        self.close()


_contexts = {}


def _context(key, setup):
    """One context per grid, set up once, as a program keeps it."""
    if key not in _contexts:
        if len(_contexts) >= 6:
            _contexts.pop(next(iter(_contexts)))
        ctx = Context(torch.cuda.current_device())
        setup(ctx)
        _contexts[key] = ctx
    return _contexts[key]


def _square(my):
    def setup(ctx):
        ctx.pseudomat(my)
        ctx.set_gauge_point(_pin(my))
    return _context(("square", my), setup)


def _pin(my):
    return (my - 2) // 2        # 1-based interior index of the kx = 0 pressure's fixed point


def _c(t):
    return t.to(torch.complex128)


def _rhs(gen, my, mz, modes, real0=True):
    """Chebyshev coefficients N(0,1) + i N(0,1) over ((1+i)(1+j))^2, at the nodes."""
    c = torch.randn(modes, mz, my, 2, generator=gen, device=DEV, dtype=torch.float64)
    i = 1.0 + torch.arange(my, device=DEV, dtype=torch.float64)
    j = 1.0 + torch.arange(mz, device=DEV, dtype=torch.float64)
    c = torch.view_as_complex(c) / (j[:, None] * i[None, :]) ** 2
    f = _c(_cheb(mz)) @ c @ _c(_cheb(my)).T
    if real0:
        f[0] = f[0].real.to(f.dtype)
    return f.contiguous()


def _cheb(m):
    p = torch.arange(m, device=DEV, dtype=torch.float64)
    return torch.cos(math.pi * torch.remainder(p[:, None] * p[None, :], 2 * (m - 1)) / (m - 1))


def _lambda(bound):
    return 0.0 if bound == "n" else 2.0 / (NU * DT)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _ducts(case):
    return [tuple(int(x) for x in d.split("x")) for d in case["ducts"].split(",")]


def _solve_inputs(case, seed):
    gen = _gen(seed)
    return [_rhs(gen, case["my"], case["my"], case["modes"]) for _ in case["fields"]]


def _rect_inputs(case, seed):
    gen = _gen(seed)
    out = [[_rhs(gen, my, mz, nm) for _ in range(4)] for my, mz, nm in _ducts(case)]
    for f in (f for d in out for f in d):
        f[:, ::f.shape[1] - 1, ::f.shape[2] - 1] = 0     # corners go through to the solution
    return out


def _rect_lambda(neumann):
    return 0.0 if neumann else 2.0 / ((1.0 / 4400.0) * 5.0e-4)


def _modes(mgalx):
    return mgalx // 3           # the 2/3 rule


def _operator_inputs(case, seed):
    gen = _gen(seed)
    return [_rhs(gen, case["my"], case["mz"], _modes(case["mgalx"])) for _ in range(4)]


def _dns_numbers(case):
    return dict(alp=0.5, fnu=1.9081638750 / (4.0 * 4400.0), dt=2.0e-4)


def _dns_inputs(case, seed):
    """The laminar profile (max 1) plus a divergence-free perturbation of
    10 % in the lowest modes: the curl of a potential that vanishes with
    its slope on the walls."""
    my, M, alp = case["my"], _modes(case["mgalx"]), _dns_numbers(case)["alp"]
    x, d1 = _nodes(my)
    lam_u = _lam_plane(my)
    kk, nt = min(8, M - 1), 4
    r = torch.view_as_complex(torch.randn(3, kk + 1, nt, nt, 2, generator=_gen(seed), device=DEV, dtype=torch.float64))
    r[:, 0] = r[:, 0].real.to(r.dtype)
    t = torch.cos(torch.arange(nt, device=DEV)[None, :] * torch.arccos(x.clamp(-1, 1))[:, None])
    bub = (1 - x * x) ** 2
    psi = torch.einsum("za,ckab,yb->ckzy", _c(t), r, _c(t)) * (bub[:, None] * bub[None, :])
    ik = 1j * alp * torch.arange(kk + 1, device=DEV, dtype=torch.float64)[:, None, None]
    dy, dz = (lambda f: f @ _c(d1).T), (lambda f: _c(d1) @ f)
    per = [dy(psi[2]) - dz(psi[1]), dz(psi[0]) - ik * psi[2], ik * psi[1] - dy(psi[0])]
    mag = sum(torch.fft.irfft(p, n=4 * (kk + 1), dim=0, norm="forward") ** 2 for p in per).sqrt().max()
    out = []
    for c in range(4):
        f = torch.zeros(M, my, my, device=DEV, dtype=torch.complex128)
        if c < 3:
            f[: kk + 1] = per[c] * (0.1 / mag)
            f[0] = f[0].real.to(f.dtype)
        if c == 0:
            f[0] += lam_u
        f[:, 0], f[:, -1], f[:, :, 0], f[:, :, -1] = 0, 0, 0, 0
        out.append(f)
    return out


class _Raw:
    """Device memory of the library seen as a torch tensor, which keeps the
    owner of that memory."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<c16", data=(ptr, False), version=3, strides=None)


# ---- prepare / run -------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "adjoint", "shen", "host"):
        my, modes = case["my"], case["modes"]
        xalp = 0.5 * np.arange(modes)
        rhs = _solve_inputs(case, seed)
        if kind == "host":
            ctx = _square(my)
            pin = [t.cpu().pin_memory() for t in rhs]
            sol = [torch.zeros_like(t).pin_memory() for t in pin]
            n = len(pin)
            return State(ctx=ctx, rhs=pin, sol=sol, xalp=xalp, n=n, bounds=case["fields"].encode(),
                         lam=np.array([_lambda(b) for b in case["fields"]]),
                         pr=(C.c_void_p * n)(*[t.data_ptr() for t in pin]),
                         ps=(C.c_void_p * n)(*[t.data_ptr() for t in sol]))
        if kind == "shen":
            ctx = _context(("shen", my), lambda c: (c.preshen(my, "d"), c.preshen(my, "n")))
        else:
            ctx = _square(my)
        sol = [torch.zeros_like(t) for t in rhs]
        fields = [dict(rhs=Field(ctx, r), sol=Field(ctx, s), xalp=xalp, alambda=_lambda(b), ib=0, bound=b)
                  for r, s, b in zip(rhs, sol, case["fields"])]
        torch.cuda.synchronize()
        gid = ctx.graph_create(fields) if case.get("graph") else None
        # the Shen entry overwrites its right-hand sides, so a program fills them for each call
        src = [r.clone() for r in rhs] if kind == "shen" else None
        return State(ctx=ctx, rhs=rhs, sol=sol, fields=fields, gid=gid, src=src, adjoint=(kind == "adjoint"))
    if kind == "rect":
        ducts = _ducts(case)

        def setup(ctx):
            for i, (my, mz, nm) in enumerate(ducts):
                ctx.pseudomat_temp(i, my, mz, 1.0, 1.0 + i)
                ctx.pseudomat_temp(4 + i, my, mz, 1.0, 1.0 + i, ("n", "n"), ("n", "n"))

        ctx = _context(("rect", case["ducts"]), setup)
        rhs = _rect_inputs(case, seed)
        sol = [[torch.zeros_like(t) for t in d] for d in rhs]
        fields = [dict(rhs=Field(ctx, rhs[i][k]), sol=Field(ctx, sol[i][k]), xalp=1.0 * np.arange(nm),
                       alambda=_rect_lambda(k == 3), ib=0, slot=i + (4 if k == 3 else 0))
                  for i, (my, mz, nm) in enumerate(ducts) for k in range(4)]
        torch.cuda.synchronize()
        gid = ctx.graph_create(fields, rect=True) if case["graph"] else None
        return State(ctx=ctx, rhs=rhs, sol=sol, fields=fields, gid=gid)
    if kind == "transforms":
        ctx = _context("lines", lambda c: None)
        f = _rhs(_gen(seed), case["my"], case["mz"], case["modes"])
        return State(ctx=ctx, f=f, dy=torch.zeros_like(f), dz=torch.zeros_like(f),
                     cut=torch.zeros(case["mz"], case["my"], case["modes"], device=DEV, dtype=torch.complex128),
                     back=torch.zeros_like(f))
    if kind == "operators":
        ctx = _context("lines", lambda c: None)
        fs = _operator_inputs(case, seed)
        M = _modes(case["mgalx"])
        big = torch.zeros(5 * M, case["mz"], case["my"], device=DEV, dtype=torch.complex128)
        out = [torch.zeros_like(fs[0]) for _ in range(8)]
        return State(ctx=ctx, fs=fs, out=out, work=big, F=[Field(ctx, t) for t in fs],
                     O=[Field(ctx, t) for t in out], W=Field(ctx, big), xalp=0.5 * np.arange(M))
    my, nums = case["my"], _dns_numbers(case)
    ctx = _square(my)
    d = Stepper(ctx, case["mgalx"], nums["alp"], nums["fnu"], nums["dt"], cmassflow=True, hist_cap=64)
    st = State(ctx=ctx, dns=d, stats=case["stats"])
    fs = _dns_inputs(case, seed)
    torch.cuda.synchronize()
    ctx._check(D.lib().ductgpu_dns_set_fields(d.h, *[C.c_void_p(t.data_ptr()) for t in fs]))
    st["out"] = [torch.as_tensor(_Raw(d, d.field_ptr(k), tuple(fs[0].shape)), device=DEV) for k in range(4)]
    return st


def run(state):
    ctx, L = state["ctx"], D.lib()
    if "dns" in state:
        state["dns"].steps(1, stats_every=state["stats"])
        return state["out"]
    if "pr" in state:
        my, modes = state["rhs"][0].shape[1], state["rhs"][0].shape[0]
        ctx._check(L.ductgpu_helm3d_batch(ctx.h, state["n"], C.cast(state["pr"], C.c_void_p),
                                          C.cast(state["ps"], C.c_void_p), state["bounds"],
                                          state["lam"].ctypes.data_as(C.c_void_p), my, my, 0, modes - 1,
                                          state["xalp"].ctypes.data_as(C.c_void_p), D.PREC_FP64))
        return state["sol"]
    if "cut" in state:
        f, dy, dz, cut, back = (state[k] for k in ("f", "dy", "dz", "cut", "back"))
        modes, mz, my = f.shape
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        for c, du in ((b"y", dy), (b"z", dz)):
            ctx._check(L.ductgpu_transyz_dev(ctx.h, p(f), my, mz, modes, c, -1))
            ctx._check(L.ductgpu_derivyz_dev(ctx.h, p(f), p(du), my, mz, modes, c, 1, 1.0, b"n", 1.0))
            ctx._check(L.ductgpu_transyz_dev(ctx.h, p(du), my, mz, modes, c, 1))
            ctx._check(L.ductgpu_transyz_dev(ctx.h, p(f), my, mz, modes, c, 1))
        ctx._check(L.ductgpu_cyzx2xyz_dev(ctx.h, p(cut), p(dy), modes, my, mz))
        ctx._check(L.ductgpu_cxyz2yzx_dev(ctx.h, p(cut), p(back), modes, my, mz))
        return [f, dy, dz, cut, back]
    if "W" in state:
        F, O, W, xalp = state["F"], state["O"], state["W"], state["xalp"]
        M = len(xalp)
        ctx.advection3d_dev(F[0], F[1], F[2], O[0], O[1], O[2], W, _mgalx(M), xalp)
        ctx.laplacian3d_dev(F[0], O[3], xalp, NU)
        ctx.grad3d_dev(F[3], O[4], O[5], O[6], xalp, -1.0)
        ctx.div3d_dev(F[0], F[1], F[2], O[7], xalp, 1.0)
        return state["out"]
    if state["gid"] is not None:
        ctx.graph_launch(state["gid"])
        return state["sol"]
    fields = state["fields"]
    if state.get("src") is not None:
        for r, s in zip(state["rhs"], state["src"]):
            ctx._check(L.ductgpu_copy(ctx.h, C.c_void_p(r.data_ptr()), C.c_void_p(s.data_ptr()), r.numel() * 16, 3))
        ctx.solve_shen_fields_dev(fields)
        return [state["sol"], state["rhs"]]
    if "slot" in fields[0]:
        ctx.solve_rect_fields_dev(fields)
    elif state.get("adjoint"):
        ctx.solve_adjoint_fields_dev(fields)
    else:
        ctx.solve_fields_dev(fields)
    return state["sol"]


def _mgalx(M):
    return {21: 64, 48: 144, 85: 256}[M]


# ---- work and tolerance --------------------------------------------------
def work(case):
    """Inputs read once, outputs written once; the flops of the half-size
    (even / odd) operator products of a solve, and of fast transforms where
    those do (a complex line of n points: 10 n log2 n for a transform pair
    with its recurrence)."""
    kind = case["kind"]

    def mode_solve(my, mz):
        def half(n):
            return (n + 1) // 2, n // 2
        (a, b), (c, d) = half(my - 2), half(mz - 2)
        return 8.0 * ((mz - 2) * (a * a + b * b) + (my - 2) * (c * c + d * d))

    def lines(my, mz, k):
        return k * my * mz * 10.0 * math.log2(my)

    if kind in ("solve", "adjoint", "host", "shen"):
        pl = len(case["fields"]) * case["modes"]
        pts = case["my"] ** 2
        if kind == "shen":
            # right-hand side read, its coefficients and the solution written
            return dict(bytes=48.0 * pts * pl, flops=pl * (1.5 * mode_solve(case["my"], case["my"]) + lines(case["my"], case["my"], 4)))
        return dict(bytes=32.0 * pts * pl, flops=pl * mode_solve(case["my"], case["my"]))
    if kind == "rect":
        return dict(bytes=sum(4 * 32.0 * my * mz * nm for my, mz, nm in _ducts(case)),
                    flops=sum(4 * nm * mode_solve(my, mz) for my, mz, nm in _ducts(case)))
    if kind == "transforms":
        pts = case["my"] * case["mz"] * case["modes"]
        return dict(bytes=96.0 * pts, flops=2 * case["modes"] * lines(case["my"], case["mz"], 1))
    M = _modes(case["mgalx"])
    mz = case.get("mz", case["my"])
    pts = case["my"] * mz * M
    fft = 9 * case["my"] * mz * 2.5 * case["mgalx"] * math.log2(case["mgalx"])
    if kind == "operators":
        return dict(bytes=16.0 * pts * 12, flops=fft + M * lines(case["my"], mz, 12))
    # a step: three substeps, each reads u, v, w, p and the old advection
    # terms and writes u, v, w, p and the new ones
    return dict(bytes=3 * 14 * 16.0 * pts,
                flops=3 * (fft + M * lines(case["my"], case["my"], 22) + 4 * M * mode_solve(case["my"], case["my"])))


def tolerance(case):
    """64-bit sums.  What one order of summation differs from another by is
    set by the conditioning: a Dirichlet solve with the viscous lambda loses
    little (1e-14 measured), a Neumann one up to n^4 eps of the operator
    (4e-11), a derivative n^2 eps (7e-12 through the transforms)."""
    neumann = dict(rel=2e-10, max=1e-7)
    if case["kind"] in ("solve", "host", "adjoint"):
        return neumann if "n" in case["fields"] else dict(rel=2e-13, max=1e-10)
    return {"rect": neumann, "shen": dict(rel=2e-12, max=1e-9), "transforms": dict(rel=4e-11, max=1e-8),
            "operators": dict(rel=4e-12, max=1e-9), "dns": neumann}[case["kind"]]


# ---- the same results from dense 64-bit linear algebra ---------------------
_dense = {}


def _nodes(m, s=1.0):
    """Ascending Gauss-Lobatto points on [-s, s] and their derivative matrix
    (differences of nodes by the sine formula, diagonal by row sums)."""
    key = ("nodes", m, s)
    if key not in _dense:
        n = m - 1
        j = np.arange(m)
        x = -np.cos(np.pi * j / n)
        w = np.where((j == 0) | (j == n), 2.0, 1.0) * (-1.0) ** j
        dx = 2.0 * np.sin(np.pi * (j[:, None] + j[None, :]) / (2 * n)) * np.sin(np.pi * (j[:, None] - j[None, :]) / (2 * n))
        d = w[:, None] / w[None, :] / (dx + np.eye(m))
        d[j, j] = 0.0
        d[j, j] = -d.sum(axis=1)
        _dense[key] = (torch.tensor(s * x, device=DEV), torch.tensor(d / s, device=DEV))
    return _dense[key]


def _eig(m, bound, s=1.0):
    """(E, P, P^-1, W): eigen-decomposition of the interior second derivative
    and the map W (m x m-2) from interior values to all points."""
    key = ("eig", m, bound, s)
    if key not in _dense:
        d = _nodes(m, s)[1].cpu().numpy()
        w = np.zeros((m, m - 2))
        w[1:-1] = np.eye(m - 2)
        if bound == "n":
            w[[0, -1]] = -np.linalg.solve(d[np.ix_([0, -1], [0, -1])], d[[0, -1]][:, 1:-1])
        b = (d @ d)[1:-1] @ w
        b = 0.5 * (b + b[::-1, ::-1])
        e, p = np.linalg.eig(b)
        e, p = e.real.copy(), p.real.copy()
        _dense[key] = tuple(torch.tensor(a, device=DEV) for a in (e, p, np.linalg.inv(p), w))
    return _dense[key]


def _helm(f, bound, lam, sy=1.0, sz=1.0, pin=None, real0=True, transpose=False):
    """(d_yy + d_zz - lam_k) u = f of a field (modes, mz, my), lam (modes,)."""
    ey, py, qy, wy = _eig(f.shape[2], bound, sy)
    ez, pz, qz, wz = _eig(f.shape[1], bound, sz)
    py, qy, wy, pz, qz, wz = (_c(t) for t in (py, qy, wy, pz, qz, wz))
    den = ez[:, None] + ey[None, :] - lam[:, None, None]
    if bound == "n":
        k, j = int(ez.abs().argmin()), int(ey.abs().argmin())
        den[lam.abs() <= 1e-10, k, j] = math.inf
    if transpose:
        g = f.clone()
        if real0:
            g[0] = g[0].real.to(g.dtype)
        if bound == "n" and pin is not None:
            for i in torch.nonzero(lam.abs() <= 1e-10).flatten().tolist():
                g[i, pin, pin] -= g[i].sum()
        g = wz.T @ g @ wy
        g = qz.T @ ((pz.T @ g @ py) / den) @ qy
        out = torch.zeros_like(f)
        out[:, 1:-1, 1:-1] = g
    else:
        u = pz @ ((qz @ f[:, 1:-1, 1:-1] @ qy.T) / den) @ py.T
        out = wz @ u @ wy.T
        if bound == "n" and pin is not None:
            for i in torch.nonzero(lam.abs() <= 1e-10).flatten().tolist():
                out[i] -= out[i, pin, pin].clone()
    if real0:
        out[0] = out[0].real.to(out.dtype)
    return out


def _lam_plane(my):
    """The laminar profile of the square duct, max 1."""
    key = ("laminar", my)
    if key not in _dense:
        one = -torch.ones(1, my, my, device=DEV, dtype=torch.complex128)
        w = _helm(one, "d", torch.zeros(1, device=DEV, dtype=torch.float64))[0]
        _dense[key] = w / w.real.max()
    return _dense[key]


def _weights(m):
    """Clenshaw-Curtis weights on [-1, 1]."""
    n = m - 1
    k = np.arange(m)
    t = np.cos(np.pi * np.outer(k, k) / n)               # T_k at the nodes
    mom = np.where(k % 2 == 0, 2.0 / (1.0 - np.where(k % 2 == 0, k, 0) ** 2.0), 0.0)
    return torch.tensor(np.linalg.solve(t, mom), device=DEV)


def _shen(f, bound, lam):
    """-lap u + lam u = f in the Legendre-Galerkin space of the wall
    condition: (u, Chebyshev coefficients of f)."""
    m = f.shape[2]
    n = m - 2
    key = ("shen", m, bound)
    if key not in _dense:
        t = _cheb(m).cpu().numpy()
        leg = np.polynomial.legendre.legvander(np.cos(np.pi * np.arange(m) / (m - 1)), m - 1)
        k = np.arange(n)
        b = -np.ones(n) if bound == "d" else -k * (k + 1.0) / ((k + 2.0) * (k + 3.0))
        e = np.zeros((m, n))
        e[k, k], e[k + 2, k] = 1.0, b                    # basis functions in Legendre coefficients
        mass = e.T @ np.diag(2.0 / (2 * np.arange(m) + 1)) @ e
        stiff = np.diag(-b * (4 * k + 6.0))
        l = np.linalg.cholesky(mass)
        li = np.linalg.inv(l)
        s, q = np.linalg.eigh(li @ stiff @ li.T)
        _dense[key] = tuple(torch.tensor(a, device=DEV) for a in (
            np.linalg.inv(t), e.T @ np.diag(2.0 / (2 * np.arange(m) + 1)) @ np.linalg.inv(leg), leg @ e, s, li.T @ q))
    ti, proj, back, s, x = _dense[key]
    cheb = _c(ti) @ f @ _c(ti).T
    g = _c(x).T @ (_c(proj) @ f @ _c(proj).T) @ _c(x)
    den = s[:, None] + s[None, :] + lam[:, None, None]
    sing = [i for i in torch.nonzero(lam.abs() <= 1e-10).flatten().tolist() if bound == "n"]
    for i in sing:
        den[i, 0, 0] = math.inf
    c = _c(x) @ (g / den) @ _c(x).T
    for i in sing:
        c[i, 0, 0] = 0.0                                 # the constant mode is pinned to zero
    u = _c(back) @ c @ _c(back).T
    u[0] = u[0].real.to(u.dtype)
    return u, cheb


def _ops(my, mz, M, alp):
    dy, dz = _c(_nodes(my)[1]), _c(_nodes(mz)[1])
    ik = 1j * alp * torch.arange(M, device=DEV, dtype=torch.float64)[:, None, None]
    return (lambda f: ik * f), (lambda f: f @ dy.T), (lambda f: dz @ f)


def _advection(u, v, w, N, ops):
    dx, dy, dz = ops
    M = u.shape[0]
    pad = torch.zeros(N // 2 + 1 - M, *u.shape[1:], device=DEV, dtype=u.dtype)

    def phys(f):
        return torch.fft.irfft(torch.cat([f, pad]), n=N, dim=0, norm="forward")

    def spec(a, b):
        return torch.fft.rfft(a * b, dim=0, norm="forward")[:M]

    a, b, c = phys(u), phys(v), phys(w)
    uv, uw, vw = spec(a, b), spec(a, c), spec(b, c)
    return [dx(spec(a, a)) + dy(uv) + dz(uw), dx(uv) + dy(spec(b, b)) + dz(vw), dx(uw) + dy(vw) + dz(spec(c, c))]


def _dns_step(case, fs):
    """One RK3/Crank-Nicolson step with the flow rate held."""
    nums = _dns_numbers(case)
    alp, nu, dt, my, N = nums["alp"], nums["fnu"], nums["dt"], case["my"], case["mgalx"]
    u, v, w, p = [f.clone() for f in fs]
    M = u.shape[0]
    ops = dx, dy, dz = _ops(my, my, M, alp)
    kx2 = (alp * torch.arange(M, device=DEV, dtype=torch.float64)) ** 2
    wc = _weights(my)
    flow = lambda f: (wc[:, None] * wc[None, :] * f[0].real).sum()  # noqa: E731
    lap = lambda f: dx(dx(f)) + dy(dy(f)) + dz(dz(f))  # noqa: E731
    csum, old = flow(u), None
    for a, b, g, r in zip((29 / 96, -3 / 40, 1 / 6), (37 / 160, 5 / 24, 1 / 6), (8 / 15, 5 / 12, 3 / 4), (0, -17 / 60, -5 / 12)):
        adv = _advection(u, v, w, N, ops)
        grad = [dx(p), dy(p), dz(p)]
        h = [f / dt + a * nu * lap(f) - g * adv[c] - (a + b) * grad[c] for c, f in enumerate((u, v, w))]
        if old is not None:
            h = [x - r * o for x, o in zip(h, old)]
        old = adv
        hel = 1.0 / (b * nu * dt)
        u, v, w = [_helm(-x / (nu * b), "d", kx2 + hel) for x in h]
        phi = _helm((dx(u) + dy(v) + dz(w)) / ((a + b) * dt), "n", kx2, pin=_pin(my))
        p = p + phi - (a + b) * dt * nu * lap(phi)
        u, v, w = [f - dt * (a + b) * d(phi) for f, d in zip((u, v, w), ops)]
        one = _helm(torch.ones(1, my, my, device=DEV, dtype=u.dtype), "d", torch.full((1,), hel, device=DEV, dtype=torch.float64))
        u[0] += (csum - flow(u)) / flow(one) * one[0]
    return [u, v, w, p]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "adjoint", "shen", "host"):
        kx2 = (0.5 * torch.arange(case["modes"], device=DEV, dtype=torch.float64)) ** 2
        rhs = _solve_inputs(case, seed)
        if kind == "shen":
            got = [_shen(f, b, kx2 + _lambda(b)) for f, b in zip(rhs, case["fields"])]
            return [[g[0] for g in got], [g[1] for g in got]]
        out = [_helm(f, b, kx2 + _lambda(b), pin=_pin(case["my"]), transpose=(kind == "adjoint"))
               for f, b in zip(rhs, case["fields"])]
        return [t.cpu() for t in out] if kind == "host" else out
    if kind == "rect":
        out = []
        for i, fs in enumerate(_rect_inputs(case, seed)):
            kx2 = torch.arange(fs[0].shape[0], device=DEV, dtype=torch.float64) ** 2
            out.append([_helm(f, "n" if k == 3 else "d", kx2 + _rect_lambda(k == 3), 1.0, 1.0 + i) for k, f in enumerate(fs)])
            for f in out[-1]:
                f[:, ::f.shape[1] - 1, ::f.shape[2] - 1] = 0
        return out
    if kind == "transforms":
        f = _rhs(_gen(seed), case["my"], case["mz"], case["modes"])
        _, dy, dz = _ops(case["my"], case["mz"], case["modes"], 0.0)
        return [f, dy(f), dz(f), dy(f).permute(1, 2, 0).contiguous(), dy(f)]
    if kind == "operators":
        u, v, w, p = _operator_inputs(case, seed)
        ops = dx, dy, dz = _ops(case["my"], case["mz"], u.shape[0], 0.5)
        return _advection(u, v, w, case["mgalx"], ops) + [NU * (dx(dx(u)) + dy(dy(u)) + dz(dz(u))), -dx(p), -dy(p), -dz(p),
                                                          dx(u) + dy(v) + dz(w)]
    return _dns_step(case, _dns_inputs(case, seed))
