"""Order of a call's work against what the caller queued on the context's stream."""
import ctypes as C

import numpy as np
import pytest

import duct_b200 as D
from duct_b200 import synth

pytestmark = pytest.mark.gpu


class Pinned:
    """A complex array in pinned host memory."""

    def __init__(self, ctx, shape):
        self.ctx, self.p = ctx, C.c_void_p()
        n = int(np.prod(shape))
        ctx._check(D.lib().ductgpu_host_alloc(ctx.h, n * 16, C.byref(self.p)))
        flat = np.frombuffer((C.c_char * (n * 16)).from_address(self.p.value), dtype=np.complex128)
        self.a = flat.reshape(shape, order="F")

    def free(self):
        self.ctx._check(D.lib().ductgpu_host_free(self.ctx.h, self.p))


@pytest.mark.parametrize("nf", [1, 2])
def test_batch_after_a_queued_download(gpu_ctx, nf):
    """ductgpu_copy is asynchronous on the context's stream: a download into
    the pinned right-hand sides of ductgpu_helm3d_batch, queued right before
    the call and behind a long copy, is what the call solves, and the zero walls
    it leaves in them are not overwritten by the download."""
    m, nm, xalp, copy = 33, 4, 0.5 * np.arange(4), D.lib().ductgpu_copy
    gpu_ctx.pseudomat(m)
    spec = [("d", 3.0e3), ("n", 2.0)][:nf]
    host = [synth.chebyshev_rhs(m, m, nm, seed=k, ib=0) + 1.0 for k in range(nf)]
    ref = gpu_ctx.helm3d_batch([f.copy(order="F") for f in host], [b for b, _ in spec], [x for _, x in spec], xalp)
    dev, rhs = [gpu_ctx.device_array(f.shape) for f in host], [Pinned(gpu_ctx, f.shape) for f in host]
    long_dev, long_host = gpu_ctx.device_array((1 << 25,)), Pinned(gpu_ctx, (1 << 25,))     # 512 MB
    try:
        for f, d, r in zip(host, dev, rhs):
            d.upload(f)
            r.a[:] = 0.0
        gpu_ctx.synchronize()
        gpu_ctx._check(copy(gpu_ctx.h, long_host.p, C.c_void_p(long_dev.ptr), long_dev.nbytes, 2))
        for d, r in zip(dev, rhs):
            gpu_ctx._check(copy(gpu_ctx.h, r.p, C.c_void_p(d.ptr), d.nbytes, 2))
        sol = gpu_ctx.helm3d_batch([r.a for r in rhs], [b for b, _ in spec], [x for _, x in spec], xalp)
        gpu_ctx.synchronize()
        for a, b in zip(sol, ref):
            assert np.array_equal(a, b)
        for f, r, (bound, _) in zip(host, rhs, spec):
            if bound == "d":
                f[0], f[-1], f[:, 0], f[:, -1] = 0.0, 0.0, 0.0, 0.0
            assert np.array_equal(r.a, f)
    finally:
        for x in dev + rhs + [long_dev, long_host]:
            x.free()
