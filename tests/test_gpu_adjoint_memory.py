"""The adjoint where the lattice-resident form's blocks of all orders (2K - 1) do not fit beside the kets, but the
per-order form's (K + 2) do: the device is filled up to a given rest, and loss and gradients are those of an
empty device, bit for bit."""
import ctypes as C
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Filled:
    """Allocates all device memory but ``rest`` bytes (allocates only; nothing touches it)."""

    def __init__(self, rest):
        self.cu, self.rest = C.CDLL("libcuda.so.1"), rest

    def __enter__(self):
        free, total = C.c_size_t(), C.c_size_t()
        assert self.cu.cuMemGetInfo_v2(C.byref(free), C.byref(total)) == 0
        self.p = C.c_uint64()
        assert self.cu.cuMemAlloc_v2(C.byref(self.p), C.c_size_t(free.value - self.rest)) == 0

    def __exit__(self, *a):
        self.cu.cuMemFree_v2(self.p)


def _problem(lm, ctx, lib):
    Lx = Ly = 64
    N, M = Lx * Ly, 4096
    lat = lm.SquareLattice(Lx, Ly)
    dh = lm.Hamiltonian(lat, 1.0, lm.PointFlux(0.1, (32.5, 32.5)), np.linspace(-0.1, 0.1, N)).device_private(ctx)
    rng = np.random.default_rng(1)
    X = (rng.standard_normal((N, 8)) + 1j * rng.standard_normal((N, 8))).astype(np.complex64) / N
    X = np.asfortranarray(np.tile(X, (1, M // 8)))
    solver = C.c_void_p()
    ctx.check(lib.lm_solver_create(ctx.handle, 1e-9, C.byref(solver)))
    ctx.check(lib.lm_solver_update(solver, dh.handle, 0.05, 0))
    psi, lam = (lm.DeviceState(lat, X, 0, "c32", ctx=ctx) for _ in range(2))
    ctx.synchronize()
    return N, M, dh, solver, psi, lam


def _step(lm, ctx, lib, prob, rest):
    """gV, gB of one step with ``rest(K)`` blocks of memory left to the adjoint."""
    N, M, dh, solver, psi, lam = prob
    K = C.c_int()
    ctx.check(lib.lm_solver_order(solver, C.byref(K), None, None))
    adj = C.c_void_p()
    ctx.check(lib.lm_adjoint_create(ctx.handle, N, M, lm._lib.LM_C32, 1, C.byref(adj)))
    ctx.check(lib.lm_adjoint_reset(adj))
    gV, gB = np.empty(N), np.empty(1)
    try:
        with Filled(int(rest(K.value) * 8 * N * M)):
            for _ in range(2):
                ctx.check(lib.lm_adjoint_step(adj, solver, dh.handle, 0, 0, psi.handle, lam.handle))
            ctx.synchronize()
        ctx.check(lib.lm_adjoint_gradients(adj, gV.ctypes.data_as(C.POINTER(C.c_double)),
                                           gB.ctypes.data_as(C.POINTER(C.c_double))))
    finally:
        lib.lm_adjoint_destroy(adj)
    return gV, gB


def test_falls_back_to_the_per_order_form():
    import lmgpu as lm
    from lmgpu.device import Context
    out = []
    for rest in (lambda K: 2 * K + 20,    # room for all
                 lambda K: K + 2 + 1.5,   # the blocks of all orders do not fit
                 lambda K: 2 * K + 1):    # they fit, but little would be left
        ctx = Context(0)  # of its own, closed after use: a context keeps freed blocks
        prob = _problem(lm, ctx, ctx.lib)
        out.append(_step(lm, ctx, ctx.lib, prob, rest))
        ctx.lib.lm_solver_destroy(prob[3])
        del prob
        gc.collect()
        ctx.close()
    assert np.all(np.isfinite(out[0][0])) and np.any(out[0][0] != 0)
    for g in out[1:]:
        assert np.array_equal(g[0], out[0][0]) and np.array_equal(g[1], out[0][1])
