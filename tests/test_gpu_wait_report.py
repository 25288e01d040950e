"""The report of a bounded wait that gave up: with the context's timeout word set from the host
(lm_ctx_raise_timeout; nothing waits on the device), every call that hands values of device states to
the host returns LM_ERR_TIMEOUT, again and again, and so does a step that would wait; with the word
clear they return LM_OK, and another context is not concerned."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PD, PI = C.POINTER(C.c_double), C.POINTER(C.c_int64)


def _readers(lm, ctx):
    """name -> a call that returns the library's code."""
    lib = ctx.lib
    lat = lm.SquareLattice(9, 7)
    N = lat.N
    rng = np.random.default_rng(1)
    X = rng.standard_normal((N, 3)) + 1j * rng.standard_normal((N, 3))
    H = lm.tightbinding_hamiltonian(lat, np.linspace(-0.2, 0.2, N), field=lm.PointFlux(0.1, (4.5, 3.5)))
    dh = H.device_private(ctx)
    a, b = (lm.KetBlock(lat, X, precision="c32", ctx=ctx) for _ in range(2))
    c = lm.KetBlock(lat, X, precision="c64", ctx=ctx)
    honey = lm.HoneycombLattice(5, 4)
    G = lm.tightbinding_hamiltonian(honey, np.zeros(honey.N), field=lm.SymmetricGauge(0.01))
    g = G.device(ctx)
    k = lm.KetBlock(honey, np.ones((honey.N, 2)), precision="c64", ctx=ctx)
    out = np.zeros(1 << 16)
    p = out.ctypes.data_as(PD)
    ring = lm.timesequence.ReadoutRing(N, 4, ctx)
    ring.push_density(a, 0.0)
    n = C.c_int64()
    adj = C.c_void_p()
    ctx.check(lib.lm_adjoint_create(ctx.handle, N, 3, lm._lib.LM_C32, 1, C.byref(adj)))
    lo, hi = -5.0, 5.0
    op = np.array([1.0, 0.0])
    calls = {
        "lm_ctx_synchronize": lambda: lib.lm_ctx_synchronize(ctx.handle),
        "lm_state_download": lambda: lib.lm_state_download(a.handle, p, N),
        "lm_state_norms": lambda: lib.lm_state_norms(a.handle, p),
        "lm_trace": lambda: lib.lm_trace(a.handle, p),
        "lm_localdensity": lambda: lib.lm_localdensity(a.handle, p),
        "lm_bond_currents": lambda: lib.lm_bond_currents(dh.handle, a.handle, p),
        "lm_ring_wait": lambda: lib.lm_ring_wait(ring.handle, 0, p, None, C.byref(n), None),
        "lm_ell_currents": lambda: lib.lm_ell_currents(g.handle, k.handle, p),
        "lm_ell_op_currents": lambda: lib.lm_ell_op_currents(g.handle, k.handle, 1, op.ctypes.data_as(PD), p),
        "lm_adjoint_seed": lambda: lib.lm_adjoint_seed(adj, a.handle, p, b.handle, p),
        "lm_adjoint_gradients": lambda: lib.lm_adjoint_gradients(adj, p, p),
        "lm_kpm_moments": lambda: lib.lm_kpm_moments(dh.handle, lo, hi, 8, c.handle, 0, p),
    }
    keep = (H, dh, a, b, c, G, g, k, out, ring, op)
    return calls, keep, adj, (g, k)


def test_every_reader_reports():
    import lmgpu as lm
    from lmgpu.device import Context
    ctx, other = Context(0), Context(0)
    calls, keep, adj, (g, k) = _readers(lm, ctx)
    calls2, keep2, adj2, _ = _readers(lm, other)
    solver = C.c_void_p()
    ctx.check(ctx.lib.lm_solver_create(ctx.handle, 1e-12, C.byref(solver)))
    ctx.check(ctx.lib.lm_ell_solver_update(solver, g.handle, 0.1, 0))
    calls["lm_solver_step"] = lambda: ctx.lib.lm_solver_step(solver, k.handle)  # a cooperative step
    assert {name: call() for name, call in calls.items()} == dict.fromkeys(calls, 0)
    ctx.check(ctx.lib.lm_ctx_raise_timeout(ctx.handle))
    for _ in range(2):
        assert {name: call() for name, call in calls.items()} == dict.fromkeys(calls, lm._lib.LM_ERR_TIMEOUT)
    assert {name: call() for name, call in calls2.items()} == dict.fromkeys(calls2, 0)
    ctx.lib.lm_solver_destroy(solver)
    for c, a in ((ctx, adj), (other, adj2)):
        c.lib.lm_adjoint_destroy(a)
