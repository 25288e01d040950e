"""Device memory that a context keeps for reuse: a state's buffer can be exported to other processes
(cudaIpcGetMemHandle wants cudaMalloc memory) as created, after steps of either parity, as a copy and out of
the kept memory; what is kept is bounded, goes back with lm_ctx_trim, and makes no allocation of the library
fail on a full device."""
import ctypes as C
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cu = None


@pytest.fixture()
def ctx():
    global cu
    import lmgpu  # noqa: F401
    from lmgpu.device import Context
    cu = C.CDLL("libcuda.so.1")
    c = Context(0)
    yield c
    gc.collect()
    c.close()


def _free():
    f, t = C.c_size_t(), C.c_size_t()
    assert cu.cuMemGetInfo_v2(C.byref(f), C.byref(t)) == 0
    return f.value, t.value


def _exportable(st):
    return cu.cuIpcGetMemHandle((C.c_char * 64)(), C.c_uint64(st.device_ptr()[0])) == 0


def _state(lm, ctx, mib):
    """A ComplexF32 state of ``mib`` MiB."""
    return lm.DeviceState(lm.SquareLattice(1024, 128), None, 0, "c32", ctx=ctx, shape=(1024 * 128, mib))


@pytest.mark.parametrize("prec,kind", [("c64", 0), ("c64", 1), ("c32", 0)])
def test_state_buffers_are_exportable(ctx, prec, kind):
    import lmgpu as lm
    lat = lm.SquareLattice(21, 13)
    dh = lm.Hamiltonian(lat, 1.0, lm.PointFlux(0.1, (10.5, 6.5))).device_private(ctx)
    solver = C.c_void_p()
    ctx.check(ctx.lib.lm_solver_create(ctx.handle, 1e-12, C.byref(solver)))
    for again in range(2):  # the second time from kept memory
        st = lm.DeviceState(lat, np.ones((lat.N, lat.N if kind else 4)), kind, prec, ctx=ctx)
        assert _exportable(st)
        for dt in (0.05, 0.1, 0.15):
            ctx.check(ctx.lib.lm_solver_update(solver, dh.handle, dt, 0))
            ctx.check(ctx.lib.lm_solver_step(solver, st.handle))
            assert _exportable(st)
        c = st.copy()
        assert _exportable(c)
        ctx.synchronize()
        del st, c
        gc.collect()
    ctx.lib.lm_solver_destroy(solver)


def test_kept_memory_is_bounded_and_given_back(ctx):
    import lmgpu as lm
    ctx.synchronize()
    before, total = _free()
    slack = 64 << 20
    for mib in (1024, 1500, 2000, 900, 1024, 1300, 1700, 9000, 300):
        st = _state(lm, ctx, mib)
        del st
        gc.collect()
        assert before - _free()[0] <= total // 32 + slack
    ctx.trim()
    assert before - _free()[0] <= slack


def test_full_device(ctx):
    import lmgpu as lm
    from lmgpu.timesequence import ReadoutRing
    st = _state(lm, ctx, 3072)
    del st
    gc.collect()
    ctx.synchronize()
    fill = C.c_uint64()
    assert cu.cuMemAlloc_v2(C.byref(fill), C.c_size_t(_free()[0] - (768 << 20))) == 0
    try:
        ring = ReadoutRing(2 << 27, 1, ctx)      # 2 GiB by cudaMalloc
        del ring
        st = _state(lm, ctx, 2500)               # a state of another size than the kept one
        del st
        gc.collect()
        adj = C.c_void_p()                       # 1 GiB of partial gradients from the pool
        ctx.check(ctx.lib.lm_adjoint_create(ctx.handle, 1 << 24, 1024, lm._lib.LM_C32, 1, C.byref(adj)))
        ctx.lib.lm_adjoint_destroy(adj)
    finally:
        cu.cuMemFree_v2(fill)
