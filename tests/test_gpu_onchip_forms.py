"""The on-chip forms where they are known to run: the number of launches (or the counter of the
lattice-resident form) tells that the form ran in one arm and not in the other, so that no case compares the
fallback with itself.

* the ComplexF64 step at every block shape (one to twelve columns per thread; kets: one per SM, which the launch
  rule always takes on chip) against the per-order kernels, 1e-14 as in the other tests of the form;
* lm_cheb_apply in double-float with one and two kets per CTA against the FP64 recurrence, 1e-12;
* the lattice-resident ComplexF32 step and adjoint, bit for bit against the region form and the per-order kernels."""
import ctypes as C

import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lm():
    import lmgpu
    return lmgpu


@pytest.fixture(scope="module")
def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def ham(lm, Lx, Ly, field, per=None, t1=-1.3):
    lat = lm.SquareLattice(Lx, Ly, boundaries=per)
    f = {"landau": lm.LandauGauge(0.03), "sum": lm.SymmetricGauge(0.02) + lm.PointFlux(0.3, (1.5, Ly / 2)),
         "flux": lm.PointFlux(0.2, (Lx // 2 + 0.5, Ly // 2 + 0.5), "singular" if per else "axial")}[field]
    return lat, lm.tightbinding_hamiltonian(lat, o.anderson_disorder(lat.N, 1.0, 4), t1=t1, field=f)


# columns per thread 1, 2, 3, 3, 5, 5, 8, 8, 9, 10, 11, 12 (several CTAs per SM up to 8, one beyond)
STEP = [(12, 10, "flux", None), (5, 60, "sum", None), (11, 33, "landau", {"axis2": True}), (24, 24, "flux", None),
        (19, 41, "sum", {"axis2": 0.7}), (32, 27, "flux", None), (31, 47, "flux", None), (47, 31, "sum", None),
        (26, 110, "flux", None), (30, 100, "sum", None), (64, 62, "flux", None), (34, 110, "sum", None)]


@pytest.mark.parametrize("Lx,Ly,field,per", STEP)
@pytest.mark.parametrize("dt", [0.1, -0.07])
def test_fp64_step(lm, sms, Lx, Ly, field, per, dt):
    lat, H = ham(lm, Lx, Ly, field, per)
    rng = np.random.default_rng(lat.N)
    X = rng.standard_normal((lat.N, sms)) + 1j * rng.standard_normal((lat.N, sms))
    ctx = lm.default_context()
    out, launches = [], []
    try:
        for on in (True, False):
            ctx.set_fused(on)
            st = lm.KetBlock(lat, X, precision="c64")
            s = lm.ChebyshevGPU()
            s.update_solver(H, dt)
            h = s._prepare(st)
            ctx.check(ctx.lib.lm_solver_step(h, st.handle))
            n = ctx.timing()[2]
            ctx.check(ctx.lib.lm_solver_step(h, st.handle))
            launches.append(ctx.timing()[2] - n)
            out.append(st.to_numpy())
    finally:
        ctx.set_fused(True)
    assert launches[0] == 1 and launches[1] > 2
    assert np.linalg.norm(out[0] - out[1]) <= 1e-14 * np.linalg.norm(out[1])


# columns per thread and kets per CTA: 1 x 1, 1 x 2, 2 x 2, 3 x 1, 4 x 2, 6 x 2, 8 x 1, 10 x 1, 12 x 1
SERIES = [(20, 18, "flux", None, 40), (20, 18, "flux", None, 310), (16, 40, "landau", {"axis1": True}, 309), (18, 64, "sum", None, 33),
          (48, 31, "sum", None, 311), (30, 70, "flux", None, 304), (40, 70, "landau", {"axis1": True, "axis2": True}, 17),
          (60, 64, "flux", None, 200), (34, 110, "flux", None, 152)]


@pytest.mark.parametrize("Lx,Ly,field,per,M", SERIES)
def test_doublefloat_series(lm, Lx, Ly, field, per, M):
    lat, H = ham(lm, Lx, Ly, field, per, 1.0)
    ctx = lm.default_context()
    lo, hi = H.bounds(ctx)
    coef = np.cos(np.arange(23.0)) / (1 + np.arange(23.0))
    rng = np.random.default_rng(lat.N)
    src = lm.DeviceState(lat, rng.standard_normal((lat.N, M)) + 1j * rng.standard_normal((lat.N, M)), 0, "c64")
    dh = H.device(ctx)
    out, launches = [], []
    try:
        for on in (True, False):
            ctx.set_kpm_doublefloat(on)
            st = lm.DeviceState(lat, None, 0, "c64", shape=(lat.N, M))
            n = ctx.timing()[2]
            ctx.check(ctx.lib.lm_cheb_apply(dh.handle, lo, hi, coef.ctypes.data_as(C.POINTER(C.c_double)), len(coef),
                                            src.handle, st.handle))
            launches.append(ctx.timing()[2] - n)
            out.append(st.to_numpy())
    finally:
        ctx.set_kpm_doublefloat(True)
    assert launches[0] == 2 and launches[1] > 20  # the tables and the series; a launch per term
    assert np.linalg.norm(out[0] - out[1]) <= 1e-12 * np.linalg.norm(out[1])


@pytest.mark.parametrize("Lx,Ly,per,field", [(13, 11, None, "flux"), (17, 5, None, "landau"), (64, 63, None, "flux"),
                                             (97, 75, None, "flux"), (95, 89, None, "landau"), (66, 32, {"axis1": True}, "flux"),
                                             (15, 28, {"axis1": True, "axis2": True}, "flux"), (3, 301, None, "flux")])
@pytest.mark.parametrize("dt", [0.02, 0.05, 0.1])
def test_resident_step(lm, Lx, Ly, per, field, dt):
    lat, H = ham(lm, Lx, Ly, field, per)
    X = o.random_kets(lat.N, 701, 3).astype(np.complex64)
    ctx = lm.default_context()
    out, ran = [], []
    try:
        ctx.set_stream_form(False)
        for on in (True, False):
            ctx.set_resident_form(on)
            st = lm.KetBlock(lat, X, precision="c32")
            s = lm.ChebyshevGPU()
            n = ctx.resident_launches()
            s.update_solver(H, dt)
            s.step(st)
            s.step(st)
            ran.append(ctx.resident_launches() - n)
            out.append(st.to_numpy())
    finally:
        ctx.set_stream_form(True)
        ctx.set_resident_form(True)
    assert ran == [2, 0]
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("Lx,Ly,M,dt", [(12, 10, 37, 0.05), (64, 64, 150, 0.05), (75, 71, 9, 0.05), (97, 75, 20, 0.05),
                                        (9, 7, 200, 0.2), (16, 16, 256, 0.02)])
def test_resident_adjoint(lm, Lx, Ly, M, dt):
    lat = lm.SquareLattice(Lx, Ly)
    rng = np.random.default_rng(8)
    psi = o.random_kets(lat.N, M, 3)
    V, B, target = rng.uniform(-0.1, 0.1, lat.N), np.array([0.1, 0.13, 0.08]), rng.uniform(0.2, 0.8, lat.N)
    ctx = lm.default_context()
    out, ran = [], []
    try:
        for on in (True, False):
            ctx.set_resident_form(on)
            n = ctx.resident_launches()
            p = lm.DensityLossAdjoint(lat, psi, target, dt, 9, 3, (Lx // 2 + 0.5, Ly // 2 + 0.5), checkpoint_every=4)
            out.append(p.loss_and_grad(V, B))
            ran.append(ctx.resident_launches() - n)
    finally:
        ctx.set_resident_form(True)
    assert ran[0] >= 2 * 9 and ran[1] == 0  # two recurrences per step
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
