"""The on-chip Chebyshev series (whole kets in shared memory) at the edges of its forms: one to
twelve columns per thread, one and two kets per CTA, rows that leave lanes idle, open, periodic and
twisted y axes, gauge-transformed and naturally real x-hops.

* the ComplexF64 step against the per-order kernels (1e-14: the same series, rounded differently,
  10 orders of an operator of norm 1) and, for a non-Hermitian operator, U A U^dagger;
* lm_cheb_apply in double-float against the FP64 recurrence (1e-12, as for the KPM moments) and the
  KPM recurrence with its dots (1e-13 mu_0)."""
import ctypes as C

import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lm():
    import lmgpu
    return lmgpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


FIELDS = {
    "none": lambda lm, Lx, Ly: None,
    "landau": lambda lm, Lx, Ly: lm.LandauGauge(0.03),
    "flux": lambda lm, Lx, Ly: lm.PointFlux(0.2, (Lx // 2 + 0.5, Ly // 2 + 0.5)),
    "sum": lambda lm, Lx, Ly: lm.SymmetricGauge(0.02) + lm.PointFlux(0.3, (1.5, Ly / 2)),
}
CASES = [(1, 1, "none", None), (2, 2, "flux", None), (1, 37, "none", None), (40, 1, "flux", None), (12, 10, "landau", None),
         (33, 16, "sum", None), (47, 31, "flux", None), (61, 7, "sum", {"axis2": True}), (13, 23, "landau", {"axis2": 0.7}),
         (30, 100, "flux", None), (64, 62, "sum", None), (5, 300, "flux", None)]


@pytest.mark.parametrize("Lx,Ly,field,per", CASES)
@pytest.mark.parametrize("kind", ["kets", "density"])
def test_fp64_step(lm, Lx, Ly, field, per, kind):
    N = Lx * Ly
    M = N if kind == "density" else 310
    if kind == "density" and N > 1500:
        pytest.skip("kets cover the larger lattices")
    rng = np.random.default_rng(N)
    X = rng.standard_normal((N, M)) + 1j * rng.standard_normal((N, M))
    lat = lm.SquareLattice(Lx, Ly, boundaries=per)
    H = lm.tightbinding_hamiltonian(lat, o.anderson_disorder(N, 1.0, 4), t1=-1.3, field=FIELDS[field](lm, Lx, Ly))
    ctx = lm.default_context()
    out = []
    try:
        for on in (True, False):
            ctx.set_fused(on)
            st = lm.DensityMatrix(lat, X) if kind == "density" else lm.KetBlock(lat, X, precision="c64")
            s = lm.ChebyshevGPU()
            for dt in (0.1, -0.07):
                s.update_solver(H, dt)
                s.step(st)
            out.append(st.to_numpy())
    finally:
        ctx.set_fused(True)
    assert rel(out[0], out[1]) <= 1e-14


@pytest.mark.parametrize("Lx,Ly,field,per,M", [
    (2, 2, "flux", None, None), (12, 10, "landau", {"axis1": True, "axis2": True}, None), (20, 18, "flux", None, None),
    (48, 31, "sum", None, 310), (48, 31, "sum", None, 17), (60, 64, "flux", None, 200), (96, 75, "flux", None, 33),
    (21, 300, "landau", {"axis1": True}, 7), (33, 9, "flux", {"axis1": True}, 5), (300, 1, "none", None, 3)])
@pytest.mark.parametrize("precision", ["c64", "c32"])
def test_real_series_doublefloat(lm, Lx, Ly, field, per, M, precision):
    N = Lx * Ly
    lat = lm.SquareLattice(Lx, Ly, boundaries=per)
    f = FIELDS[field](lm, Lx, Ly)
    if per and field == "flux":
        f = lm.PointFlux(0.2, (Lx // 2 + 0.5, Ly // 2 + 0.5), "singular")
    H = lm.tightbinding_hamiltonian(lat, o.anderson_disorder(N, 1.0, 4), field=f)
    ctx = lm.default_context()
    lo, hi = H.bounds(ctx)
    lo, hi = lo - 0.01, hi + 0.01
    coef = np.cos(np.arange(23.0)) / (1 + np.arange(23.0))
    src = None
    if M is not None:
        rng = np.random.default_rng(N)
        src = lm.DeviceState(lat, rng.standard_normal((N, M)) + 1j * rng.standard_normal((N, M)), 0, "c64")
    out = []
    try:
        for on in (True, False):
            ctx.set_kpm_doublefloat(on)
            st = lm.DeviceState(lat, None, 1 if M is None else 0, precision, shape=(N, M or N))
            dh = H.device(ctx)
            ctx.check(ctx.lib.lm_cheb_apply(dh.handle, lo, hi, coef.ctypes.data_as(C.POINTER(C.c_double)), len(coef),
                                            src.handle if src is not None else None, st.handle))
            out.append(st.to_numpy())
            mu, _ = lm.kpm.moments(H, 41, src, per_site=True, bounds=(lo, hi))
            out.append(mu)
    finally:
        ctx.set_kpm_doublefloat(True)
    assert rel(out[0], out[2]) <= (1e-12 if precision == "c64" else 1e-7)
    assert np.abs(out[1] - out[3]).max() <= 1e-13 * np.abs(out[3][:, 0]).max()


@pytest.mark.parametrize("Lx,Ly,per,M", [(24, 130, {"axis1": True, "axis2": True}, 200), (16, 300, {"axis2": True}, 200),
                                         (24, 300, None, 201), (5, 259, {"axis2": True}, 199)])
def test_doublefloat_chunks_of_rows(lm, Lx, Ly, per, M):
    """Blocks that hold a part of a column's rows (chunks of 44, 100, 50 and 87 here, the last ones shorter)."""
    test_real_series_doublefloat(lm, Lx, Ly, "landau", per, M, "c64")
