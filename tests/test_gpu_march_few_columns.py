"""The double-float passes on blocks so small that a thread takes one to three columns of its row: the series
against the FP64 recurrence (1e-12) and the moments (1e-13 mu_0), the bars of the other shapes, on lattices that the
on-chip form does not take (periodic x with complex hops, or too large), for one to five kets."""
import ctypes as C

import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,per", [(2, 3, {"axis1": True}), (3, 40, {"axis1": True}), (17, 9, {"axis1": True, "axis2": True}),
                                       (64, 64, None), (64, 64, {"axis1": True}), (301, 33, None), (150, 140, {"axis2": True})])
@pytest.mark.parametrize("M", [1, 2, 5])
def test_few_columns(Lx, Ly, per, M):
    import lmgpu as lm
    ctx = lm.default_context()
    lat = lm.SquareLattice(Lx, Ly, boundaries=per)
    f = lm.PointFlux(0.2, (Lx // 2 + 0.5, Ly // 2 + 0.5), "singular" if per else "axial")
    H = lm.tightbinding_hamiltonian(lat, o.anderson_disorder(lat.N, 1.0, 4), field=f)
    lo, hi = H.bounds(ctx)
    coef = np.cos(np.arange(23.0)) / (1 + np.arange(23.0))
    rng = np.random.default_rng(lat.N)
    src = lm.DeviceState(lat, rng.standard_normal((lat.N, M)) + 1j * rng.standard_normal((lat.N, M)), 0, "c64")
    out = []
    try:
        for on in (True, False):
            ctx.set_kpm_doublefloat(on)
            st = lm.DeviceState(lat, None, 0, "c64", shape=(lat.N, M))
            ctx.check(ctx.lib.lm_cheb_apply(H.device(ctx).handle, lo, hi, coef.ctypes.data_as(C.POINTER(C.c_double)), len(coef),
                                            src.handle, st.handle))
            out.append((st.to_numpy(), lm.kpm.moments(H, 41, src, per_site=True, bounds=(lo, hi))[0]))
    finally:
        ctx.set_kpm_doublefloat(True)
    assert np.linalg.norm(out[0][0] - out[1][0]) <= 1e-12 * np.linalg.norm(out[1][0])
    assert np.abs(out[0][1] - out[1][1]).max() <= 1e-13 * np.abs(out[1][1][:, 0]).max()
