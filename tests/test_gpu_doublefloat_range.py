"""lm_cheb_apply in double-float on blocks of small values: the launch-per-term form (a periodic x axis with
complex hops) and the on-chip form keep FP32 subnormals, as a conversion to FP32 does.  The bar is FP32's
spacing there, 2^-149 per rounding: some 30 roundings for each of 23 terms of norm at most 1."""
import ctypes as C

import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,per", [(33, 9, {"axis1": True}), (12, 10, None)])
@pytest.mark.parametrize("scale", [2.0 ** -60, 2.0 ** -100, 2.0 ** -124, 2.0 ** -130])
def test_small_blocks(Lx, Ly, per, scale):
    import lmgpu as lm
    lat = lm.SquareLattice(Lx, Ly, boundaries=per)
    f = lm.PointFlux(0.2, (Lx // 2 + 0.5, Ly // 2 + 0.5), "singular" if per else "axial")
    H = lm.tightbinding_hamiltonian(lat, o.anderson_disorder(lat.N, 1.0, 4), field=f)
    ctx = lm.default_context()
    lo, hi = H.bounds(ctx)
    coef = np.cos(np.arange(23.0)) / (1 + np.arange(23.0))
    rng = np.random.default_rng(3)
    X = scale * (rng.uniform(-1, 1, (lat.N, 5)) + 1j * rng.uniform(-1, 1, (lat.N, 5)))
    src = lm.DeviceState(lat, X, 0, "c64")
    out = []
    try:
        for on in (True, False):
            ctx.set_kpm_doublefloat(on)
            st = lm.DeviceState(lat, None, 0, "c64", shape=(lat.N, 5))
            ctx.check(ctx.lib.lm_cheb_apply(H.device(ctx).handle, lo, hi, coef.ctypes.data_as(C.POINTER(C.c_double)),
                                            len(coef), src.handle, st.handle))
            out.append(st.to_numpy())
    finally:
        ctx.set_kpm_doublefloat(True)
    bound = 1e-12 * scale + 23 * 30 * 2.0 ** -149
    assert np.abs(out[0] - out[1]).max() <= bound
    assert np.abs(out[1]).max() > 100 * bound
