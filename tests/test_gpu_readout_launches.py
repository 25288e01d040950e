"""Readouts of few ComplexF32 kets are one launch: currents, and density and currents together, at one and
four sites per lane, odd and even x-hops' kinds, one ket to the last count below a second slice; values
against the FP64 sums (1e-13 of the scale)."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,per,field,M", [(5, 5, None, "landau", 1), (97, 75, None, "flux", 8), (25, 25, None, "flux", 255),
                                               (24, 24, None, "flux", 1), (24, 24, {"axis2": True}, "landau", 127),
                                               (2, 7, {"axis1": True}, "landau", 40), (1, 1, None, "landau", 2)])
def test_one_launch(Lx, Ly, per, field, M):
    import lmgpu as lm
    from lmgpu.timesequence import ReadoutRing
    ctx = lm.default_context()
    lat = lm.SquareLattice(Lx, Ly, boundaries=per)
    f = lm.LandauGauge(0.02) if field == "landau" else lm.PointFlux(0.3, (Lx // 2 + 0.5, Ly // 2 + 0.5))
    H = lm.tightbinding_hamiltonian(lat, field=f)
    X = o.random_kets(lat.N, M, 5).astype(np.complex64)
    st = lm.KetBlock(lat, X, precision="c32")
    H.device(ctx)
    rho, cur = ReadoutRing(lat.N, 2, ctx), ReadoutRing(max(lat.nbonds(), 1), 2, ctx)
    n0 = ctx.timing()[2]
    a, b = rho.push_both(cur, H, st, 0.0)
    n1 = ctx.timing()[2]
    c = cur.push_currents(H, st, 0.0)
    assert (n1 - n0, ctx.timing()[2] - n1) == (1, 1 if lat.nbonds() else 0)
    X = X.astype(np.complex128)
    ref = (np.abs(X) ** 2).sum(axis=1)
    assert np.abs(rho.wait(a)[1] - ref).max() <= 1e-13 * ref.max()
    if not lat.nbonds():
        return
    src, dst = (np.asarray(v) - 1 for v in lat.bonds())
    colptr, rowval, nz = H.csc()
    h = np.asarray(sp.csc_matrix((nz, rowval - 1, colptr - 1), shape=(lat.N, lat.N)).tocsr()[src, dst]).ravel()
    t = X[dst] * X[src].conj()
    J, scale = 2 * (h * t.sum(axis=1)).imag, 2 * (np.abs(h) * np.abs(t).sum(axis=1)).max()
    for q in (b, c):
        assert np.abs(cur.wait(q)[1] - J).max() <= 1e-13 * scale
