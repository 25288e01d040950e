"""Bond currents of weighted ComplexF32 kets over slices of the kets: against the sums in FP64 (1e-13 of the
products' scale, the bar of the other readouts), at ragged site and ket counts, real and complex x-hops, a
two-site periodic axis and a single row; small lattices with many kets take slices (two launches), few kets
or a lattice that fills the device one launch."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,per,field,M,launches", [
    (48, 48, None, "flux", 1024, 2), (48, 48, None, "landau", 1024, 2), (23, 25, None, "sym", 513, 2),
    (97, 75, None, "flux", 650, 2), (33, 20, {"axis2": True}, "landau", 517, 2), (1, 40, None, "none", 300, 2),
    (2, 2, {"axis1": True, "axis2": True}, "landau", 131, 2), (2, 5, {"axis1": 0.4}, "sym", 200, 2),
    (24, 24, None, "flux", 127, 1), (7, 9, None, "landau", 1, 1), (256, 320, None, "flux", 130, 1)])
def test_weighted_currents(Lx, Ly, per, field, M, launches):
    import lmgpu as lm
    ctx = lm.default_context()
    lat = lm.SquareLattice(Lx, Ly, boundaries=per)
    f = {"none": None, "landau": lm.LandauGauge(0.02), "sym": lm.SymmetricGauge(0.03),
         "flux": lm.PointFlux(0.3, (Lx // 2 + 0.5, Ly // 2 + 0.5))}[field]
    H = lm.tightbinding_hamiltonian(lat, o.anderson_disorder(lat.N, 1.0, 2), field=f)
    w = np.random.default_rng(1).uniform(-0.5, 1, M)
    X = o.random_kets(lat.N, M, 5).astype(np.complex64)
    st = lm.KetBlock(lat, X, weights=w, precision="c32")
    H.device(ctx)
    before = ctx.timing()[2]
    J = lm.DensityCurrents(H, st).bond_values()
    assert ctx.timing()[2] - before == launches
    src, dst = (np.asarray(v) - 1 for v in lat.bonds())
    X = X.astype(np.complex128)
    colptr, rowval, nz = H.csc()
    h = np.asarray(sp.csc_matrix((nz, rowval - 1, colptr - 1), shape=(lat.N, lat.N)).tocsr()[src, dst]).ravel()
    p, scale = np.empty(len(src), complex), np.empty(len(src))
    for b in range(0, len(src), 4096):
        q = slice(b, b + 4096)
        t = X[dst[q]] * X[src[q]].conj() * w
        p[q], scale[q] = t.sum(axis=1), np.abs(t).sum(axis=1)
    assert np.abs(J - 2 * (h * p).imag).max() <= 1e-13 * (2 * np.abs(h) * scale).max()
