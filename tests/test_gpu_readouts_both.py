"""Density and currents in one pass (timesequences with one of each): against the sums of the same FP32
kets in FP64 (1e-13, the bar of the separate readouts), for one and four sites per lane, real and
complex x-hops, several ket slices, ragged site counts, a two-site periodic axis and single sites."""
import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu

CASES = [(12, 12, None, "landau", 6), (97, 75, None, "flux", 650), (16, 32, {"axis1": True, "axis2": True}, "landau", 70),
         (33, 20, {"axis2": True}, "sym", 517), (2, 2, {"axis1": True, "axis2": True}, "landau", 9), (1, 1, None, "none", 3),
         (1, 40, None, "none", 65), (5, 3, {"axis1": 0.4}, "landau", 12), (64, 66, None, "flux", 1)]


@pytest.mark.parametrize("Lx,Ly,per,field,M", CASES)
@pytest.mark.parametrize("precision,weighted", [("c32", False), ("c32", True), ("c64", False)])
def test_both_readouts(Lx, Ly, per, field, M, precision, weighted):
    import lmgpu as lm
    lat = lm.SquareLattice(Lx, Ly, boundaries=per)
    f = {"none": None, "landau": lm.LandauGauge(0.02), "sym": lm.SymmetricGauge(0.03),
         "flux": lm.PointFlux(0.3, (Lx // 2 + 0.5, Ly // 2 + 0.5))}[field]
    H = lm.tightbinding_hamiltonian(lat, o.anderson_disorder(lat.N, 1.0, 2), field=f)
    w = np.random.default_rng(1).uniform(0.1, 1, M) if weighted else None
    st = lm.KetBlock(lat, o.random_kets(lat.N, M, 5), weights=w, precision=precision)
    ev = lm.Evolution(lm.ChebyshevGPU(), H, st)
    rho, J = lm.timesequences([lm.moment_density, lm.moment_currents], ev([0.0, 0.05]), nslots=2)
    X = ev.current_states()[0].to_numpy().astype(np.complex128)
    ww = np.ones(M) if w is None else w
    P = (X * ww) @ X.conj().T if lat.N <= 1500 else None
    ref = (np.abs(X) ** 2 * ww).sum(axis=1)
    assert np.linalg.norm(rho.values[1].values - ref) <= 1e-13 * np.linalg.norm(ref)
    src, dst = lat.bonds()
    assert len(J.values[1]) == len(src)
    if len(src) == 0:
        return
    colptr, rowval, nz = H.csc()
    import scipy.sparse as sp
    Hm = sp.csc_matrix((nz, rowval - 1, colptr - 1), shape=(lat.N, lat.N)).tocsr()
    h = np.asarray(Hm[src - 1, dst - 1]).ravel()
    p = P[dst - 1, src - 1] if P is not None else (X[dst - 1] * X[src - 1].conj() * ww).sum(axis=1)
    Jref = 2 * (h * p).imag
    scale = np.linalg.norm(2 * np.abs(h) * np.sqrt(ref[dst - 1] * ref[src - 1]))
    assert np.linalg.norm(J.values[1] - Jref) <= 1e-13 * scale
    # the separate readouts of the same state
    assert np.linalg.norm(rho.values[1].values - lm.localdensity(ev.current_states()[0]).values) <= 1e-13 * np.linalg.norm(ref)
    assert np.linalg.norm(J.values[1] - lm.DensityCurrents(H, ev.current_states()[0]).bond_values()) <= 1e-13 * scale
