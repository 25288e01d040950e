"""A general Hamiltonian's step in one cooperative launch against one launch per order, bit for bit: rows
of 3 to 8 entries, odd and even numbers of orders, one ket and several, one site, grids that are full to
the last thread and one element beyond the form."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu


def ring_matrix(n, hops, seed):
    """Hermitian, n x n, with 2 * hops off-diagonal entries per row."""
    rng = np.random.default_rng(seed)
    H = sp.csc_matrix((n, n), dtype=np.complex128)
    for j in range(1, hops + 1):
        v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        U = sp.csc_matrix((v, (np.arange(n), (np.arange(n) + j) % n)), shape=(n, n))
        H = H + U + U.conj().T
    return (H + sp.diags(rng.standard_normal(n))).tocsc()


@pytest.mark.parametrize("n,hops,M", [(1, 0, 1), (9, 1, 1), (33, 2, 5), (1000, 3, 7), (4864, 4, 32), (155648, 1, 1),
                                      (155649, 1, 1), (31, 2, 700)])
@pytest.mark.parametrize("precision", ["c64", "c32"])
@pytest.mark.parametrize("dt", [0.02, 0.31])
def test_coop_bit_identical(n, hops, M, precision, dt):
    import lmgpu as lm
    ctx = lm.default_context()
    sites = lm.Sites(n)
    H = lm.SparseHamiltonian(sites, ring_matrix(n, hops, 3) if hops else sp.csc_matrix(np.array([[0.7 + 0j]])))
    X = o.random_kets(n, M, 1)
    out = []
    try:
        for on in (True, False):
            ctx.set_fused(on)
            st = lm.KetBlock(sites, X, precision=precision)
            s = lm.ChebyshevGPU()
            s.update_solver(H, dt)
            for _ in range(3):
                s.step(st)
            out.append(st.to_numpy())
    finally:
        ctx.set_fused(True)
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("make", ["HoneycombLattice", "KagomeLattice", "TriangularLattice"])
def test_coop_lattices(make):
    import lmgpu as lm
    ctx = lm.default_context()
    lat = getattr(lm, make)(23, 18)
    H = lm.tightbinding_hamiltonian(lat, np.linspace(-0.3, 0.3, lat.N), t1=-2.8, field=lm.SymmetricGauge(0.01))
    X = o.random_kets(lat.N, 2, 1)
    out = []
    try:
        for on in (True, False):
            ctx.set_fused(on)
            ev = lm.Evolution(lm.ChebyshevGPU(), H, lm.KetBlock(lat, X, precision="c64"))
            ts = lm.TimeSequence(lm.moment_density, ev([0.1 * k for k in range(1, 6)]))
            out.append(np.stack([v.values for v in ts.values]))
    finally:
        ctx.set_fused(True)
    assert np.array_equal(out[0], out[1])
