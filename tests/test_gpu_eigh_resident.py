"""The on-chip eigensystem stages at the edges of their ranges: one column per CTA to eight, the
first size beyond the shared-memory form, and cluster and block counts of the solves.  Bars as in
the general eigensystem tests (1e-13 |H| for values, 1e-12 for residuals and orthonormality)."""
import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu

SIZES = [(1, 2), (3, 1), (5, 7), (17, 9), (19, 16), (5, 61), (32, 27), (32, 38), (29, 42)]


@pytest.mark.parametrize("Lx,Ly", SIZES)
@pytest.mark.parametrize("clean", [False, True])
def test_eigensystem_edges(Lx, Ly, clean):
    import lmgpu
    if clean and Lx * Ly > 400:
        pytest.skip("degenerate levels are covered by the smaller sizes")
    ol, ll = o.SquareLattice(Lx, Ly), lmgpu.SquareLattice(Lx, Ly)
    V = None if clean else o.anderson_disorder(ol.N, 2.0, 7)
    pt = ((Lx + 1) / 2.0, (Ly + 1) / 2.0)
    of, lf = (None, None) if clean else (o.PointFlux(0.2, pt), lmgpu.PointFlux(0.2, pt))
    Hd = o.tightbinding_hamiltonian(ol, field=of, onsite=V).toarray()
    eig = lmgpu.diagonalize(lmgpu.tightbinding_hamiltonian(ll, *([] if clean else [V]), field=lf))
    w = np.linalg.eigvalsh(Hd)
    hn = max(1.0, np.abs(w).max())
    assert np.abs(eig.values - w).max() <= 1e-13 * hn
    X = eig.vectors().to_numpy()
    n = ol.N
    assert np.linalg.norm(Hd @ X - X * eig.values) <= 1e-12 * hn * np.sqrt(n)
    assert np.abs(X.conj().T @ X - np.eye(n)).max() <= 1e-12
    wt = np.random.default_rng(5).uniform(0, 1, n)
    P = eig.projector(wt).to_numpy()
    Pr = (X * wt) @ X.conj().T
    assert np.linalg.norm(P - Pr) <= 1e-12 * np.linalg.norm(Pr)


@pytest.mark.parametrize("ex", [-470, -300, 300, 470])
def test_eigenvalues_scaled(ex):
    """Scaling H by a power of two scales the eigenvalues: the reflectors' roots and reciprocals inside
    and beyond the range of their scaled iteration."""
    import lmgpu
    ol, ll = o.SquareLattice(11, 13), lmgpu.SquareLattice(11, 13)
    V, sc = o.anderson_disorder(ol.N, 2.0, 7), 2.0 ** ex
    pt = (6.0, 7.0)
    w = np.linalg.eigvalsh(o.tightbinding_hamiltonian(ol, field=o.PointFlux(0.2, pt), onsite=V).toarray())
    eig = lmgpu.diagonalize(lmgpu.tightbinding_hamiltonian(ll, V * sc, t1=sc, field=lmgpu.PointFlux(0.2, pt)))
    assert np.abs(eig.values / sc - w).max() <= 1e-13 * np.abs(w).max()
