"""The lattice-resident kernels on a single lattice: the step of a ket block (one CTA, several kets per
CTA, a cluster of two, odd sides, a last item that is not full) bit for bit against the region form,
lm_solver_step_to against copy and step, and the adjoint's recurrences and sums bit for bit against the
per-order kernels."""
import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lm():
    import lmgpu
    return lmgpu


def problem(lm, Lx, Ly, per, landau):
    lat = lm.SquareLattice(Lx, Ly, boundaries=per)
    f = lm.LandauGauge(0.02) if landau else lm.PointFlux(0.3, (Lx // 2 + 0.5, Ly // 2 + 0.5),
                                                         "singular" if per else "axial")
    return lat, lambda: lm.tightbinding_hamiltonian(lat, o.anderson_disorder(lat.N, 1.0, 6), field=f)


@pytest.mark.parametrize("Lx,Ly,per,landau", [(13, 11, None, False), (17, 5, None, True), (64, 63, None, False),
                                              (97, 75, None, False), (95, 97, None, True), (66, 32, {"axis1": True}, False),
                                              (15, 28, {"axis1": True, "axis2": True}, False), (3, 301, None, False)])
@pytest.mark.parametrize("dt", [0.02, 0.05, 0.1])
def test_step_bit_identical_to_region_form(lm, Lx, Ly, per, landau, dt):
    lat, ham = problem(lm, Lx, Ly, per, landau)
    X = o.random_kets(lat.N, 701, 3).astype(np.complex64)
    ctx = lm.default_context()
    out = []
    try:
        ctx.set_stream_form(False)
        for on in (True, False):
            ctx.set_resident_form(on)
            st = lm.KetBlock(lat, X, precision="c32")
            s = lm.ChebyshevGPU()
            s.update_solver(ham(), dt)
            s.step(st)
            s.step(st)
            out.append(st.to_numpy())
    finally:
        ctx.set_stream_form(True)
        ctx.set_resident_form(True)
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("Lx,Ly,prec,dt", [(13, 11, "c32", 0.05), (97, 75, "c32", 0.1), (30, 64, "c32", 0.03),
                                           (13, 11, "c64", 0.1), (20, 20, "c32", 0.5)])
def test_step_to(lm, Lx, Ly, prec, dt):
    lat, ham = problem(lm, Lx, Ly, None, False)
    X = o.random_kets(lat.N, 40, 3)
    ctx = lm.default_context()
    a, b, c = (lm.KetBlock(lat, X, precision=prec) for _ in range(3))
    s = lm.ChebyshevGPU()
    s.update_solver(ham(), dt)
    s.step(a)
    h = s._prepare(b)
    ctx.check(ctx.lib.lm_solver_step_to(h, b.handle, c.handle))
    assert np.array_equal(a.to_numpy(), c.to_numpy())
    assert np.array_equal(b.to_numpy(), X.astype(b.dtype))
    assert ctx.lib.lm_solver_step_to(h, b.handle, b.handle) != 0


@pytest.mark.parametrize("Lx,Ly,M,dt", [(12, 10, 37, 0.05), (64, 64, 150, 0.05), (75, 71, 9, 0.05), (9, 7, 200, 0.2),
                                        (16, 16, 256, 0.02)])
def test_adjoint_forms_agree(lm, Lx, Ly, M, dt):
    lat = lm.SquareLattice(Lx, Ly)
    rng = np.random.default_rng(8)
    psi = o.random_kets(lat.N, M, 3)
    V, B, target = rng.uniform(-0.1, 0.1, lat.N), np.array([0.1, 0.13, 0.08]), rng.uniform(0.2, 0.8, lat.N)
    ctx = lm.default_context()
    out = []
    try:
        for on in (True, False):
            ctx.set_resident_form(on)
            p = lm.DensityLossAdjoint(lat, psi, target, dt, 9, 3, (Lx // 2 + 0.5, Ly // 2 + 0.5), checkpoint_every=4)
            out.append(p.loss_and_grad(V, B))
    finally:
        ctx.set_resident_form(True)
    (l0, v0, b0), (l1, v1, b1) = out
    assert l0 == l1
    assert np.array_equal(v0, v1) and np.array_equal(b0, b1)
