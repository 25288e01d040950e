"""A solver steps with the Hamiltonian it was updated with, whatever its lm_ham holds by then
(update_solver! keeps the propagator, src/evolution.jl:80-94): the device Hamiltonian is assembled
anew between the update and the step, before the first step and between two steps, and a field
component of another kind is added to it.  Every form of the step gives what it gives without that, bit
for bit; the on-chip ComplexF64 form also agrees with the per-order kernels to 1e-13 (rounding)."""
import ctypes as C

import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu

FORMS = [(12, 10, "c64", "kets"), (12, 10, "c64", "density"), (23, 17, "c64", "kets"), (48, 64, "c64", "kets"),
         (13, 11, "c32", "kets"), (40, 32, "c32", "kets"), (97, 75, "c32", "kets")]
FIELDS = {
    "flux": lambda lm, a: lm.PointFlux(a, (5.5, 4.5)),
    "symmetric": lambda lm, a: lm.SymmetricGauge(a / 10),
    "landau": lambda lm, a: lm.LandauGauge(a / 10),
}


def _state(lm, lat, X, prec, kind):
    return lm.DensityMatrix(lat, X, precision=prec) if kind == "density" else lm.KetBlock(lat, X, precision=prec)


@pytest.mark.parametrize("Lx,Ly,prec,kind", FORMS)
@pytest.mark.parametrize("field", sorted(FIELDS))
@pytest.mark.parametrize("change", ["amplitude", "added field"])
def test_step_after_reassembly(Lx, Ly, prec, kind, field, change):
    import lmgpu as lm
    ctx = lm.default_context()
    lat = lm.SquareLattice(Lx, Ly)
    X = o.random_kets(lat.N, lat.N if kind == "density" else 152, 5)
    V = o.anderson_disorder(lat.N, 1.0, 4)

    def ham(a):
        return lm.tightbinding_hamiltonian(lat, V, t1=-1.3, field=FIELDS[field](lm, a))

    def other(dh, n):  # another H of the same structure in the same lm_ham, or one more component
        amps = [0.4 + 0.1 * n]
        if change == "added field":
            kind_id = lm._lib.LM_FIELD_SYMMETRIC
            ctx.check(ctx.lib.lm_ham_add_field(dh.handle, kind_id, 0.0, 0.0, 1, None))
            amps = [0.4] + [0.05] * (n + 1)
        ctx.check(ctx.lib.lm_ham_assemble(dh.handle, np.array(amps).ctypes.data_as(C.POINTER(C.c_double)), len(amps)))

    def run(disturb):
        dh = ham(0.2).device_private(ctx)
        h = C.c_void_p()
        ctx.check(ctx.lib.lm_solver_create(ctx.handle, 1e-12, C.byref(h)))
        try:
            ctx.check(ctx.lib.lm_solver_update(h, dh.handle, 0.1, 0))
            st = _state(lm, lat, X, prec, kind)
            for n in range(2):
                if disturb:
                    other(dh, n)
                ctx.check(ctx.lib.lm_solver_step(h, st.handle))
            return st.to_numpy()
        finally:
            ctx.lib.lm_solver_destroy(h)

    plain = run(False)
    assert np.array_equal(plain, run(True))
    if prec == "c64":
        try:
            ctx.set_fused(False)
            per_order = run(True)
        finally:
            ctx.set_fused(True)
        assert np.linalg.norm(plain - per_order) <= 1e-13 * np.linalg.norm(per_order)
