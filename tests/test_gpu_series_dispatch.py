"""The rule between the on-chip ComplexF64 step and a launch per order, on both sides of its line: the number
of launches of a step tells the form.  The expected sides are the faster ones as measured on 152 SMs (the rule
counts SMs, so they hold for that device)."""
import ctypes as C

import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu

CASES = [  # lattice, field, kets (None: dense), on chip
    (10, 10, "flux", None, True), (24, 24, "flux", None, True), (40, 33, "flux", None, False),
    (32, 27, "flux", 304, True), (32, 27, "flux", 330, False), (32, 27, "flux", 700, False), (32, 27, "landau", 456, False),
    (24, 24, "flux", 330, False), (24, 24, "flux", 912, True), (24, 24, "landau", 152, True), (31, 47, "flux", 700, False),
    (31, 47, "flux", 1216, True), (40, 33, "flux", 456, False), (6, 6, "flux", 1, True), (32, 27, "landau", 8, False)]


@pytest.mark.parametrize("Lx,Ly,field,M,on_chip", CASES)
def test_form(Lx, Ly, field, M, on_chip):
    import lmgpu as lm
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("sides measured on 152 SMs")
    ctx = lm.default_context()
    lat = lm.SquareLattice(Lx, Ly)
    f = lm.LandauGauge(0.02) if field == "landau" else lm.PointFlux(0.3, (Lx // 2 + 0.5, Ly // 2 + 0.5))
    H = lm.tightbinding_hamiltonian(lat, np.linspace(-0.3, 0.3, lat.N), field=f)
    X = o.random_kets(lat.N, M or lat.N, 3)
    st = lm.KetBlock(lat, X, precision="c64") if M else lm.DensityMatrix(lat, X)
    s = lm.ChebyshevGPU()
    s.update_solver(H, 0.1)
    h = s._prepare(st)
    K = C.c_int()
    ctx.check(ctx.lib.lm_solver_order(h, C.byref(K), None, None))
    n = []
    for _ in range(2):
        before = ctx.timing()[2]
        ctx.check(ctx.lib.lm_solver_step(h, st.handle))
        n.append(ctx.timing()[2] - before)
    passes = 1 if M else 2
    assert n[1] == (passes if on_chip else passes * K.value)
