"""Measured workloads: what a program that uses this framework has it do.

Each case is one of the eight kinds of calls below, through the public ``lmgpu`` entry points,
at sizes of the repository's own configurations, tests and benchmark or of the same order:

  ramp       Evolution(t -> h(t), P_0) of a dense ComplexF64 density matrix on an open square
             lattice under a PointFlux ramp, localdensity and DensityCurrents at every moment
  kets       a block of kets on a square lattice (Landau field on a torus, or a point flux on an
             open lattice), H(t) changing every step, both readouts at every moment
  graphene   kets of a honeycomb patch under a constant H, localdensity at every moment
  batch      one step of many uneven lattices, each with its own dense P
  adjoint    loss and gradients of a density loss through a whole evolution
  kpm        Chebyshev moments of a block of random-phase vectors
  fermi      densitymatrix(H; mu, T) at T > 0
  eigen      densitymatrix(H; mu) at T = 0
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "latticemodels.jl_gb300"))
import lmgpu  # noqa: E402

DEV = "cuda"


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def listed():
    return [
        # the first program of the README: a 10 x 10 lattice, the ramp read out every step; small
        # launches and host calls only
        {"name": "ramp_10x10", "kind": "ramp", "Lx": 10, "Ly": 10, "steps": 20},
        # the same program on a lattice of a thousand sites, odd and not square
        {"name": "ramp_47x31", "kind": "ramp", "Lx": 47, "Ly": 31, "steps": 4},
        # the benchmark workload: 2048 compensated FP32 kets on a 256 x 256 torus with disorder
        {"name": "kets_256_comp", "kind": "kets", "Lx": 256, "Ly": 256, "M": 2048, "torus": True, "form": "comp",
         "steps": 4},
        # the same torus in the plain FP64 form, with the kets that one run usually has
        {"name": "kets_256_c64", "kind": "kets", "Lx": 256, "Ly": 256, "M": 384, "torus": True, "form": "c64",
         "steps": 2},
        # an open lattice of odd sides around a point flux (complex hops on both axes), FP32
        {"name": "kets_97x75_c32", "kind": "kets", "Lx": 97, "Ly": 75, "M": 650, "torus": False, "form": "c32",
         "steps": 4},
        # the evolution benchmark of the framework's reference: one FP64 ket on 1e5 graphene sites
        {"name": "graphene_224_ket", "kind": "graphene", "a": 224, "b": 224, "M": 1, "steps": 40},
        # a block of FP32 kets on graphene
        {"name": "graphene_180_c32", "kind": "graphene", "a": 180, "b": 180, "M": 512, "steps": 4},
        # uneven lattices of 16..96 sites a side with dense P, stepped together
        {"name": "batch_24", "kind": "batch", "lattices": 24, "Lmin": 16, "Lmax": 96, "sizes": 3},
        # control of a density: gradients through 120 steps with 1024 occupied kets
        {"name": "adjoint_64", "kind": "adjoint", "L": 64, "M": 1024, "steps": 120},
        # density of states of the benchmark's torus from 256 random-phase vectors
        {"name": "kpm_256", "kind": "kpm", "L": 256, "R": 256, "nmom": 384},
        # a thermal state: the start of every run at finite temperature
        {"name": "fermi_48", "kind": "fermi", "Lx": 48, "Ly": 48, "T": 0.1},
        # a ground state: the start of every run at zero temperature
        {"name": "eigen_32x27", "kind": "eigen", "Lx": 32, "Ly": 27},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ramp", "kets", "kets", "graphene", "batch", "adjoint", "kpm", "fermi", "eigen"])
    if kind == "ramp":
        Lx, Ly = _log(rng, 6, 48), _log(rng, 6, 48)
        return {"kind": kind, "Lx": Lx, "Ly": Ly, "steps": rng.randint(2, 20 if Lx * Ly < 400 else 5)}
    if kind == "kets":
        torus = rng.random() < 0.5
        form = rng.choice(["c32", "c64", "comp"] if torus else ["c32", "c64"])
        Lx, Ly = _log(rng, 24, 320), _log(rng, 24, 320)
        if form == "comp":  # the compensated state takes lattices with an even Ly
            Ly += Ly % 2
        cap = (1 << 25 if form == "c64" else 1 << 27) // (Lx * Ly)
        return {"kind": kind, "Lx": Lx, "Ly": Ly, "M": min(cap, _log(rng, 16, 2048)), "torus": torus, "form": form,
                "steps": rng.randint(1, 4)}
    if kind == "graphene":
        a, b = _log(rng, 20, 224), _log(rng, 20, 224)
        M = 1 if rng.random() < 0.5 else _log(rng, 8, 512)
        return {"kind": kind, "a": a, "b": b, "M": M, "steps": rng.randint(5, 40) if M == 1 else rng.randint(1, 4)}
    if kind == "batch":
        lo = _log(rng, 12, 40)
        return {"kind": kind, "lattices": rng.randint(3, 24), "Lmin": lo, "Lmax": min(96, lo + _log(rng, 4, 60)),
                "sizes": rng.randint(1, 1 << 20)}
    if kind == "adjoint":
        L = _log(rng, 16, 64)
        return {"kind": kind, "L": L, "M": min(L * L, _log(rng, 32, 1024)), "steps": rng.randint(20, 120)}
    if kind == "kpm":
        return {"kind": kind, "L": _log(rng, 32, 256), "R": _log(rng, 16, 256), "nmom": _log(rng, 64, 384)}
    if kind == "fermi":
        return {"kind": kind, "Lx": _log(rng, 10, 48), "Ly": _log(rng, 10, 48), "T": round(rng.uniform(0.08, 0.4), 3)}
    return {"kind": kind, "Lx": _log(rng, 6, 32), "Ly": _log(rng, 6, 32)}


def _sides(case):
    """The sides of a batch's lattices."""
    r = np.random.default_rng(case["sizes"])
    return [int(v) for v in r.integers(case["Lmin"], case["Lmax"] + 1, case["lattices"])]


# ------------------------------------------------------------------------------------------
# inputs from a seed, shared by prepare() and exact()
# ------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _disorder(seed, N, W):
    return np.random.default_rng([int(seed), 1]).uniform(-W / 2, W / 2, N)


def _kets(seed, N, M, dtype):
    """M normalised complex Gaussian kets, ket by ket (M x N)."""
    g = _gen(seed)
    X = torch.empty(M, N, dtype=dtype, device=DEV)
    for k in range(0, M, 256):
        x = torch.randn(min(256, M - k), N, dtype=dtype, device=DEV, generator=g)
        X[k:k + 256] = x / torch.linalg.vector_norm(x, dim=1, keepdim=True)
    return X


def _phase_vectors(seed, N, R):
    th = torch.rand(R, N, dtype=torch.float64, device=DEV, generator=_gen(seed)) * (2 * math.pi)
    return torch.polar(torch.ones_like(th), th)


def _hermitian(seed, N):
    """A Hermitian N x N block with density-like entries (half on the diagonal, small elsewhere)."""
    A = torch.randn(N, N, dtype=torch.complex64, device=DEV, generator=_gen(seed))
    A = (A + A.conj().T) * (0.25 / math.sqrt(N))
    A.diagonal().add_(0.5)
    return A


def _projector(seed, Lx, Ly):
    """The zero-temperature density matrix at mu = 0 of the field-free lattice with disorder."""
    hx, hy, V = _hops(Lx, Ly, False, ("none",), _disorder(seed, Lx * Ly, 1.0))
    w, v = torch.linalg.eigh(_dense(hx, hy, V).real)
    v = v[:, w <= 0]
    return (v @ v.T).to(torch.complex128)


def _standing_waves(L, M):
    """The M lowest eigenstates of the clean open L x L lattice (M x N), FP32."""
    q = np.pi * np.arange(1, L + 1) / (L + 1)
    s = np.sqrt(2 / (L + 1)) * np.sin(np.outer(q, np.arange(1, L + 1)))
    E = 2 * np.cos(q)[:, None] + 2 * np.cos(q)[None, :]
    k = np.argsort(E.ravel(), kind="stable")[:M]
    return np.einsum("kx,ky->kxy", s[k // L], s[k % L]).reshape(len(k), L * L).astype(np.complex64)


def _control(case, seed):
    """On-site potentials, flux amplitudes and the target density of an adjoint case."""
    L, spi = case["L"], 8
    r = np.random.default_rng([int(seed), 2])
    V = r.uniform(-0.1, 0.1, L * L)
    B = 0.1 + r.uniform(-0.02, 0.02, (case["steps"] + spi - 1) // spi)
    c = r.uniform(0.3 * L, 0.7 * L, 2)
    x = np.stack(np.meshgrid(np.arange(1, L + 1), np.arange(1, L + 1), indexing="ij"), -1).reshape(-1, 2)
    target = 0.5 + 0.2 * np.exp(-((x - c) ** 2).sum(1) / (2 * 6.0 ** 2))
    return V, B, target, (L // 2 + 0.5, L // 2 + 0.5), spi


def _kets_field(case, t):
    """The field of a kets case at time t: a modulated Landau field, or a ramped point flux."""
    if case["torus"]:
        return ("landau", 0.01 * (1 + 0.1 * math.sin(t + 0.5)))
    return ("flux", 0.2 * min(t + 0.5, 10.0) / 10, case["Lx"] // 2 + 0.5, case["Ly"] // 2 + 0.5)


def _ramp_field(case, t):
    return ("flux", 0.2 * min(t, 10.0) / 10, case["Lx"] // 2 + 0.5, case["Ly"] // 2 + 0.5)


def _graphene(case):
    """t1, the symmetric-gauge field and dt: the FP64 benchmark model, or a Landau-scale block."""
    return (-2.8, 3.0 * 1.519e-3, 0.1) if case["M"] == 1 else (1.0, 0.01, 0.05)


def _graphene_onsite(case, seed):
    a, b = case["a"], case["b"]
    j1, j2, s = np.meshgrid(np.arange(1, a + 1), np.arange(1, b + 1), np.arange(2), indexing="ij")
    x = j1 + 0.5 * j2 + 0.5 * s
    y = math.sqrt(3) / 2 * j2 + math.sqrt(3) / 6 * s
    r = math.sqrt(2 * a * b * math.sqrt(3) / 4 / math.pi)
    V = np.where((x - x.mean()) ** 2 + (y - y.mean()) ** 2 < (r / 2) ** 2, 0.2, 0.0).ravel()
    return V + _disorder(seed, V.size, 0.1)


# ------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------
class _Buffer:
    """A state's device buffer (one row per column of the state) for torch.as_tensor."""

    def __init__(self, st):
        ptr, ld = st.device_ptr()
        size = np.dtype(st.dtype).itemsize
        self.state = st
        self.__cuda_array_interface__ = {"shape": (st.m, st.n), "strides": (ld * size, size), "data": (ptr, False),
                                         "typestr": np.dtype(st.dtype).str, "version": 3}


def _tensor(st):
    return torch.as_tensor(_Buffer(st), device=DEV)


def _fill(st, rows):
    st.ctx.synchronize()
    _tensor(st).copy_(rows)
    torch.cuda.synchronize()
    return st


def _ket_block(lat, rows, precision):
    st = lmgpu.DeviceState(lat, None, lmgpu._lib.LM_KETS, precision, shape=(lat.N, rows.shape[0]))
    return _fill(st, rows)


def _field(f):
    if f[0] == "landau":
        return lmgpu.LandauGauge(f[1])
    return lmgpu.PointFlux(f[1], (f[2], f[3]))


@functools.lru_cache(maxsize=16)
def _honeycomb(a, b):
    return lmgpu.HoneycombLattice(a, b)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "steps": case.get("steps", 0)}
    if kind == "ramp":
        lat = lmgpu.SquareLattice(case["Lx"], case["Ly"])
        V = _disorder(seed, lat.N, 1.0)
        s["h"] = lambda t: lmgpu.tightbinding_hamiltonian(lat, V, field=_field(_ramp_field(case, t)))
        s["P0"] = _fill(lmgpu.DensityMatrix(lat, None), _projector(seed, case["Lx"], case["Ly"]).T)
        s["times"] = [0.1 * (k + 1) for k in range(case["steps"])]
    elif kind == "kets":
        axes = {"axis1": True, "axis2": True} if case["torus"] else None
        lat = lmgpu.SquareLattice(case["Lx"], case["Ly"], boundaries=axes)
        V = _disorder(seed, lat.N, 2.0)
        prec = "c64" if case["form"] == "c64" else "c32"
        st = _ket_block(lat, _kets(seed, lat.N, case["M"], torch.complex128 if prec == "c64" else torch.complex64), prec)
        if case["form"] == "comp":
            st.set_compensation(True)
        solver = lmgpu.ChebyshevGPU(renorm_every=0 if prec == "c64" else 20)
        s["ev"] = lmgpu.Evolution(
            solver, lambda t: lmgpu.tightbinding_hamiltonian(lat, V, field=_field(_kets_field(case, t))), st)
        s["dt"] = 0.05
    elif kind == "graphene":
        lat = _honeycomb(case["a"], case["b"])
        t1, B, dt = _graphene(case)
        prec = "c64" if case["M"] == 1 else "c32"
        s["H"] = lmgpu.tightbinding_hamiltonian(lat, _graphene_onsite(case, seed), t1=t1, field=lmgpu.SymmetricGauge(B))
        s["psi"] = _ket_block(lat, _kets(seed, lat.N, case["M"], torch.complex128 if prec == "c64" else torch.complex64),
                              prec)
        s["times"] = [dt * (k + 1) for k in range(case["steps"])]
    elif kind == "batch":
        batch, s["states"] = lmgpu.Batch("density", "c32"), []
        r = np.random.default_rng([int(seed), 3])
        for i, L in enumerate(_sides(case)):
            lat = lmgpu.SquareLattice(L, L)
            V, flux = _disorder(seed + 1000 * i, L * L, r.uniform(0, 3)), r.uniform(0, 0.3)
            P = _fill(lmgpu.DensityMatrix(lat, None, "c32"), _hermitian(seed + 1000 * i, L * L).T)
            batch.add(lmgpu.tightbinding_hamiltonian(lat, V, field=lmgpu.PointFlux(flux, (L // 2 + 0.5, L // 2 + 0.5))), P)
            s["states"].append(P)
        batch.update(0.1)
        s["batch"] = batch
    elif kind == "adjoint":
        s["V"], s["B"], target, point, spi = _control(case, seed)
        lat = lmgpu.SquareLattice(case["L"], case["L"])
        psi0 = _standing_waves(case["L"], case["M"]).T
        s["problem"] = lmgpu.DensityLossAdjoint(lat, psi0, target, 0.05, case["steps"], spi, point)
    elif kind == "kpm":
        lat = lmgpu.SquareLattice(case["L"], case["L"], boundaries={"axis1": True, "axis2": True})
        s["H"] = lmgpu.tightbinding_hamiltonian(lat, _disorder(seed, lat.N, 2.0), field=lmgpu.LandauGauge(0.01))
        s["vecs"] = _ket_block(lat, _phase_vectors(seed, lat.N, case["R"]), "c64")
        s["nmom"] = case["nmom"]
    else:  # fermi, eigen
        lat = lmgpu.SquareLattice(case["Lx"], case["Ly"])
        s["H"] = lmgpu.tightbinding_hamiltonian(
            lat, _disorder(seed, lat.N, 2.0), field=lmgpu.PointFlux(0.2, (case["Lx"] // 2 + 0.5, case["Ly"] // 2 + 0.5)))
        s["T"] = case.get("T", 0.0)
    return s


def run(s):
    kind = s["kind"]
    if kind == "ramp":  # the whole program, from P_0 at t = 0
        ev = lmgpu.Evolution(s["h"], s["P0"])
        rho, J = lmgpu.timesequences([lmgpu.moment_density, lmgpu.moment_currents], ev(s["times"]))
        return {"density": np.stack([v.values for v in rho.values]), "currents": np.stack(J.values),
                "P": _tensor(ev.current_states()[0])}
    if kind == "kets":  # the next steps of a long run
        ev = s["ev"]
        t = ev.time
        rho, J = lmgpu.timesequences([lmgpu.moment_density, lmgpu.moment_currents],
                                     ev([t + s["dt"] * (k + 1) for k in range(s["steps"])]))
        return {"density": np.stack([v.values for v in rho.values]), "currents": np.stack(J.values),
                "kets": _tensor(ev.current_states()[0])}
    if kind == "graphene":
        ev = lmgpu.Evolution(s["H"], s["psi"])
        rho = lmgpu.TimeSequence(lmgpu.moment_density, ev(s["times"]))
        return {"density": np.stack([v.values for v in rho.values]), "kets": _tensor(ev.current_states()[0])}
    if kind == "batch":
        s["batch"].step()
        return [_tensor(P) for P in s["states"]]
    if kind == "adjoint":
        loss, gV, gB = s["problem"].loss_and_grad(s["V"], s["B"])
        return {"loss": loss, "gV": gV, "gB": gB}
    if kind == "kpm":
        mu, bounds = lmgpu.kpm.moments(s["H"], s["nmom"], s["vecs"])
        return {"mu": mu, "bounds": np.array(bounds)}
    return _tensor(lmgpu.densitymatrix(s["H"], mu=0.0, T=s["T"]))


# ------------------------------------------------------------------------------------------
# the work that a pass cannot do without: each input read once, each output written once, and
# the arithmetic of the shortest Chebyshev series to the form's tolerance (16 fused
# multiply-adds per site and order where the x-hops are real, 20 where all hops are complex, 16
# on the honeycomb)
# ------------------------------------------------------------------------------------------
def _order(x, tol):
    """Chebyshev order K >= 2 of exp(-i x cos) to ``tol`` (Bessel tail by backward recurrence)."""
    n = int(x) + 40
    J = np.zeros(n + 2)
    J[n] = 1e-300
    for k in range(n, 0, -1):
        J[k - 1] = 2 * k / x * J[k] - J[k + 1]
    J = np.abs(J / (J[0] + 2 * J[2::2].sum()))
    K = 2
    while 2 * J[K + 1:].sum() > tol:
        K += 1
    return K


def work(case):
    kind = case["kind"]
    n = case.get("steps", 0)
    if kind == "ramp":
        N = case["Lx"] * case["Ly"]
        return {"bytes": n * (2 * 16.0 * N * N + 8 * 3 * N), "flops": n * 2 * 40.0 * _order(0.45, 1e-12) * N * N}
    if kind == "kets":
        N, M = case["Lx"] * case["Ly"], case["M"]
        per = {"c32": 16.0, "comp": 24.0, "c64": 32.0}[case["form"]]
        K = _order(0.25, 1e-12 if case["form"] == "c64" else 1e-9)
        return {"bytes": n * (per * N * M + 8 * 3 * N), "flops": n * (32.0 if case["torus"] else 40.0) * K * N * M}
    if kind == "graphene":
        N, M = 2 * case["a"] * case["b"], case["M"]
        t1, _, dt = _graphene(case)
        K = _order((3 * abs(t1) + 0.15) * dt, 1e-12 if M == 1 else 1e-9)
        return {"bytes": n * ((32.0 if M == 1 else 16.0) * N * M + 8 * N), "flops": n * 32.0 * K * N * M}
    if kind == "batch":
        S = sum(float(L) ** 4 for L in _sides(case))
        return {"bytes": 2 * 8 * S, "flops": 2 * 40.0 * _order(0.5, 1e-9) * S}
    if kind == "adjoint":  # forward, co-state and the gradient recurrences of every step
        N, M, K = case["L"] ** 2, case["M"], _order(0.22, 1e-9)
        return {"bytes": 8.0 * N * M + 8 * 2 * N, "flops": n * 4 * 40.0 * K * N * M}
    if kind == "kpm":  # two new Chebyshev vectors' worth of moments per pass over the block
        N, R = case["L"] ** 2, case["R"]
        return {"bytes": 16.0 * N * R, "flops": case["nmom"] / 2 * 44.0 * N * R}
    N = case["Lx"] * case["Ly"]
    if kind == "fermi":
        return {"bytes": 16.0 * N * N, "flops": 5.1 / case["T"] * 9.7 * 44.0 * N * N}
    return {"bytes": 16.0 * N * N, "flops": (16 / 3 + 8 / 2 + 4 / 2) * float(N) ** 3}


# ------------------------------------------------------------------------------------------
# the same in 64 bits with plain torch
# ------------------------------------------------------------------------------------------
def _line(f, x1, y1, x2, y2):
    """The field's line integral from (x1, y1) to (x2, y2), in flux quanta."""
    if f[0] == "landau":
        return (x1 + x2) * (y2 - y1) * f[1] / 2
    if f[0] == "symmetric":
        return (x1 * y2 - x2 * y1) / 2 * f[1]
    if f[0] == "flux":
        u1, v1, u2, v2 = x1 - f[2], y1 - f[3], x2 - f[2], y2 - f[3]
        n = torch.sqrt(u1 * u1 + v1 * v1) * torch.sqrt(u2 * u2 + v2 * v2)
        det = u1 * v2 - u2 * v1
        far = n > 1e-10
        c = (u1 * u2 + v1 * v2) / torch.where(far, n, torch.ones_like(n)) / (1 + 1e-11)
        return torch.where(far, torch.acos(c) * torch.sign(det) * f[1] / (2 * math.pi), torch.zeros_like(n))
    return torch.zeros_like(x1)


def _phase(li):
    return torch.polar(torch.ones_like(li), -2 * math.pi * li)


def _hops(Lx, Ly, torus, field, V):
    """H[s, s + x], H[s, s + y] (0 where there is no bond) and the diagonal, as Lx x Ly arrays."""
    x, y = torch.meshgrid(torch.arange(1, Lx + 1, dtype=torch.float64, device=DEV),
                          torch.arange(1, Ly + 1, dtype=torch.float64, device=DEV), indexing="ij")
    hx, hy = _phase(_line(field, x, y, x + 1, y)), _phase(_line(field, x, y, x, y + 1))
    if not torus:
        hx, hy = hx * (x < Lx), hy * (y < Ly)
    return hx, hy, torch.as_tensor(V, device=DEV).reshape(Lx, Ly)


def _square(hx, hy, V):
    def H(p):  # p: ... x Lx x Ly
        return (V * p + hx * p.roll(-1, -2) + (hx.conj() * p).roll(1, -2)
                + hy * p.roll(-1, -1) + (hy.conj() * p).roll(1, -1))
    return H


def _brick(case, seed):
    a, b = case["a"], case["b"]
    t1, B, _ = _graphene(case)
    j1, j2 = torch.meshgrid(torch.arange(1, a + 1, dtype=torch.float64, device=DEV),
                            torch.arange(1, b + 1, dtype=torch.float64, device=DEV), indexing="ij")
    q = math.sqrt(3) / 6
    ax, ay = j1 + 0.5 * j2, 3 * q * j2
    V = torch.as_tensor(_graphene_onsite(case, seed), device=DEV).reshape(a, b, 2)
    h = [t1 * _phase(_line(("symmetric", B), ax, ay, ax + dx, ay + dy)) for dx, dy in ((0.5, q), (-0.5, q), (0.0, -2 * q))]
    h[1][0], h[2][:, 0] = 0, 0

    def H(p):  # p: ... x a x b x 2; A(j) meets B(j), B(j1 - 1, j2) and B(j1, j2 - 1)
        A, C = p[..., 0], p[..., 1]
        up = h[0] * C + h[1] * C.roll(1, -2) + h[2] * C.roll(1, -1)
        dn = h[0].conj() * A + (h[1].conj() * A).roll(-1, -2) + (h[2].conj() * A).roll(-1, -1)
        return V * p + torch.stack([up, dn], -1)
    return H


def _evolve(H, p, dt, norm):
    """exp(-i H dt) p by its Taylor series to 1e-18; ``norm`` bounds |H|."""
    y, k, size = p.clone(), 0, 1.0
    while size > 1e-18:
        k += 1
        size *= norm * abs(dt) / k
        p = H(p) * (-1j * dt / k)
        y += p
    return y


def _dense(hx, hy, V):
    """The matrix of a square lattice."""
    N = V.numel()
    eye = torch.eye(N, dtype=torch.complex128, device=DEV).reshape(N, *V.shape)
    return _square(hx, hy, V)(eye).reshape(N, N).T.contiguous()


def _bond_values(hx, hy, cx, cy, torus):
    """2 Im(H[s, s'] P[s', s]) on every bond: +x bonds, then +y bonds; cx, cy hold P[s', s]."""
    jx, jy = 2 * (hx * cx).imag, 2 * (hy * cy).imag
    if not torus:
        jx, jy = jx[:-1], jy[:, :-1]
    return torch.cat([jx.reshape(-1), jy.reshape(-1)])


def exact(case, seed):
    kind = case["kind"]
    if kind == "ramp":
        Lx, Ly = case["Lx"], case["Ly"]
        N, V = Lx * Ly, _disorder(seed, Lx * Ly, 1.0)
        T = _projector(seed, Lx, Ly).T.contiguous()  # row j: column j of P
        sites = torch.arange(N, device=DEV).reshape(Lx, Ly)
        rho, J = [], []
        for k in range(case["steps"]):
            hx, hy, d = _hops(Lx, Ly, False, _ramp_field(case, 0.1 * k), V)
            for _ in range(2):  # P <- U (U P)^H, Hermitian P
                T = _evolve(_square(hx, hy, d), T.reshape(N, Lx, Ly), 0.1, 5.0).reshape(N, N).T.conj().contiguous()
            rho.append(T.diagonal().real.clone())
            J.append(_bond_values(hx, hy, T[sites, sites.roll(-1, 0)], T[sites, sites.roll(-1, 1)], False))
        return {"density": torch.stack(rho), "currents": torch.stack(J), "P": T}
    if kind == "kets":
        Lx, Ly, M, torus = case["Lx"], case["Ly"], case["M"], case["torus"]
        N, V = Lx * Ly, _disorder(seed, Lx * Ly, 2.0)
        X = _kets(seed, N, M, torch.complex128 if case["form"] == "c64" else torch.complex64)
        rho = torch.zeros(case["steps"], Lx, Ly, dtype=torch.float64, device=DEV)
        cx, cy = rho.to(torch.complex128), rho.to(torch.complex128)
        ham = [_hops(Lx, Ly, torus, _kets_field(case, 0.05 * k), V) for k in range(case["steps"])]
        out = torch.empty(M, N, dtype=torch.complex128, device=DEV)
        for m in range(0, M, 256):
            p = X[m:m + 256].to(torch.complex128).reshape(-1, Lx, Ly)
            for k, h in enumerate(ham):
                p = _evolve(_square(*h), p, 0.05, 5.0)
                rho[k] += (p.real ** 2 + p.imag ** 2).sum(0)
                cx[k] += (p.roll(-1, -2) * p.conj()).sum(0)
                cy[k] += (p.roll(-1, -1) * p.conj()).sum(0)
            out[m:m + 256] = p.reshape(-1, N)
        J = [_bond_values(h[0], h[1], cx[k], cy[k], torus) for k, h in enumerate(ham)]
        return {"density": rho.reshape(-1, N), "currents": torch.stack(J), "kets": out}
    if kind == "graphene":
        a, b, M = case["a"], case["b"], case["M"]
        t1, _, dt = _graphene(case)
        H = _brick(case, seed)
        p = _kets(seed, 2 * a * b, M, torch.complex128 if M == 1 else torch.complex64).to(torch.complex128)
        p = p.reshape(M, a, b, 2)
        rho = []
        for _ in range(case["steps"]):
            p = _evolve(H, p, dt, 3 * abs(t1) + 0.3)
            rho.append((p.real ** 2 + p.imag ** 2).sum(0).reshape(-1))
        return {"density": torch.stack(rho), "kets": p.reshape(M, -1)}
    if kind == "batch":
        out, r = [], np.random.default_rng([int(seed), 3])
        for i, L in enumerate(_sides(case)):
            V, flux = _disorder(seed + 1000 * i, L * L, r.uniform(0, 3)), r.uniform(0, 0.3)
            H = _square(*_hops(L, L, False, ("flux", flux, L // 2 + 0.5, L // 2 + 0.5), V))
            T = _hermitian(seed + 1000 * i, L * L).T.to(torch.complex128)
            for _ in range(2):
                T = torch.cat([_evolve(H, t.reshape(-1, L, L), 0.1, 5.5).reshape(-1, L * L) for t in T.split(2048)])
                T = T.T.conj().contiguous()
            out.append(T.to(torch.complex128))
        return out
    if kind == "adjoint":
        L, M, n = case["L"], case["M"], case["steps"]
        V, B, target, point, spi = _control(case, seed)
        V = torch.as_tensor(V, device=DEV).requires_grad_()
        B = torch.as_tensor(B, device=DEV).requires_grad_()
        target = torch.as_tensor(target, device=DEV)

        def step(k, p):
            return _evolve(_square(*_hops(L, L, False, ("flux", B[k // spi], *point), V)), p, 0.05, 4.2)
        p0 = torch.as_tensor(_standing_waves(L, M), device=DEV).to(torch.complex128).reshape(-1, L, L)
        states = [p0]
        with torch.no_grad():
            for k in range(n):
                states.append(step(k, states[-1]))
            diff = (states[-1].real ** 2 + states[-1].imag ** 2).sum(0).reshape(-1) - target
            loss, lam = (diff ** 2).sum(), 4 * diff.reshape(L, L) * states[-1]
        gV, gB = torch.zeros_like(V), torch.zeros_like(B)
        for k in range(n - 1, -1, -1):
            p = states[k].detach().requires_grad_()
            q = step(k, p)
            gp, dV, dB = torch.autograd.grad(q, [p, V, B], grad_outputs=lam)
            gV, gB, lam = gV + dV, gB + dB, gp
            states.pop()
        return {"loss": float(loss), "gV": gV, "gB": gB}
    if kind == "kpm":
        L, R, nmom = case["L"], case["R"], case["nmom"]
        V = _disorder(seed, L * L, 2.0)
        lo, hi = V.min() - 4.0, V.max() + 4.0
        lo, hi = lo - 1e-3 * (hi - lo), hi + 1e-3 * (hi - lo)
        a, b = (hi - lo) / 2, (hi + lo) / 2
        H = _square(*_hops(L, L, True, ("landau", 0.01), V))
        mu = torch.zeros(nmom + 2, dtype=torch.float64, device=DEV)
        for v in _phase_vectors(seed, L * L, R).reshape(R, L, L).split(64):
            t0, t1 = v, (H(v) - b * v) / a
            m0, m1 = (v.conj() * v).sum().real, (v.conj() * t1).sum().real
            for k in range(nmom // 2 + 1):  # mu_2k = 2 <T_k|T_k> - mu_0, mu_2k+1 = 2 <T_k+1|T_k> - mu_1
                if 2 * k < nmom:
                    mu[2 * k] += 2 * (t0.conj() * t0).sum().real - m0
                    mu[2 * k + 1] += 2 * (t1.conj() * t0).sum().real - m1
                t0, t1 = t1, 2 * (H(t1) - b * t1) / a - t0
        return {"mu": mu[:nmom], "bounds": np.array([lo, hi])}
    Lx, Ly = case["Lx"], case["Ly"]
    h = _hops(Lx, Ly, False, ("flux", 0.2, Lx // 2 + 0.5, Ly // 2 + 0.5), _disorder(seed, Lx * Ly, 2.0))
    w, v = torch.linalg.eigh(_dense(*h))
    f = 0.5 * (1 - torch.tanh(w / (2 * case["T"]))) if kind == "fermi" else (w <= 0).to(torch.float64)
    return ((v * f) @ v.conj().T).T
