"""Timed workloads of the mesh solver, each through the library's public entry points.

A case is a dict of plain values; `kind` says which part of a run it is:

  eigh      mg_eigh_batched_noalloc on the symmetric blocks of an HFB step
  density   DeriveBasis, UpdateDensities and the read-out of the densities
  hpsi      DeriveBasis and h.psi of a basis on the symmetry-free box
  step      one gradient step of spinors that the host program keeps: upload,
            DeriveBasis, GradDesc with its Gram-Schmidt, download
  coulomb   moments and one cold Coulomb solve for a new proton density
  pairing   one HFB pairing step of uploaded spinors
  evolve    Evolve passes (the whole iteration) and the read-out of the state

Host buffers are page-locked, as in a program that drives the library every
step; spinors are harmonic-oscillator states with a seeded perturbation, the
fields Woods-Saxon wells with their spin-orbit form factor.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from mocca_gb300 import (MG_CAN_BASIS, MG_FP64, MG_HF_BASIS, MG_MIXED, MG_PAIRING_HF,
                         MG_PAIRING_HFB, SLY4, RunParams, _abi)
from mocca_gb300.mesh import MeshState

DX = 0.8
DT, MOMENTUM = 0.010, 0.3
F64 = torch.float64


def listed():
    return [
        # the four blocks (two isospins, two parities) of the HFB matrix of the
        # benchmark configuration, 24^3 with nwt=160
        {"name": "eigh_4x92", "kind": "eigh", "nb": 4, "n0": 92, "n1": 90, "n2": 70, "n3": 68},
        # densities of the README Mg24 run (10^3, 40 spwfs): the smallest mesh
        # call, made thousands of times in a run
        {"name": "density_fp64_10c", "kind": "density", "prec": "fp64", "nx": 10, "ny": 10,
         "nz": 10, "nwt": 40},
        # the same at the benchmark configuration in the FP64 form (parity runs,
        # the polish that ends a mixed run)
        {"name": "density_fp64_24c", "kind": "density", "prec": "fp64", "nx": 24, "ny": 24,
         "nz": 24, "nwt": 160},
        # a mid-size nucleus in a box with three different, odd line lengths, as
        # in a batch of uneven instances, mixed form
        {"name": "density_mixed_odd", "kind": "density", "prec": "mixed", "nx": 21, "ny": 23,
         "nz": 27, "nwt": 114},
        # the symmetry-free microbenchmark box (32^3, 200 spwfs)
        {"name": "hpsi_fp64_full32", "kind": "hpsi", "prec": "fp64", "nx": 32, "ny": 32,
         "nz": 32, "nwt": 200},
        # one step of a host program that keeps the spinors, FP64 and mixed; the
        # second is the large configuration (36^3, nwt=300), the heaviest case
        {"name": "step_fp64_24c", "kind": "step", "prec": "fp64", "nx": 24, "ny": 24, "nz": 24,
         "nwt": 160},
        {"name": "step_mixed_36c", "kind": "step", "prec": "mixed", "nx": 36, "ny": 36, "nz": 36,
         "nwt": 300},
        # Coulomb potential of a new density: the default conjugate-gradient
        # solver on the benchmark mesh, the multigrid on a large one
        {"name": "coulomb_cg_24c", "kind": "coulomb", "solver": 1, "nx": 24, "ny": 24, "nz": 24},
        {"name": "coulomb_mg_48c", "kind": "coulomb", "solver": 2, "nx": 48, "ny": 48, "nz": 48},
        # one pairing step of a mid-size nucleus, FP64
        {"name": "pairing_fp64_18c", "kind": "pairing", "prec": "fp64", "nx": 18, "ny": 17,
         "nz": 20, "nwt": 96},
        # whole iterations: the README Mg24 input (FP64, MixingScheme 2,
        # ParameterEstimation 1, Q20 constraint), and the benchmark
        # configuration in the mixed form
        {"name": "evolve_fp64_10c", "kind": "evolve", "prec": "fp64", "nx": 10, "ny": 10,
         "nz": 10, "nwt": 40, "neutrons": 12, "protons": 12, "estimate": True, "iters": 5},
        {"name": "evolve_mixed_24c", "kind": "evolve", "prec": "mixed", "nx": 24, "ny": 24,
         "nz": 24, "nwt": 160, "neutrons": 28, "protons": 28, "estimate": False, "iters": 5},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _mesh(rng, lo, hi):
    n = rng.randint(lo, hi)
    return {"nx": n, "ny": max(lo, n - rng.randint(0, 2)), "nz": min(hi, n + rng.randint(0, 3))}


def draw(rng):
    kind = rng.choice(["eigh", "density", "density", "hpsi", "step", "step", "coulomb", "pairing",
                       "evolve"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "eigh":
        nb = rng.choice([1, 2, 4, 4, 4])
        n = [_log_int(rng, 16, 128) for _ in range(4)]
        return {"kind": kind, "nb": nb, "n0": n[0], "n1": n[1], "n2": n[2], "n3": n[3]}
    if kind == "density":
        return {"kind": kind, "prec": prec, **_mesh(rng, 10, 30), "nwt": 2 * _log_int(rng, 12, 90)}
    if kind == "hpsi":
        return {"kind": kind, "prec": prec, **_mesh(rng, 16, 32), "nwt": 2 * _log_int(rng, 12, 90)}
    if kind == "step":
        hi = 36 if prec == "mixed" else 28
        return {"kind": kind, "prec": prec, **_mesh(rng, 10, hi),
                "nwt": 2 * _log_int(rng, 20, 130 if prec == "mixed" else 80)}
    if kind == "coulomb":
        return {"kind": kind, "solver": 1, **_mesh(rng, 10, 36)}
    if kind == "pairing":
        return {"kind": kind, "prec": prec, **_mesh(rng, 12, 22), "nwt": 2 * _log_int(rng, 24, 70)}
    half = _log_int(rng, 6, 20)
    return {"kind": kind, "prec": prec, **_mesh(rng, 12, 22), "nwt": 2 * round(2.8 * half),
            "neutrons": 2 * half, "protons": 2 * half, "estimate": False, "iters": 5}


# ---- inputs ---------------------------------------------------------------------


def _full(case):
    return case["kind"] == "hpsi"


def _axes(case):
    half = not _full(case)
    out = []
    for k in ("nx", "ny", "nz"):
        i = torch.arange(case[k], dtype=F64, device="cuda")
        out.append(DX * (i + 0.5) if half else DX * (i + 0.5) - 0.5 * DX * case[k])
    return out


def _volume(case):
    return case["nx"] * case["ny"] * case["nz"]


def _dv(case):
    return DX ** 3 * (1.0 if _full(case) else 8.0)


def _hermite(n, x):
    h0, h1 = torch.ones_like(x), 2 * x
    if n == 0:
        return h0
    for k in range(1, n):
        h0, h1 = h1, 2 * x * h1 - 2 * k * h0
    return h1


def _outer(fx, fy, fz):
    return fz[:, None, None] * fy[None, :, None] * fx[None, None, :]


def _particles(case):
    """(N, Z) of the nucleus that a basis of this size holds."""
    return (case["neutrons"], case["protons"]) if "neutrons" in case else (
        2 * max(2, round(case["nwt"] / 5.6)),) * 2


def _spinors(case, seed):
    """Spinors [nwt, 4, nz, ny, nx] on the GPU, quantum numbers [nwt, 4] and
    single-particle energies [nwt].

    EV8 box: the lowest states of a triaxial oscillator, each in the spinor
    component that its mirror parities allow, plus a uniform perturbation of
    1e-3 of its maximum.  Full box: random Gaussian-Hermite functions."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    nwt = case["nwt"]
    x, y, z = _axes(case)
    psi = torch.zeros((nwt, 4, case["nz"], case["ny"], case["nx"]), dtype=F64, device="cuda")
    qn = np.zeros((nwt, 4), dtype=np.int32)
    en = np.zeros(nwt)
    if _full(case):
        for i in range(nwt):
            for comp in range(4):
                w, c, d = rng.uniform(1.5, 3.0), rng.uniform(-3.0, 3.0, 3), rng.integers(0, 4, 3)
                f = [_hermite(int(d[a]), (g - c[a]) / w) * torch.exp(-0.5 * ((g - c[a]) / w) ** 2)
                     for a, g in enumerate((x, y, z))]
                psi[i, comp] = _outer(*f)
        qn[:, 0] = np.where(np.arange(nwt) < nwt // 2, -1, 1)
    else:
        A = sum(_particles(case))
        hw = 41.0 * A ** (-1.0 / 3.0)
        scale = np.array([1.04, 0.98, 0.94]) * (1.0 + rng.uniform(-0.01, 0.01, 3))
        b = np.sqrt(41.47 / (hw * scale))
        orbitals = sorted(((i, j, k) for i in range(14) for j in range(14) for k in range(14)
                           if i + j + k < 14),
                          key=lambda q: (sum(q), -q[0], -q[1]))
        comp = {(0, 0): 0, (1, 1): 1, (1, 0): 2, (0, 1): 3}
        for it, (first, count) in enumerate(((0, nwt // 2), (nwt // 2, nwt - nwt // 2))):
            f = [[_hermite(q, g / b[a]) * torch.exp(-0.5 * (g / b[a]) ** 2) for q in range(14)]
                 for a, g in enumerate((x, y, z))]
            for k, (i, j, l) in enumerate(orbitals[:count]):
                c = comp[(i % 2, j % 2)]
                psi[first + k, c] = _outer(f[0][i], f[1][j], f[2][l])
                parity = (-1) ** l if c in (0, 1) else -((-1) ** l)
                qn[first + k] = (2 * it - 1, parity, 1, 1)
                en[first + k] = (-50.0 + 2.0 * it
                                 + hw * float(scale @ np.array([i + 0.5, j + 0.5, l + 0.5])))
        top = psi.flatten(1).abs().amax(1)
        for i in range(nwt):
            u = torch.rand(psi[i].shape, dtype=F64, device="cuda", generator=gen)
            psi[i] += 1e-3 * top[i] * (2.0 * u - 1.0)
    psi /= ((psi ** 2).flatten(1).sum(1) * _dv(case)).sqrt()[:, None, None, None, None]
    return psi, qn, en


def _occupations(case):
    """v^2 of a filled well with a diffuse edge, times two for the partner states."""
    k = np.arange(case["nwt"]) % max(1, case["nwt"] // 2)
    n0 = sum(_particles(case)) / 4.0
    return 2.0 / (1.0 + np.exp(np.clip((k + 0.5 - n0) / (0.06 * case["nwt"] + 1.0), -60, 60)))


def _fields(case, seed):
    """U, B, grad B, W, div W of a triaxial Woods-Saxon well, both isospins."""
    rng = np.random.default_rng(seed + 17)
    x, y, z = _axes(case)
    Z, Y, X = torch.meshgrid(z, y, x, indexing="ij")
    s = np.array([0.97, 1.0, 1.08]) * (1.0 + rng.uniform(-0.02, 0.02, 3))
    r = (X ** 2 / s[0] ** 2 + Y ** 2 / s[1] ** 2 + Z ** 2 / s[2] ** 2).sqrt()
    R, a = 1.2 * sum(_particles(case)) ** (1.0 / 3.0), 0.65
    f = 1.0 / (1.0 + torch.exp((r - R) / a))
    df = -f * (1 - f) / a / r
    g = torch.stack([(df * X / s[0] ** 2), (df * Y / s[1] ** 2), (df * Z / s[2] ** 2)]).flatten(1)
    V = _volume(case)
    U = torch.stack([-52.0 * f, -48.0 * f]).reshape(2, V)
    B = torch.stack([8.0 * f, 7.5 * f]).reshape(2, V)
    nB = torch.stack([8.0 * g, 7.5 * g])
    W = torch.zeros((2, 3, 3, V), dtype=F64, device="cuda")
    for k, m, n in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        for it in range(2):
            W[it, n, m] = -(60.0 - 2.0 * it) * g[k]
            W[it, m, n] = (60.0 - 2.0 * it) * g[k]
    return U, B, nB, W, torch.zeros((2, 3, V), dtype=F64, device="cuda")


def _proton_density(case, seed):
    """rho of neutrons and protons [2, V]: deformed Fermi distributions."""
    rng = np.random.default_rng(seed)
    x, y, z = _axes(case)
    Z, Y, X = torch.meshgrid(z, y, x, indexing="ij")
    s = np.array([0.95, 1.0, 1.12]) * (1.0 + rng.uniform(-0.04, 0.04, 3))
    r = (X ** 2 / s[0] ** 2 + Y ** 2 / s[1] ** 2 + Z ** 2 / s[2] ** 2).sqrt()
    R = 0.42 * DX * min(case["nx"], case["ny"], case["nz"])
    f = 1.0 / (1.0 + torch.exp((r - min(R, 6.5)) / 0.55))
    return torch.stack([0.085 * f, 0.075 * f]).reshape(2, -1)


def _eigh_matrices(case, seed):
    """HFB-shaped blocks [[e, D], [D, -e]] (odd sizes: one more level)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    sizes = [case["n%d" % b] for b in range(case["nb"])]
    ld = max(sizes)
    a = torch.zeros((case["nb"], ld, ld), dtype=F64, device="cuda")
    for b, n in enumerate(sizes):
        h = n // 2
        e = torch.linspace(-38.0, 26.0, h, dtype=F64, device="cuda")
        e = e + 0.7 * torch.rand(h, dtype=F64, device="cuda", generator=gen)
        d = torch.randn((h, h), dtype=F64, device="cuda", generator=gen)
        idx = torch.arange(h, device="cuda")
        d = 0.12 * (d + d.T) * torch.exp(-0.2 * (idx[:, None] - idx[None, :]).abs().to(F64))
        d[idx, idx] = 1.3
        d = d * torch.exp(-((e[:, None] + e[None, :]) / 60.0) ** 2)
        a[b, :h, :h] = torch.diag(e)
        a[b, h:2 * h, h:2 * h] = -torch.diag(e)
        a[b, :h, h:2 * h] = d
        a[b, h:2 * h, :h] = d.T
        if n % 2:
            a[b, n - 1, n - 1] = 31.0
    return a, sizes, ld


# ---- states and passes ------------------------------------------------------------


def _pinned(*shape):
    return torch.empty(shape, dtype=F64, pin_memory=True)


def _ptr(t):
    return C.cast(t.data_ptr(), _abi._D)


def _grids(t):
    n, step = t.shape[0], t[0].numel() * 8
    return (C.c_void_p * n)(*[t.data_ptr() + i * step for i in range(n)])


def _call(s, name, *args, **kw):
    st = getattr(s["g"].lib, name)(s["g"].h, *args)
    return _abi.check(name, st, **kw)


def _params(case, **kw):
    n, z = _particles(case) if "nwt" in case else (40, 40)
    sym = 0 if _full(case) else 1
    return RunParams(nx=case["nx"], ny=case["ny"], nz=case["nz"], dx=DX, pc=sym, sc=sym, tsc=sym,
                     nwt=case.get("nwt", 2), neutrons=float(n), protons=float(z),
                     precision=MG_MIXED if case.get("prec") == "mixed" else MG_FP64, **kw)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "eigh":
        a, sizes, ld = _eigh_matrices(case, seed)
        nb = case["nb"]
        s.update(a=a, nb=nb, ld=ld, sizes=(C.c_int * nb)(*sizes),
                 w=torch.zeros((nb, ld), dtype=F64, device="cuda"),
                 z=torch.zeros((nb, ld, ld), dtype=F64, device="cuda"),
                 info=torch.zeros(nb, dtype=torch.int32, device="cuda"),
                 half=[n // 2 for n in sizes])
        return s
    V = _volume(case)
    if kind == "coulomb":
        s["g"] = MeshState(_params(case, coulomb_solver=case["solver"], coulomb_max=1000), SLY4)
        s["rho"] = _pinned(2, V)
        s["rho"].copy_(_proton_density(case, seed))
        s["coulomb"], s["exchange"] = _pinned(V), _pinned(V)
        return s
    nwt = case["nwt"]
    if kind == "evolve":
        kw = dict(pairing=MG_PAIRING_HFB)
        if case["estimate"]:
            kw.update(mixing_scheme=2, parameter_estimation=1)
        g = s["g"] = MeshState(_params(case, **kw), SLY4)
        # a triaxial start: no level of it is degenerate
        g.NilssonStart(nwt // 2, ho=(0.21, 0.196, 0.18), amplitude=1e-3, seed=seed)
        g.set_pairing()
        if case["estimate"]:
            g.add_constraint(2, 0, 50.0, iteration=10)
        g.Start()
        g.Evolve(15, DT, MOMENTUM)
        s.update(iters=case["iters"], psi=_pinned(nwt, 4 * V), e=_pinned(nwt), disp=_pinned(nwt),
                 rho=_pinned(2, V), tau=_pinned(2, V))
        s["out_grids"] = _grids(s["psi"])
        s["energy"] = _abi.MgEnergyTerms()
        return s
    psi, qn, en = _spinors(case, seed)
    s["psi"] = _pinned(nwt, 4 * V)
    s["psi"].copy_(psi.reshape(nwt, -1))
    del psi
    s["in_grids"] = _grids(s["psi"])
    pairing = MG_PAIRING_HFB if kind == "pairing" else MG_PAIRING_HF
    g = s["g"] = MeshState(_params(case, coulomb_solver=0, pairing=pairing), SLY4)
    q = np.ascontiguousarray(qn.reshape(-1))
    _call(s, "mg_upload_spinors", MG_HF_BASIS, s["in_grids"], q.ctypes.data_as(_abi._I), 0, nwt)
    g.synchronize()
    g.set_energies(en)
    s["energies"] = en
    if kind == "density":
        g.set_occupations(_occupations(case))
        s.update(rho=_pinned(2, V), tau=_pinned(2, V), nablaj=_pinned(2, V),
                 derrho=_pinned(2, 3, V), laprho=_pinned(2, V))
    elif kind == "pairing":
        pp = _abi.MgPairingParams.defaults()
        for it in range(2):
            pp.fermi_start[it] = float(np.sort(en[:nwt // 2])[_particles(case)[it] // 2])
        g.set_pairing(pp)
        s["rho"] = _proton_density(case, seed).cpu()
        g.set_densities(rho=s["rho"].numpy())
        par = qn[:, 1] > 0
        s["blocks"] = []
        for b in range(4):
            h = int(((qn[:, 0] == (1 if b >= 2 else -1)) & (par == bool(b % 2))).sum())
            s["blocks"].append([_pinned(2 * h, 2 * h) for _ in range(3)])
        s.update(re=_pinned(2, V), dfac=_pinned(2, V), occ=_pinned(nwt),
                 info=_abi.MgPairingInfo())
    else:
        g.set_potentials(*(f.cpu().numpy() for f in _fields(case, seed)))
        s.update(e=_pinned(nwt), disp=_pinned(nwt), out=_pinned(nwt, 4 * V))
        s["out_grids"] = _grids(s["out"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "eigh":
        lib = _abi.load()
        _abi.check("mg_eigh_batched_noalloc", lib.mg_eigh_batched_noalloc(
            s["nb"], s["sizes"], s["ld"], s["a"].data_ptr(), s["w"].data_ptr(), s["z"].data_ptr(),
            s["info"].data_ptr(), torch.cuda.current_stream().cuda_stream))
        # the block's density matrix, as an HFB step forms it: the sum over the
        # lower half of the spectrum (vectors alone are defined up to a sign)
        rho = [s["z"][b, :, :h] @ s["z"][b, :, :h].T for b, h in enumerate(s["half"])]
        return {"w": s["w"], "rho": rho}
    g = s["g"]
    if kind == "density":
        _call(s, "mg_derive_basis", MG_HF_BASIS)
        _call(s, "mg_update_densities")
        keys = ("rho", "tau", "nablaj", "derrho", "laprho")
        _call(s, "mg_get_densities", *(_ptr(s[k]) for k in keys))
        return {k: s[k] for k in keys}
    if kind == "hpsi":
        _call(s, "mg_derive_basis", MG_HF_BASIS)
        _call(s, "mg_hpsi", MG_HF_BASIS, _ptr(s["out"]), _ptr(s["e"]), _ptr(s["disp"]))
        return {"hpsi": s["out"], "e": s["e"], "disp": s["disp"]}
    if kind == "step":
        nwt = len(s["e"])
        _call(s, "mg_upload_spinors", MG_HF_BASIS, s["in_grids"], None, 0, nwt)
        _call(s, "mg_derive_basis", MG_HF_BASIS)
        _call(s, "mg_grad_desc", C.c_double(DT), C.c_double(MOMENTUM))
        _call(s, "mg_download_spinors", MG_HF_BASIS, s["out_grids"], 0, nwt)
        _call(s, "mg_get_energies", MG_HF_BASIS, _ptr(s["e"]), _ptr(s["disp"]))
        return {"psi": s["out"], "e": s["e"], "disp": s["disp"]}
    if kind == "coulomb":
        _call(s, "mg_set_densities", _ptr(s["rho"]), None, None, None, None)
        _call(s, "mg_calculate_moments")
        _call(s, "mg_coulomb_reset")
        g.SolveCoulomb()
        _call(s, "mg_get_potentials", None, None, None, None, None, _ptr(s["coulomb"]),
              _ptr(s["exchange"]))
        return {"coulomb": s["coulomb"], "exchange": s["exchange"]}
    if kind == "pairing":
        nwt = len(s["occ"])
        _call(s, "mg_upload_spinors", MG_HF_BASIS, s["in_grids"], None, 0, nwt)
        _call(s, "mg_solve_pairing", C.byref(s["info"]), allow_not_converged=True)
        for b in range(4):
            g.lib.mg_get_hfb_block(g.h, b, *(_ptr(m) for m in s["blocks"][b]))
        _call(s, "mg_get_pairing_field", _ptr(s["re"]), None, _ptr(s["dfac"]))
        _call(s, "mg_get_occupations", MG_CAN_BASIS, _ptr(s["occ"]))
        return {"blocks": s["blocks"], "field": s["re"], "dfac": s["dfac"], "occ": s["occ"],
                "fermi": np.array(list(s["info"].fermi))}
    nwt = len(s["e"])
    _call(s, "mg_iterate", s["iters"], C.c_double(DT), C.c_double(MOMENTUM),
          C.byref(s["energy"]), allow_not_converged=True)
    _call(s, "mg_download_spinors", MG_HF_BASIS, s["out_grids"], 0, nwt)
    _call(s, "mg_get_energies", MG_HF_BASIS, _ptr(s["e"]), _ptr(s["disp"]))
    _call(s, "mg_get_densities", _ptr(s["rho"]), _ptr(s["tau"]), None, None, None)
    return {"psi": s["psi"], "e": s["e"], "rho": s["rho"], "tau": s["tau"],
            "total": float(s["energy"].total)}


# ---- work that a pass cannot do without ---------------------------------------------


def _block_sizes(case):
    """(isospin, parity) block sizes of an EV8 basis, about equal halves."""
    h = case["nwt"] / 4.0
    return [h] * 4


def work(case):
    kind = case["kind"]
    if kind == "eigh":
        n = [case["n%d" % b] for b in range(case["nb"])]
        # tridiagonal reduction, QL and back-transformation; the projector
        return {"bytes": sum(8 * (2 * k * k + k) for k in n), "flops": sum(10 * k ** 3 for k in n)}
    V = _volume(case)
    lines = case["nx"] + case["ny"] + case["nz"]
    if kind == "coulomb":
        # the separable solve: forward and back along each axis
        return {"bytes": 8 * 5 * V, "flops": 4 * V * lines + 120 * V}
    nwt = case["nwt"]
    psi = 8 * 4 * V * nwt
    derive = 16 * V * nwt * lines   # four components, first and second derivative per axis
    gs = sum(2 * h * h * 4 * V for h in _block_sizes(case))
    pair = sum(3 * 2 * h * h * 4 * V for h in _block_sizes(case))
    diag = sum(2 * 10 * (2 * h) ** 3 for h in _block_sizes(case))
    if kind == "density":
        return {"bytes": psi + 8 * 14 * V, "flops": derive + 100 * V * nwt}
    if kind == "hpsi":
        return {"bytes": 2 * psi + 8 * 34 * V, "flops": derive + 200 * V * nwt}
    if kind == "step":
        return {"bytes": 4 * psi + 8 * 34 * V, "flops": derive + 210 * V * nwt + gs}
    if kind == "pairing":
        return {"bytes": 2 * psi + 8 * 6 * V, "flops": pair + diag}
    # spinors and their update history in and out, the canonical spinors out
    return {"bytes": case["iters"] * (5 * psi + 8 * 60 * V) + psi,
            "flops": case["iters"] * (2 * derive + 510 * V * nwt + gs + pair + diag)}


# ---- plain 64-bit results -------------------------------------------------------------


def _lagrange(n, folded, sign):
    """First and second derivative matrices of a line (Baye and Heenen 1986):
    folded on a half line of even (sign 1) or odd (-1) functions, or the
    full line with zero extension."""
    N = 2 * n if folded else n
    k = np.arange(1, N)
    s, c, sg = np.sin(np.pi * k / N), np.cos(np.pi * k / N), (-1.0) ** k
    c1 = np.concatenate([[0.0], np.pi / (N * DX) * sg / s])
    c2 = np.concatenate([[-(np.pi ** 2) / (3 * DX ** 2) * (1 - 1 / N ** 2)],
                         -sg * 2 * (np.pi / (N * DX)) ** 2 * c / s ** 2])
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    d1, d2 = np.sign(i - j) * c1[abs(i - j)], c2[abs(i - j)]
    if folded:
        d1, d2 = d1 + sign * c1[i + j + 1], d2 + sign * c2[i + j + 1]
    return torch.from_numpy(d1).cuda(), torch.from_numpy(d2).cuda()


def _apply(m, f, axis):
    """m along x, y or z (0, 1, 2) of [..., z, y, x]."""
    return torch.movedim(torch.movedim(f, -1 - axis, -1) @ m.T, -1, -1 - axis)


def _derivatives(f, signs, folded):
    """d/dx, d/dy, d/dz and the Laplacian of grids [..., z, y, x]."""
    der, lap = [], 0.0
    for axis in range(3):
        d1, d2 = _lagrange(f.shape[-1 - axis], folded, signs[axis])
        der.append(_apply(d1, f, axis))
        lap = lap + _apply(d2, f, axis)
    return torch.stack(der), lap


def _signs(parity, comp):
    """Mirror signs along x, y, z of component comp (0..3) of an EV8 spinor of
    signature and time simplex one."""
    return (1 if comp in (0, 3) else -1, 1 if comp in (0, 2) else -1,
            parity if comp in (0, 1) else -parity)


def _spinor_derivatives(psi, qn, folded):
    """[nwt, 3, 4, z, y, x] and [nwt, 4, z, y, x]."""
    der = torch.empty((psi.shape[0], 3) + psi.shape[1:], dtype=F64, device="cuda")
    lap = torch.empty_like(psi)
    for parity in sorted(set(qn[:, 1].tolist())):
        rows = torch.from_numpy(np.nonzero(qn[:, 1] == parity)[0]).cuda()
        for comp in range(4):
            d, l = _derivatives(psi[rows, comp], _signs(parity, comp), folded)
            der[rows, :, comp] = d.transpose(0, 1)
            lap[rows, comp] = l
    return der, lap


def _sigma(p, k):
    """sigma_x, sigma_y, sigma_z (k = 0, 1, 2) on components [..., 4, V]."""
    a, b, c, d = p.unbind(-2)
    return torch.stack(((c, d, a, b), (d, -c, -b, a), (a, b, -c, -d))[k], dim=-2)


def _imag(a, b):
    return (a[..., 0, :] * b[..., 1, :] - a[..., 1, :] * b[..., 0, :]
            + a[..., 2, :] * b[..., 3, :] - a[..., 3, :] * b[..., 2, :])


def _exact_density(case, seed):
    psi, qn, _ = _spinors(case, seed)
    der, _ = _spinor_derivatives(psi, qn, True)
    occ = torch.from_numpy(_occupations(case)).cuda()
    V = _volume(case)
    shape = (case["nz"], case["ny"], case["nx"])
    out = {k: [] for k in ("rho", "tau", "nablaj", "derrho", "laprho")}
    for iso in (-1, 1):
        rows = torch.from_numpy(np.nonzero(qn[:, 0] == iso)[0]).cuda()
        p, d, o = psi[rows].flatten(2), der[rows].flatten(3), occ[rows]
        rho = torch.einsum("i,ilv->v", o, p * p)
        out["rho"].append(rho)
        out["tau"].append(torch.einsum("i,imlv->v", o, d * d))
        nj = 0.0
        for i, j, k in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
            nj = nj + _imag(d[:, i], _sigma(d[:, j], k)) - _imag(d[:, j], _sigma(d[:, i], k))
        out["nablaj"].append(torch.einsum("i,iv->v", o, nj))
        dr, lr = _derivatives(rho.reshape(shape), (1, 1, 1), True)
        out["derrho"].append(dr.reshape(3, V))
        out["laprho"].append(lr.reshape(V))
    return {k: torch.stack(v) for k, v in out.items()}


def _exact_hpsi(case, seed):
    psi, qn, _ = _spinors(case, seed)
    V = _volume(case)
    der, lap = _spinor_derivatives(psi, qn, not _full(case))
    U, B, nB, W, dW = _fields(case, seed)
    N, Z = _particles(case)
    mass = (939.565379 + 938.272046) / 2
    kin = 20.73551910 * (1.0 - mass / (N * mass + Z * mass))
    h = torch.empty((case["nwt"], 4, V), dtype=F64, device="cuda")
    for i in range(case["nwt"]):
        it = 0 if qn[i, 0] < 0 else 1
        p, d, l = psi[i].reshape(4, V), der[i].reshape(3, 4, V), lap[i].reshape(4, V)
        w = sum(W[it, nu, mu] * _sigma(d[mu], nu) for mu in range(3) for nu in range(3))
        w = w + sum(0.5 * dW[it, nu] * _sigma(p, nu) for nu in range(3))
        h[i] = (-(B[it] + kin) * l - (nB[it][:, None] * d).sum(0) + U[it] * p
                + torch.stack((w[1], -w[0], w[3], -w[2])))
    p = psi.reshape(case["nwt"], 4 * V)
    h = h.reshape(case["nwt"], 4 * V)
    e = (p * h).sum(1) * _dv(case)
    return p, h, e, (h * h).sum(1) * _dv(case) - e * e, qn


def _exact_step(case, seed):
    p, h, e, disp, qn = _exact_hpsi(case, seed)
    p = p - DT / 6.58211928 * h
    out = torch.empty_like(p)
    for iso in (-1, 1):
        for parity in (-1, 1):
            rows = np.nonzero((qn[:, 0] == iso) & (qn[:, 1] == parity))[0]
            rows = torch.from_numpy(rows[np.argsort(e.cpu().numpy()[rows], kind="stable")]).cuda()
            r = torch.linalg.cholesky(p[rows] @ p[rows].T * _dv(case))
            out[rows] = torch.linalg.solve_triangular(r, p[rows], upper=False)
    return {"psi": out, "e": e, "disp": disp}


def _solid_harmonics(x, y, z, lmax=10):
    """r^l Y_lm (real part, l and m even) of the box's moments."""
    r = (x * x + y * y + z * z).sqrt()
    ct, phi = z / r, torch.atan2(y, x)
    st = (1.0 - ct * ct).sqrt()
    out = []
    for l in range(0, lmax + 1, 2):
        for m in range(0, l + 1, 2):
            pmm = torch.ones_like(ct)
            for q in range(1, m + 1):
                pmm = -pmm * (2 * q - 1) * st
            p0, p1 = pmm, ct * (2 * m + 1) * pmm
            if l == m:
                p1 = pmm
            for q in range(m + 2, l + 1):
                p0, p1 = p1, ((2 * q - 1) * ct * p1 - (q + m - 1) * p0) / (q - m)
            f = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m)
                          / math.factorial(l + m))
            out.append((l, f * r ** l * p1 * torch.cos(m * phi)))
    return r, out


def _exact_coulomb(case, seed):
    rho = _proton_density(case, seed)[1]
    n = (case["nx"], case["ny"], case["nz"])
    axes = [DX * (torch.arange(k + 2, dtype=F64, device="cuda") + 0.5) for k in n]
    Z, Y, X = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    r, sh = _solid_harmonics(X, Y, Z)
    dens = rho.reshape(n[2], n[1], n[0])
    inside = (slice(0, n[2]), slice(0, n[1]), slice(0, n[0]))
    e2 = 1.43996446
    bound = torch.zeros_like(r)
    for l, y in sh:
        q = (y[inside] * dens).sum() * 8 * DX ** 3
        bound = bound + q * e2 * 4 * math.pi / (2 * l + 1) * y / r ** (2 * l + 1)
    bound[inside] = 0.0
    cf = (-1.0 / 12, 4.0 / 3, -5.0 / 2, 4.0 / 3, -1.0 / 12)
    b, eig = -4 * math.pi * e2 * dens, []
    for axis in range(3):
        A = torch.zeros((n[axis], n[axis] + 2), dtype=F64, device="cuda")
        for i in range(n[axis]):
            for q in range(-2, 3):
                A[i, i + q if i + q >= 0 else -(i + q) - 1] += cf[q + 2]
        g = bound[tuple(slice(None) if 2 - a == axis else inside[a] for a in range(3))]
        b = b - _apply(A, g, axis) / DX ** 2
        eig.append(torch.linalg.eigh(A[:, :n[axis]]))
    for axis in range(3):
        b = _apply(eig[axis][1].T, b, axis)
    mu = (eig[2][0][:, None, None] + eig[1][0][None, :, None] + eig[0][0][None, None, :])
    b = b * DX ** 2 / mu
    for axis in range(3):
        b = _apply(eig[axis][1], b, axis)
    return {"coulomb": b.reshape(-1),
            "exchange": -(3 / math.pi) ** (1 / 3.0) * e2 * rho ** (1 / 3.0)}


def _exact_eigh(case, seed):
    a, sizes, ld = _eigh_matrices(case, seed)
    w = torch.zeros((len(sizes), ld), dtype=F64)
    rho = []
    for b, n in enumerate(sizes):
        lam, v = np.linalg.eigh(a[b, :n, :n].cpu().numpy())
        w[b, :n] = torch.from_numpy(lam)
        p = torch.zeros((ld, ld), dtype=F64)
        p[:n, :n] = torch.from_numpy(v[:, :n // 2] @ v[:, :n // 2].T)
        rho.append(p)
    return {"w": w, "rho": rho}


def exact(case, seed):
    kind = case["kind"]
    if kind == "eigh":
        return _exact_eigh(case, seed)
    if kind == "density":
        return _exact_density(case, seed)
    if kind == "hpsi":
        _, h, e, disp, _ = _exact_hpsi(case, seed)
        return {"hpsi": h, "e": e, "disp": disp}
    if kind == "step":
        return _exact_step(case, seed)
    if kind == "coulomb":
        return _exact_coulomb(case, seed)
    return None   # a self-consistent search or an iteration: no closed form
