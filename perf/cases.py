"""Performance cases of the RI-GW engine, measured through its public Python entry points.

Every case is one call (or the short sequence of calls) that a program makes for one result:

* ``g0w0``      one G0W0 solve, ``Engine.g0w0``
* ``batch``     many molecules of uneven sizes in one call, ``Engine.g0w0_batch``
* ``resident``  the drop-in sequence of the Fortran driver: W with its factors kept on the device
                (``polarizability_grid_scalapack``), then Sigma_c (``gw_selfenergy_imag_scalapack``)
* ``aomo``      the AO->MO transform of the W window, ``calculate_eri_3center_mo``
* ``contour``   G0W0 by contour deformation, ``g0w0_contour``
* ``sox``       second-order screened exchange, ``sox_selfenergy_imag_grid``

The inputs have the distributions of ``molgw_b200.synth``: occupied energies uniform in
[-30, -8] eV, empty ones in [0.5, 40] eV, M ~ N(0, s^2) with s such that the largest eigenvalue
of -chi0(i0) is 0.8.  They are drawn on the GPU from the seed alone.
"""
import math
import random

import numpy as np
import torch

HA_EV = 27.21138505
PRECISION = {"fp64": 0, "bf16x3": 1, "ozaki3": 19, "ozaki4": 20, "ozaki5": 21, "ozaki6": 22, "ozaki7": 23}
# Sigma grid of the benchmark workloads
NC, STEP_CALC, NREAL, STEP_REAL, ETA = 50, 0.075, 101, 0.025, 0.01
# real-axis grid of the contour workload; a step that is exact in binary, so that host and device
# agree to the bit on the largest real frequency that a residue asks for
CD_REAL, CD_SIGMA, CD_STEP, CD_ETA = 6, 11, 0.0625, 0.001


# ---------------------------------------------------------------- cases
def listed():
    return [
        # the smallest molecule a user runs (water in cc-pVDZ, 16 frequencies), arrays in host
        # memory as a host program has them: launches and latency
        {"name": "water", "kind": "g0w0", "precision": "fp64", "nocc": 5, "nvirt": 19, "naux": 84,
         "nomega": 16, "qp_only": False, "host": True},
        # a small molecule through the Fortran driver's sequence of calls, odd sizes
        {"name": "resident_367", "kind": "resident", "precision": "fp64", "nocc": 9, "nvirt": 83, "naux": 367,
         "nomega": 24},
        # the ordinary single solve of the benchmark, tensors in device memory
        {"name": "single_840", "kind": "g0w0", "precision": "fp64", "nocc": 21, "nvirt": 207, "naux": 840,
         "nomega": 32, "qp_only": False, "host": False},
        # a larger molecule in FP64
        {"name": "single_2000", "kind": "g0w0", "precision": "fp64", "nocc": 50, "nvirt": 500, "naux": 2000,
         "nomega": 32, "qp_only": False, "host": False},
        # molecules of uneven sizes in one FP64 call, QP energies only
        {"name": "batch_fp64", "kind": "batch", "precision": "fp64", "count": 8, "nocc_min": 5, "nocc_max": 30,
         "sizes": 11, "nomega": 32},
        # the ordinary single solve with chi0 in split bf16
        {"name": "single_840_bf16x3", "kind": "g0w0", "precision": "bf16x3", "nocc": 21, "nvirt": 207, "naux": 840,
         "nomega": 32, "qp_only": False, "host": False},
        # the large instance of the precision sweep, as served
        {"name": "large_4000_bf16x3", "kind": "g0w0", "precision": "bf16x3", "nocc": 100, "nvirt": 1100,
         "naux": 4000, "nomega": 48, "qp_only": True, "host": False},
        # the serving mix: molecules of uneven sizes in one split-precision call
        {"name": "batch_bf16x3", "kind": "batch", "precision": "bf16x3", "count": 16, "nocc_min": 5, "nocc_max": 60,
         "sizes": 4, "nomega": 32},
        # chi0 in four int8 slices, the sliced precision that holds 1 meV on every workload
        {"name": "single_1483_ozaki4", "kind": "g0w0", "precision": "ozaki4", "nocc": 37, "nvirt": 333,
         "naux": 1483, "nomega": 32, "qp_only": False, "host": False},
        # the transform that makes the W window of the ordinary solve, on the device
        {"name": "aomo_840", "kind": "aomo", "precision": "fp64", "nbf": 228, "naux": 840, "nocc": 21},
        # contour deformation with the frequency grids of the reference's water input
        {"name": "contour_480", "kind": "contour", "nocc": 12, "nvirt": 108, "naux": 480, "nomega": 16},
        # the vertex correction beside the ordinary solve
        {"name": "sox_840", "kind": "sox", "nocc": 21, "nvirt": 207, "naux": 840},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _window(rng, naux):
    """Occupied and empty states of a molecule with about this many auxiliary functions."""
    nocc = max(2, int(round(naux / 4.0 / (1.0 + rng.uniform(8.0, 10.0)))))
    return nocc, max(4, int(round(naux / 4.0)) - nocc + rng.randint(-3, 3))


def draw(rng):
    kind = rng.choice(["g0w0"] * 5 + ["batch"] * 2 + ["resident", "aomo", "contour", "sox"])
    if kind == "g0w0":
        prec = rng.choice(["fp64", "fp64", "fp64", "bf16x3", "bf16x3", "ozaki4", "ozaki5"])
        naux = _log_uniform(rng, 84, 2000 if prec == "fp64" else 2600)
        nocc, nvirt = _window(rng, naux)
        return {"kind": kind, "precision": prec, "nocc": nocc, "nvirt": nvirt, "naux": naux,
                "nomega": rng.randint(12, 36), "qp_only": rng.random() < 0.5, "host": naux < 300}
    if kind == "batch":
        prec = rng.choice(["fp64", "bf16x3"])
        lo = rng.randint(3, 12)
        return {"kind": kind, "precision": prec, "count": rng.randint(3, 8 if prec == "fp64" else 16),
                "nocc_min": lo, "nocc_max": rng.randint(lo + 6, 28 if prec == "fp64" else 56),
                "sizes": rng.randint(0, 10 ** 6), "nomega": rng.choice([16, 24, 32])}
    if kind == "resident":
        naux = _log_uniform(rng, 84, 900)
        nocc, nvirt = _window(rng, naux)
        return {"kind": kind, "precision": rng.choice(["fp64", "fp64", "bf16x3"]), "nocc": nocc, "nvirt": nvirt,
                "naux": naux, "nomega": rng.randint(12, 32)}
    if kind == "aomo":
        nbf = _log_uniform(rng, 40, 400)
        return {"kind": kind, "precision": rng.choice(["fp64", "fp64", "bf16x3", "ozaki5"]), "nbf": nbf,
                "naux": int(nbf * rng.uniform(3.0, 4.0)), "nocc": max(2, nbf // rng.randint(8, 12))}
    if kind == "contour":
        naux = _log_uniform(rng, 100, 700)
        nocc, nvirt = _window(rng, naux)
        return {"kind": kind, "nocc": nocc, "nvirt": nvirt, "naux": naux, "nomega": rng.randint(8, 24)}
    naux = _log_uniform(rng, 100, 1600)
    nocc, nvirt = _window(rng, naux)
    return {"kind": "sox", "nocc": nocc, "nvirt": nvirt, "naux": naux}


def _members(case):
    """(nocc, nvirt, naux) of the molecules of a batch: Nvirt = Nocc U[8, 10], Naux = 4 (Nocc + Nvirt)."""
    r = random.Random(case["sizes"])
    out = []
    for _ in range(case["count"]):
        no = r.randint(case["nocc_min"], case["nocc_max"])
        nv = int(round(no * r.uniform(8.0, 10.0)))
        out.append((no, nv, 4 * (no + nv)))
    return out


# ---------------------------------------------------------------- inputs
def _molecule(nocc, nvirt, naux, seed):
    """Energies (numpy, Ha), M [nocc, nvirt, naux] and M_sigma [2, nstate, naux] on the GPU."""
    host = np.random.default_rng(seed)
    energy = np.concatenate([np.sort(host.uniform(-30.0, -8.0, nocc)), np.sort(host.uniform(0.5, 40.0, nvirt))]) / HA_EV
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    m = torch.randn((nocc, nvirt, naux), generator=gen, dtype=torch.float64, device="cuda")
    e = torch.from_numpy(energy).cuda()
    scale = torch.sqrt(4.0 / (e[nocc:][None, :] - e[:nocc][:, None]).reshape(-1, 1))
    rows = m.view(-1, naux)
    v = torch.ones((naux, 1), dtype=torch.float64, device="cuda") / math.sqrt(naux)
    for _ in range(30):                       # largest eigenvalue of sum_t (4/de_t) M_t M_t^T
        u = rows.T @ (scale * scale * (rows @ v))
        lam = torch.linalg.vector_norm(u)
        v = u / lam
    s = torch.sqrt(0.8 / lam)
    m.mul_(s)
    ms = torch.empty((2, nocc + nvirt, naux), dtype=torch.float64, device="cuda")
    ms[0, :nocc] = torch.randn((nocc, naux), generator=gen, dtype=torch.float64, device="cuda") * s
    ms[0, nocc:] = m[nocc - 1]
    ms[1, :nocc] = m[:, 0]
    ms[1, nocc:] = torch.randn((nvirt, naux), generator=gen, dtype=torch.float64, device="cuda") * s
    return energy, m, ms


def _ao(case, seed):
    """AO tensor [naux, npair] on the GPU, pair index, orbitals [nbf, nbf] (rows are states)."""
    nbf, naux = case["nbf"], case["naux"]
    low, high = np.tril_indices(nbf)          # pairs (k <= l), l outermost
    index = np.stack([high + 1, low + 1], axis=1).astype(np.int32)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    eri = torch.randn((naux, index.shape[0]), generator=gen, dtype=torch.float64, device="cuda") * 0.05
    c = np.linalg.qr(np.random.default_rng(seed).standard_normal((nbf, nbf)))[0]
    return eri, index, np.ascontiguousarray(c)


_ENGINE = []


def _engine():
    """The one context that a program keeps for all its solves."""
    if not _ENGINE:
        from molgw_b200.rigw import Engine
        _ENGINE.append(Engine(0))
    return _ENGINE[0]


def _instance(nocc, nvirt, naux, nomega, energy, m, ms):
    from molgw_b200.synth import GWInstance
    occ = np.concatenate([np.full(nocc, 2.0), np.zeros(nvirt)])
    return GWInstance(nocc=nocc, nvirt=nvirt, naux=naux, nomega=nomega, energy=energy, occupation=occ, m_ia=m,
                      m_sigma=ms, nsemin=nocc, nsemax=nocc + 1, nomega_sigma_calc=NC, step_sigma_calc=STEP_CALC,
                      nomega_sigma=NREAL, step_sigma=STEP_REAL, eta=ETA)


def _on_device(nocc, nvirt, naux, nomega, seed):
    energy, m, ms = _molecule(nocc, nvirt, naux, seed)
    inst = _instance(nocc, nvirt, naux, nomega, energy, None, None)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    occ = inst.occupation
    arrays = {"m_ia": m, "m_pm": ms, "e_occ": dev(energy[:nocc]), "e_virt": dev(energy[nocc:]),
              "occ_occ": dev(occ[:nocc]), "occ_virt": dev(occ[nocc:]), "e_p": dev(energy),
              "e_sig": dev(energy[nocc - 1:nocc + 1]), "occ_sig": dev(occ[nocc - 1:nocc + 1])}
    return inst, arrays


def prepare(case, seed):
    eng, kind = _engine(), case["kind"]
    st = {"case": case, "eng": eng}
    if kind == "batch":
        mols = [_on_device(no, nv, na, case["nomega"], seed * 1000 + k)
                for k, (no, nv, na) in enumerate(_members(case))]
        st["insts"], st["arrays"] = [x for x, _ in mols], [a for _, a in mols]
    elif kind == "aomo":
        st["eri"], st["index"], st["c"] = _ao(case, seed)
    elif kind == "resident" or (kind == "g0w0" and case["host"]):
        energy, m, ms = _molecule(case["nocc"], case["nvirt"], case["naux"], seed)
        st["inst"], st["arrays"] = _instance(case["nocc"], case["nvirt"], case["naux"], case["nomega"], energy,
                                             m.cpu().numpy(), ms.cpu().numpy()), None
    else:
        st["inst"], st["arrays"] = _on_device(case["nocc"], case["nvirt"], case["naux"], case.get("nomega", 1), seed)
    if kind == "sox":
        e, no = st["inst"].energy, case["nocc"]
        st["z"] = 0.5 * (e[no - 1] + e[no]) + 1j * STEP_CALC * np.arange(NC)
    return st


# ---------------------------------------------------------------- one pass
def _g0w0_outputs(case, out):
    d = {"erpa": out.erpa, "sigma_calc": out.sigma_calc, "energy_qp_g": out.energy_qp_g}
    if case["kind"] == "g0w0" and not case["qp_only"]:
        d["egw"] = out.egw
    if case["precision"] == "fp64":
        # Sigma on the real axis and what is read off it beyond the QP energy: the 99-point
        # continuation turns the rounding of the split precisions into other poles there
        d.update(sigma=out.sigma, energy_qp_z=out.energy_qp_z, zz=out.zz)
    return d


def run(state):
    case, eng = state["case"], state["eng"]
    kind = case["kind"]
    if kind == "g0w0":
        return _g0w0_outputs(case, eng.g0w0(state["inst"], PRECISION[case["precision"]],
                                            device_arrays=state["arrays"], qp_only=case["qp_only"]))
    if kind == "batch":
        outs = eng.g0w0_batch(state["insts"], PRECISION[case["precision"]], device_arrays=state["arrays"],
                              qp_only=True)
        return {"erpa": np.array([o.erpa for o in outs]), "sigma_calc": np.stack([o.sigma_calc for o in outs]),
                "energy_qp_g": np.stack([o.energy_qp_g for o in outs])}
    if kind == "resident":
        inst = state["inst"]
        erpa, egw, wpol = eng.polarizability_grid_scalapack(inst, PRECISION[case["precision"]])
        sigma = eng.gw_selfenergy_imag_scalapack(wpol, inst)
        wpol.release()
        return {"erpa": erpa, "egw": egw, "sigma_calc": sigma}
    if kind == "aomo":
        return eng.calculate_eri_3center_mo(state["eri"], state["index"], state["c"], case["nocc"] + 1, case["nbf"],
                                            1, case["nocc"], PRECISION[case["precision"]])
    inst, arrays = state["inst"], state["arrays"]
    if kind == "contour":
        out = eng.g0w0_contour(inst.energy, inst.occupation, arrays["m_ia"], arrays["m_pm"], inst.nsemin, inst.nsemax,
                               case["nomega"], CD_REAL, CD_SIGMA, CD_STEP, CD_ETA)
        return {"sigma": out.sigma, "rank": out.rank, "energy_qp_g": out.energy_qp_g, "energy_qp_z": out.energy_qp_z,
                "zz": out.zz, "omega_real": out.omega_real}
    return eng.sox_selfenergy_imag_grid(inst, state["z"], device_arrays={"m_ov": arrays["m_ia"],
                                                                         "m_pq": arrays["m_pm"]})


# ---------------------------------------------------------------- what a pass cannot do without
def _gw_work(nocc, nvirt, naux, nomega, qp_only):
    nia, cols = nocc * nvirt, 2 * (nocc + nvirt)
    chi0 = nomega * naux * (naux + 1.0) * nia                               # upper triangle of M D M^T
    factor = nomega * (naux ** 3 / 3.0 + float(naux) ** 2 * cols)           # Cholesky, U^-T M_sigma
    if not qp_only:
        factor += nomega * naux ** 3 / 3.0                                  # U^-T for tr eps^-1
    return {"bytes": 8.0 * (nia * naux + cols * naux + 2 * NC * 2 + NREAL * 4), "flops": chi0 + factor}


def work(case):
    kind = case["kind"]
    if kind == "g0w0":
        return _gw_work(case["nocc"], case["nvirt"], case["naux"], case["nomega"], case["qp_only"])
    if kind == "resident":
        return _gw_work(case["nocc"], case["nvirt"], case["naux"], case["nomega"], False)
    if kind == "batch":
        each = [_gw_work(no, nv, na, case["nomega"], True) for no, nv, na in _members(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "aomo":
        n, q, o = case["nbf"], case["naux"], case["nocc"]
        return {"bytes": 8.0 * (q * n * (n + 1) / 2 + n * n + q * o * (n - o)),
                "flops": 2.0 * q * o * n * n + 2.0 * q * o * (n - o) * n}
    no, nv, na = case["nocc"], case["nvirt"], case["naux"]
    nia, cols = no * nv, 2 * (no + nv)
    if kind == "contour":
        nw = case["nomega"] + CD_REAL
        # chi0, a symmetric eigenproblem with vectors (4/3 + 4/3 + 2 n^3), V^T M
        return {"bytes": 8.0 * (nia + cols) * na,
                "flops": nw * (na * (na + 1.0) * nia + 14.0 / 3.0 * na ** 3 + 2.0 * na * na * cols)}
    # (p q|j c), then about 8 operations per (product, evaluation point)
    terms = no * no * nv + no * nv * nv
    return {"bytes": 8.0 * (nia + cols) * na, "flops": 2.0 * cols * nia * na + 2.0 * terms * NC * 8}


# About four times what is seen when the auxiliary functions are taken in another order (every sum
# and the elimination order change, no result does).  FP64: Sigma_c 5e-16; E_RPA and E_GW 2e-11,
# because the weight of the highest frequency multiplies a difference of two sums of Naux terms;
# QP energies up to 3e-9, and Sigma on the real axis 3e-6, through the 99-point continuation.
# Split precisions: four times the distance from 64 bits (bf16x3: 8e-6, four slices: 3e-7), since
# the order of the sums is not what limits them.
def tolerance(case):
    kind, prec = case["kind"], case.get("precision", "fp64")
    if prec == "bf16x3":
        return {"rel": 4e-5, "max": 4e-4}
    if prec.startswith("ozaki"):
        rel = max(2e-8, 1.5e-6 * 128.0 ** (4 - int(prec[5:])))
        return {"rel": rel, "max": 10 * rel}
    return {"g0w0": {"rel": 2e-5, "max": 2e-4}, "batch": {"rel": 1e-8, "max": 1e-7},
            "resident": {"rel": 1e-10, "max": 1e-10}, "contour": {"rel": 1e-11, "max": 1e-10},
            "aomo": {"rel": 4e-15, "max": 4e-14}, "sox": {"rel": 4e-15, "max": 4e-14}}[kind]


# ---------------------------------------------------------------- the same in 64 bits, plain torch
def _imaginary_grid(n):
    x, w = np.polynomial.legendre.leggauss(n)
    x, w = 0.5 * (x + 1.0), 0.5 * w
    return 2.0 * x / (1.0 - x), 2.0 * w / (1.0 - x) ** 2


def _exact_gw(nocc, nvirt, naux, nomega, seed, qp_only):
    energy, m, ms = _molecule(nocc, nvirt, naux, seed)
    e = torch.from_numpy(energy).cuda()
    de = (e[nocc:][None, :] - e[:nocc][:, None]).reshape(-1, 1)
    rows, cols = m.view(-1, naux), ms.view(-1, naux).T.contiguous()
    omega, weight = _imaginary_grid(nomega)
    z = torch.from_numpy(0.5 * (energy[nocc - 1] + energy[nocc]) + 1j * STEP_CALC * np.arange(NC)).cuda()
    x = z[:, None] - e[None, :]
    norm = (cols * cols).sum(0)
    erpa = egw = 0.0
    sigma = torch.zeros((2, NC), dtype=torch.complex128, device="cuda")
    scaled = torch.empty_like(rows)
    eye = torch.eye(naux, dtype=torch.float64, device="cuda")
    for om, wt in zip(omega, weight):
        torch.mul(rows, 4.0 * de / (om * om + de * de), out=scaled)
        eps = eye + rows.T @ scaled
        low = torch.linalg.cholesky(eps)
        trace = eps.diagonal().sum()
        erpa += float((2.0 * low.diagonal().log().sum() + naux - trace).item()) * wt / (2 * math.pi)
        if not qp_only:
            inv = torch.linalg.solve_triangular(low, eye, upper=False)
            egw += float((2.0 * naux - (inv * inv).sum() - trace).item()) * wt / (2 * math.pi)
        y = torch.linalg.solve_triangular(low, cols, upper=False)
        v = ((y * y).sum(0) - norm).view(2, -1).to(torch.complex128)
        f = 1.0 / (x + 1j * om) + 1.0 / (x - 1j * om)
        sigma -= wt / (2 * math.pi) * (v @ f.T)
    out = {"erpa": erpa, "sigma_calc": sigma.cpu().numpy()}
    if not qp_only:
        out["egw"] = egw
    return out


def _exact_contour(case, seed):
    no, nv, na, nw = case["nocc"], case["nvirt"], case["naux"], case["nomega"]
    energy, m, ms = _molecule(no, nv, na, seed)
    e = torch.from_numpy(energy).cuda()
    de = (e[no:][None, :] - e[:no][:, None]).reshape(-1, 1)
    rows = m.view(-1, na)
    half = CD_SIGMA // 2
    grid = CD_STEP * np.arange(-half, half + 1)
    e0 = energy[no - 1:no + 1]
    # distance of every pole that is passed: occupied above, empty below the evaluation point
    occ_de = energy[:no][None, None, :] - (e0[:, None, None] + grid[None, :, None])
    emp_de = e0[:, None, None] + grid[None, :, None] - energy[no:][None, None, :]
    top = max([0.0] + [d.max() for d in (occ_de[occ_de >= -CD_ETA], emp_de[emp_de >= -CD_ETA]) if d.size])
    real = top * np.arange(CD_REAL) / (CD_REAL - 1.0)
    omega, weight = _imaginary_grid(nw)
    freqs = [(-om * om) for om in omega] + [om * om for om in real]
    v, rank = [], []
    for w2 in freqs:                                       # g = lambda / (1 - lambda), small ones dropped
        chi0 = rows.T @ (rows * (4.0 * de / (w2 - de * de)))
        lam, vec = torch.linalg.eigh(chi0)
        g = lam / (1.0 - lam)
        keep = g.abs() > 1e-3
        rank.append(int(keep.sum().item()))
        zt = vec[:, keep].T @ ms.view(-1, na).T
        v.append(((zt * zt) * g[keep][:, None]).sum(0).view(2, -1).cpu().numpy())
    sigma = np.zeros((grid.size, 2), dtype=complex)
    for s in range(2):
        x = e0[s] + grid[:, None] - energy[None, :]
        live = np.abs(x) > CD_ETA
        for k in range(nw):
            term = 2.0 * x / (x * x + omega[k] ** 2) * v[k][s][None, :] / (2 * math.pi)
            sigma[:, s] -= weight[k] * np.where(live, term, 0.0).sum(1)
        for sign, d, first in ((-1.0, occ_de[s], 0), (1.0, emp_de[s], no)):
            for io, p in zip(*np.nonzero(d >= -CD_ETA)):
                near = int(np.argmin(np.abs(real - abs(d[io, p]))))
                sigma[io, s] += sign * v[nw + near][s][first + p] * (0.5 if abs(d[io, p]) < CD_ETA else 1.0)
    return {"sigma": sigma, "omega_real": real}


def _exact_sox(case, seed):
    no, nv, na = case["nocc"], case["nvirt"], case["naux"]
    energy, m, ms = _molecule(no, nv, na, seed)
    e = torch.from_numpy(energy).cuda()
    eo, ev = e[:no], e[no:]
    z = torch.from_numpy(0.5 * (energy[no - 1] + energy[no]) + 1j * STEP_CALC * np.arange(NC)).cuda()
    rows = m.view(-1, na)
    d1 = eo[:, None, None] + eo[None, :, None] - ev[None, None, :]
    d2 = ev[:, None, None] + ev[None, None, :] - eo[None, :, None]
    out = torch.zeros((2, NC), dtype=torch.complex128, device="cuda")
    for p in range(2):
        c = (ms[p] @ rows.T).view(no + nv, no, nv)
        w1 = c[:no] * c[:no].transpose(0, 1)
        w2 = c[no:] * c[no:].permute(2, 1, 0)
        for k in range(NC):
            out[p, k] = -(w1 / (z[k] - d1)).sum() - (w2 / (z[k] - d2)).sum()
    return out.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("g0w0", "resident"):
        return _exact_gw(case["nocc"], case["nvirt"], case["naux"], case["nomega"], seed,
                         case.get("qp_only", False))
    if kind == "batch":
        each = [_exact_gw(no, nv, na, case["nomega"], seed * 1000 + k, True)
                for k, (no, nv, na) in enumerate(_members(case))]
        return {"erpa": np.array([x["erpa"] for x in each]), "sigma_calc": np.stack([x["sigma_calc"] for x in each]),
                "energy_qp_g": None}
    if kind == "aomo":
        eri, index, c = _ao(case, seed)
        n, no = case["nbf"], case["nocc"]
        i, j = (torch.from_numpy(index[:, k].astype(np.int64) - 1).cuda() for k in (0, 1))
        ct = torch.from_numpy(c).cuda()
        out = torch.empty((no, n - no, case["naux"]), dtype=torch.float64, device="cuda")
        for q in range(case["naux"]):
            full = torch.zeros((n, n), dtype=torch.float64, device="cuda")
            full[i, j] = eri[q]                            # diagonal pairs are stored halved
            full = full + full.T
            out[:, :, q] = ct[:no] @ full @ ct[no:].T
        return out
    if kind == "contour":
        return _exact_contour(case, seed)
    return _exact_sox(case, seed)
