"""Performance cases: the work users of this library have it do, through its public entry points.

A case is a dict of plain values whose "kind" names the call:

  sigma   B200Backend.sigma_c on a resident system (real form at eta = 0, complex form otherwise)
  whole   run_g0w0 on a system in host memory: upload, grid, screening, contraction, Pade, QP
  matrix  B200Backend.sigma_c_matrix: Sigma_c between the requested states
  batch   run_g0w0_batch: molecules of uneven size in shared launches
  serve   B200Server: a burst of requests of uneven size, submitted and waited for
  post    B200Backend.qp for every state and B200Backend.pade_sweep (QP table and E_c.out)

Inputs follow the recipe of minigw_b200/synthetic.py (random symmetric factors L, V = L^T L, the
orbital energies and their gap), drawn on the GPU from the seed.  Calls that also return QP energies
are represented by their self-energies: the QP energies are a function of Sigma_c alone, which the
Pade continuation of these random systems amplifies by many orders of magnitude, and "post" covers
that function on inputs of its own.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from minigw_b200 import (B200Backend, B200Server, GwInput, GwSettings, GwSlices, generate_transformed_legendre_grid,
                         run_g0w0, run_g0w0_batch)


# ---------------------------------------------------------------------------------------------
# The cases

def _molecule_sizes(count: int, lo: int, hi: int) -> list[int]:
    """`count` orbital counts spread evenly over [lo, hi]."""
    return [lo + round((hi - lo) * t / max(1, count - 1)) for t in range(count)]


def listed() -> list[dict]:
    return [
        # smallest request of a screening service: 16 orbitals, 32 frequencies, the HOMO alone
        {"name": "sigma_small_16", "kind": "sigma", "nmo": 16, "nocc": 3, "nfreq": 32, "below": 0, "above": -1,
         "precision": "fp64", "eta": 0.0},
        # one small molecule, H2O-shaped: 24 orbitals, the CLI's default 200 frequencies, the HOMO
        {"name": "sigma_h2o_24", "kind": "sigma", "nmo": 24, "nocc": 5, "nfreq": 200, "below": 0, "above": -1,
         "precision": "fp64", "eta": 0.0},
        # a medium molecule at odd sizes (737 pairs), HOMO and LUMO
        {"name": "sigma_medium_78", "kind": "sigma", "nmo": 78, "nocc": 11, "nfreq": 64, "below": 0, "above": 0,
         "precision": "fp64", "eta": 0.0},
        # a large molecule in the mixed form: 2000 pairs, six states around the gap
        {"name": "sigma_mixed_120", "kind": "sigma", "nmo": 120, "nocc": 20, "nfreq": 64, "below": 2, "above": 2,
         "precision": "mixed", "eta": 0.0},
        # the same molecule in the mixed form refined to FP64 accuracy
        {"name": "sigma_refined_120", "kind": "sigma", "nmo": 120, "nocc": 20, "nfreq": 64, "below": 2, "above": 2,
         "precision": "mixed-refined", "eta": 0.0},
        # the largest solve: 5100 pairs, 128 frequencies, ten states
        {"name": "sigma_large_200", "kind": "sigma", "nmo": 200, "nocc": 30, "nfreq": 128, "below": 4, "above": 4,
         "precision": "fp64", "eta": 0.0},
        # with broadening (--eta): the complex form
        {"name": "sigma_eta_60", "kind": "sigma", "nmo": 60, "nocc": 10, "nfreq": 48, "below": 1, "above": 1,
         "precision": "fp64", "eta": 0.01},
        # a molecule as the program reads it, every step of the solve: the full ERI in host memory
        {"name": "whole_48", "kind": "whole", "nmo": 48, "nocc": 8, "nfreq": 100, "below": 1, "above": 1,
         "precision": "fp64"},
        # the off-diagonal self-energy of eight states
        {"name": "matrix_90", "kind": "matrix", "nmo": 90, "nocc": 15, "nfreq": 48, "below": 3, "above": 3},
        # a screening campaign: molecules of 20 to 120 orbitals in one call, FP64-accurate
        {"name": "batch_16", "kind": "batch", "count": 16, "lo": 20, "hi": 120, "nfreq": 64, "npade": 12,
         "precision": "mixed-refined"},
        # a burst of requests of a serving loop: 12 requests, 16 to 96 orbitals, 4 slots
        {"name": "serve_12", "kind": "serve", "count": 12, "lo": 16, "hi": 96, "nfreq": 64, "npade": 12, "slots": 4,
         "precision": "fp64"},
        # the tables after a solve: QP energies of all states, the E_c.out sweep of the HOMO
        {"name": "post_60", "kind": "post", "nmo": 60, "nocc": 10, "nfreq": 100, "npade": 16, "npts": 19836},
    ]


def draw(rng) -> dict:
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def window(nocc, nvir, most):
        """A contiguous state window around the gap of 1 to `most` states."""
        count = rng.randint(1, most)
        below = min(count // 2, nocc - 1)
        return below, min(count - below - 2, nvir - 1)

    kind = rng.choice(["sigma", "sigma", "sigma", "refined", "mixed", "eta", "whole", "matrix", "batch", "serve",
                       "post"])
    if kind in ("sigma", "refined", "mixed"):
        nmo = log_int(16, 150) if kind == "sigma" else log_int(60, 140)
        nocc = max(2, round(nmo / 6) + rng.randint(-1, 1))
        below, above = window(nocc, nmo - nocc, 8)
        return {"kind": "sigma", "nmo": nmo, "nocc": nocc, "nfreq": rng.randint(32, 128), "below": below,
                "above": above, "precision": {"sigma": "fp64", "refined": "mixed-refined"}.get(kind, "mixed"),
                "eta": 0.0}
    if kind in ("eta", "whole"):
        nmo = log_int(16, 72)
        nocc = max(2, round(nmo / 6))
        below, above = window(nocc, nmo - nocc, 6)
        c = {"kind": "sigma" if kind == "eta" else "whole", "nmo": nmo, "nocc": nocc, "nfreq": rng.randint(32, 128),
             "below": below, "above": above, "precision": "fp64"}
        if kind == "eta":
            c["eta"] = rng.choice([0.001, 0.01, 0.05])
        return c
    if kind == "matrix":
        nmo = log_int(24, 110)
        nocc = max(2, round(nmo / 6))
        below, above = window(nocc, nmo - nocc, 12)
        return {"kind": "matrix", "nmo": nmo, "nocc": nocc, "nfreq": rng.randint(32, 64), "below": below,
                "above": above}
    if kind in ("batch", "serve"):
        c = {"kind": kind, "count": rng.randint(4, 16), "lo": rng.randint(16, 32), "hi": log_int(48, 120),
             "nfreq": rng.randint(32, 96), "npade": 12,
             "precision": rng.choice(["mixed-refined", "mixed"] if kind == "batch" else ["fp64", "mixed-refined"])}
        if kind == "serve":
            c["hi"] = min(c["hi"], 96)
            c["slots"] = rng.randint(2, 4)
        return c
    nmo = log_int(16, 200)
    return {"kind": "post", "nmo": nmo, "nocc": max(2, round(nmo / 6)), "nfreq": rng.randint(32, 200),
            "npade": rng.choice([8, 12, 16, 24, 32]), "npts": log_int(2000, 40000)}


# ---------------------------------------------------------------------------------------------
# Inputs

def _states(case: dict) -> list[int]:
    """HOMO - below .. LUMO + above (0-based; above = -1: up to the HOMO)."""
    return list(range(case["nocc"] - 1 - case["below"], case["nocc"] + case["above"] + 1))


def _orbitals(nmo: int, nocc: int, gen) -> tuple[np.ndarray, float]:
    u = torch.rand(nmo, generator=gen, device="cuda", dtype=torch.float64).cpu().numpy()
    mo = np.concatenate([np.sort(-1.2 + 0.9 * u[:nocc]), np.sort(0.05 + 2.95 * u[nocc:])])
    return mo, float(0.5 * (mo[nocc - 1] + mo[nocc]))


def _factors(nmo: int, gen) -> torch.Tensor:
    """L[K, p, q] ~ N(0, 1) 0.3 exp(-|p - q| / 8), symmetric in (p, q), K < 2 nmo."""
    g = torch.randn((2 * nmo, nmo, nmo), generator=gen, device="cuda", dtype=torch.float64)
    idx = torch.arange(nmo, device="cuda", dtype=torch.float64)
    decay = 0.3 * torch.exp(-(idx[:, None] - idx[None, :]).abs() / 8.0)
    return (torch.triu(g) + torch.triu(g, 1).transpose(1, 2)) * decay


def _vxc(nmo: int, gen) -> np.ndarray:
    off = torch.randn((nmo, nmo), generator=gen, device="cuda", dtype=torch.float64) * 0.01
    diag = -0.6 + 0.4 * torch.rand(nmo, generator=gen, device="cuda", dtype=torch.float64)
    off = torch.triu(off, 1)
    return (off + off.t() + torch.diag(diag)).cpu().numpy()


def _device_system(nmo: int, nocc: int, states: list[int], seed: int) -> dict:
    """V_ph, the states' panel rows and the diagonals, as GPU tensors."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    mo, fermi = _orbitals(nmo, nocc, gen)
    fac = _factors(nmo, gen)
    lov = fac[:, :nocc, nocc:].reshape(2 * nmo, -1)
    v = lov.t() @ lov
    return {"mo": mo, "fermi": fermi, "nocc": nocc, "states": states, "v": 0.5 * (v + v.t()),
            "panel": torch.cat([fac[:, p, :].t() @ lov for p in states], dim=0),
            "xdiag": (fac[:, :, :nocc] ** 2).sum(dim=0), "vxc": _vxc(nmo, gen)}


def _slices(nmo: int, nocc: int, states: list[int], seed: int) -> GwSlices:
    d = _device_system(nmo, nocc, states, seed)
    return GwSlices(mo_energy=d["mo"], nocc=nocc, fermi_energy=d["fermi"], states=np.array(states, dtype=np.int64),
                    vph=d["v"].cpu().numpy(), panel=d["panel"].cpu().numpy(), xdiag=d["xdiag"].cpu().numpy(),
                    vxc_diag=np.ascontiguousarray(np.diag(d["vxc"])))


def _input(nmo: int, nocc: int, seed: int) -> GwInput:
    """The whole system with its nmo^4 ERI tensor in host memory."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    mo, fermi = _orbitals(nmo, nocc, gen)
    lmat = _factors(nmo, gen).reshape(2 * nmo, nmo * nmo)
    eri = lmat.t() @ lmat
    eri = (0.5 * (eri + eri.t())).cpu().numpy().reshape(nmo, nmo, nmo, nmo)
    return GwInput(eri_mo=eri, mo_energy=mo, vxc_mo=_vxc(nmo, gen), nocc=nocc, fermi_energy=fermi)


def _molecules(case: dict) -> list[dict]:
    """Batch and serve: nocc = round(nmo / 6), HOMO and LUMO."""
    out = []
    for nmo in _molecule_sizes(case["count"], case["lo"], case["hi"]):
        nocc = max(2, round(nmo / 6))
        out.append({"nmo": nmo, "nocc": nocc, "states": [nocc - 1, nocc]})
    return out


def _model_sigma(nmo: int, nocc: int, nfreq: int, seed: int):
    """Sigma_c(iw) of every state from screened forms that fall off smoothly with frequency, as solves
    give them."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    mo, fermi = _orbitals(nmo, nocc, gen)
    om, w = _grid(nfreq)
    amp = 0.02 * torch.rand((nmo, nmo), generator=gen, device="cuda", dtype=torch.float64)
    width = 0.5 + 2.0 * torch.rand((nmo, nmo), generator=gen, device="cuda", dtype=torch.float64)
    wf = torch.from_numpy(om).cuda()
    q = -amp[None] * width[None] ** 2 / (wf[:, None, None] ** 2 + width[None] ** 2)
    return mo, fermi, om, w, _contract(q, mo, fermi, om, w).cpu().numpy(), _vxc(nmo, gen), gen


class _Server:
    """A server that is shut down when its state goes."""

    def __init__(self, slots: int):
        self.server = B200Server(0, slots, 6 << 30)

    def __del__(self):
        try:
            self.server.close()
        except Exception:
            pass


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"case": case}
    if kind in ("sigma", "matrix"):
        st["states"] = _states(case)
        st["om"], st["w"] = generate_transformed_legendre_grid(case["nfreq"])
        st["be"] = B200Backend(0)
        st["be"].load_slices(_slices(case["nmo"], case["nocc"], st["states"], seed))
    elif kind == "whole":
        st["inp"] = _input(case["nmo"], case["nocc"], seed)
        st["settings"] = GwSettings(num_freq_points_total=case["nfreq"], num_pade_params=16, eta=0.0,
                                    states=_states(case), precision=case["precision"])
        st["be"] = B200Backend(0)
    elif kind == "batch":
        st["mols"] = _molecules(case)
        st["be"] = []
        for i, m in enumerate(st["mols"]):
            b = B200Backend(0)
            b.load_slices(_slices(m["nmo"], m["nocc"], m["states"], 1000 * seed + i))
            st["be"].append(b)
    elif kind == "serve":
        st["mols"] = _molecules(case)
        st["inputs"] = [_slices(m["nmo"], m["nocc"], m["states"], 1000 * seed + i) for i, m in enumerate(st["mols"])]
        st["server"] = _Server(case["slots"])
    elif kind == "post":
        nmo, nocc = case["nmo"], case["nocc"]
        mo, fermi, st["om"], _, st["sigma"], vxc, gen = _model_sigma(nmo, nocc, case["nfreq"], seed)
        n = nocc * (nmo - nocc)
        xdiag = 0.1 * torch.rand((nmo, nocc), generator=gen, device="cuda", dtype=torch.float64).cpu().numpy()
        st["be"] = B200Backend(0)
        # the QP step needs the orbital energies and the exchange and vxc diagonals of the loaded system
        st["be"].load_slices(GwSlices(mo_energy=mo, nocc=nocc, fermi_energy=fermi, states=np.array([nocc - 1]),
                                      vph=np.zeros((n, n)), panel=np.zeros((nmo, n)), xdiag=xdiag,
                                      vxc_diag=np.ascontiguousarray(np.diag(vxc))))
    else:
        raise ValueError(kind)
    return st


# ---------------------------------------------------------------------------------------------
# One pass

def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "sigma":
        return st["be"].sigma_c(st["om"], st["w"], st["states"], case["eta"], case["precision"])[0]
    if kind == "matrix":
        return st["be"].sigma_c_matrix(st["om"], st["w"], st["states"])[0]
    if kind == "whole":
        r = run_g0w0(st["inp"], st["settings"], st["be"])
        return {"sigma": r.sigma_c_im_points, "sigma_x": r.sigma_x_diag, "omegas": r.omegas, "weights": r.weights}
    if kind == "batch":
        return run_g0w0_batch(st["be"], case["nfreq"], case["npade"], [m["states"] for m in st["mols"]],
                              case["precision"])["sigma"]
    if kind == "serve":
        server = st["server"].server
        tickets = [server.submit(inp, case["nfreq"], case["npade"], m["states"], precision=case["precision"])
                   for inp, m in zip(st["inputs"], st["mols"])]
        done = [server.wait(t) for t in tickets]
        return [{"sigma": d["sigma"], "sigma_x": d["sigma_x_diag"]} for d in done]
    qp = st["be"].qp(st["om"], st["sigma"], case["npade"], list(range(case["nmo"])))
    sweep = st["be"].pade_sweep(st["om"], st["sigma"][case["nocc"] - 1], case["npade"], case["npts"])
    return {"qp": qp, "sweep": sweep}


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without

def _solve_work(nmo: int, nocc: int, nstates: int, nfreq: int, form: float = 1.0) -> tuple[float, float]:
    n, m = float(nocc * (nmo - nocc)), float(nstates * nmo)
    flops = form * nfreq * (n ** 3 / 3.0 + n * n * m + 3.0 * n * m) + 10.0 * nfreq * nfreq * m
    return 8.0 * (n * n + n * m) + 16.0 * nmo * nfreq, flops


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("sigma", "matrix", "whole"):
        ns = len(_states(case))
        # a complex multiply-add is four real ones
        b, f = _solve_work(case["nmo"], case["nocc"], ns, case["nfreq"], 4.0 if case.get("eta") else 1.0)
        if kind == "matrix":
            n = case["nocc"] * (case["nmo"] - case["nocc"])
            f += case["nfreq"] * case["nmo"] * ns * (ns + 1.0) * n
        if kind == "whole":  # the (pq|o.) part of the ERI is read from host memory
            b = 8.0 * case["nmo"] ** 3 * case["nocc"] + 16.0 * case["nmo"] * case["nfreq"]
        return {"bytes": b, "flops": f}
    if kind in ("batch", "serve"):
        parts = [_solve_work(m["nmo"], m["nocc"], 2, case["nfreq"]) for m in _molecules(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    # complex recurrences: the coefficients of every state, about ten QP steps a state, the sweep
    points = case["nmo"] * (case["npade"] + 10.0) + case["npts"]
    return {"bytes": 16.0 * case["nmo"] * case["nfreq"] + 24.0 * case["npts"], "flops": 25.0 * case["npade"] * points}


# ---------------------------------------------------------------------------------------------
# The same values from plain torch in 64 bits

def _grid(nfreq: int) -> tuple[np.ndarray, np.ndarray]:
    """Gauss-Legendre nodes y on (-1, 1) mapped to w = (1 + y) / (2 (1 - y))."""
    y, wy = np.polynomial.legendre.leggauss(nfreq)
    return 0.5 * (1.0 + y) / (1.0 - y), wy / (1.0 - y) ** 2


def _contract(q: torch.Tensor, mo, fermi: float, om, w) -> torch.Tensor:
    """Sigma[s, n] = -(1/pi) sum_{f, k} w_f a / (a^2 + w_f^2) q[f, s, k], a = i w_n + E_F - e_k."""
    e = torch.from_numpy(np.ascontiguousarray(mo)).cuda()
    omt, wt = torch.from_numpy(om).cuda(), torch.from_numpy(w).cuda()
    out = torch.empty((q.shape[1], omt.shape[0]), dtype=torch.complex128, device="cuda")
    qc = (q * wt[:, None, None]).to(torch.complex128)
    for n in range(omt.shape[0]):
        a = torch.complex(fermi - e, torch.full_like(e, float(om[n])))
        g = a[None, :] / (a[None, :] ** 2 + omt[:, None] ** 2)  # [f, k]
        out[:, n] = -torch.einsum("fk,fsk->s", g, qc) / math.pi
    return out


def _forms(v: torch.Tensor, panel: torch.Tensor, mo, nocc: int, nstates: int, om, eta: float = 0.0,
           cross: bool = False) -> torch.Tensor:
    """q[f, s, k] = x_sk^T W_c(i w_f) x_sk, or q[f, s * ns + t, k] between the states."""
    nmo = len(mo)
    e = torch.from_numpy(np.ascontiguousarray(mo)).cuda()
    delta = (e[None, nocc:] - e[:nocc, None]).reshape(-1)
    n = delta.shape[0]
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    out = []
    for w in om:
        if eta == 0.0:
            d = torch.sqrt(4.0 * delta / (float(w) ** 2 + delta ** 2))
            y = torch.linalg.solve_triangular(torch.linalg.cholesky(d[:, None] * v * d[None, :] + eye),
                                              (panel * d[None, :]).t().contiguous(), upper=False)
            if cross:
                y3 = y.reshape(n, nstates, nmo)
                out.append(-torch.einsum("nsk,ntk->stk", y3, y3).reshape(nstates * nstates, nmo))
            else:
                out.append(-(y * y).sum(dim=0).reshape(nstates, nmo))
        else:
            z = complex(0.0, float(w))
            p = 2.0 * (1.0 / (z - delta + 1j * eta) - 1.0 / (z + delta - 1j * eta))
            x = panel.to(torch.complex128)
            y = torch.linalg.solve(eye - p[:, None] * v, p[:, None] * x.t())
            out.append((x.t() * y).sum(dim=0).reshape(nstates, nmo))
    return torch.stack(out)


def _exact_rows(nmo, nocc, states, nfreq, seed, eta=0.0, cross=False):
    d = _device_system(nmo, nocc, states, seed)
    om, w = _grid(nfreq)
    q = _forms(d["v"], d["panel"], d["mo"], nocc, len(states), om, eta, cross)
    return _contract(q, d["mo"], d["fermi"], om, w), d


def _exact_sigma(nmo, nocc, states, nfreq, seed, eta=0.0):
    rows, d = _exact_rows(nmo, nocc, states, nfreq, seed, eta)
    out = torch.zeros((nmo, nfreq), dtype=torch.complex128, device="cuda")
    out[torch.tensor(states, device="cuda")] = rows
    return out.cpu().numpy(), d


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "sigma":
        return _exact_sigma(case["nmo"], case["nocc"], _states(case), case["nfreq"], seed, case["eta"])[0]
    if kind == "matrix":
        ns = len(_states(case))
        rows, _ = _exact_rows(case["nmo"], case["nocc"], _states(case), case["nfreq"], seed, cross=True)
        return rows.reshape(ns, ns, case["nfreq"]).cpu().numpy()
    if kind == "whole":
        nmo, nocc, states = case["nmo"], case["nocc"], _states(case)
        inp = _input(nmo, nocc, seed)
        eri = torch.from_numpy(inp.eri_mo).cuda()
        n = nocc * (nmo - nocc)
        v = eri[:nocc, nocc:, :nocc, nocc:].reshape(n, n)
        panel = eri[states][:, :, :nocc, nocc:].reshape(len(states) * nmo, n)
        om, w = _grid(case["nfreq"])
        sigma = torch.zeros((nmo, case["nfreq"]), dtype=torch.complex128, device="cuda")
        sigma[torch.tensor(states, device="cuda")] = _contract(_forms(v, panel, inp.mo_energy, nocc, len(states), om),
                                                               inp.mo_energy, inp.fermi_energy, om, w)
        sx = -torch.einsum("pipi->p", eri[:, :nocc, :, :nocc])
        return {"sigma": sigma.cpu().numpy(), "sigma_x": sx.cpu().numpy(), "omegas": None, "weights": None}
    if kind in ("batch", "serve"):
        out = []
        for i, m in enumerate(_molecules(case)):
            s, d = _exact_sigma(m["nmo"], m["nocc"], m["states"], case["nfreq"], 1000 * seed + i)
            out.append(s if kind == "batch" else {"sigma": s, "sigma_x": (-d["xdiag"].sum(dim=1)).cpu().numpy()})
        return out
    return None  # the tables of "post" are the reference's arithmetic bit for bit, not a converged value
