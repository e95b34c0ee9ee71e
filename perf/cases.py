"""The calls a user of the phonon library makes, as cases that can be timed.

Every case is one call (or one forward and backward pass) of a public entry
point on a twisted-bilayer cell of the synthetic spring model: the plain FP64
form and the mixed form, host and device entry points, frequencies alone,
group velocities, eigenvectors, an index range, cells of uneven size, the
gradient of a fit, a caller's own matrix, and the density of states.

A case is a plain dict; `kind` names the entry point:

  solve   PhononContext.solve            (host arrays in and out)
  device  PhononContext.solve_device     (device tensors in and out)
  multi   solve_multi                    (cells of different size)
  fit     PhononSpectrum.frequencies and its backward pass
  values  heevx_values_noalloc           (eigenvalues of a caller's matrix)
  dos     linear_triangulation_device    (density of states of a q-grid)

Cells are the commensurate cells of twist index m, N = 4 (3 m^2 + 3 m + 1)
atoms: m = 1, 3, 5, 8, 11 give N = 28, 148, 364, 868, 1588.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from parphom_gb300 import api, autograd, dos, geometry, synth

PI_F = float(np.float32(3.141592653589793))   # the reference's single-precision literals
C1 = float(np.float32(15.633302))
C2 = float(np.float32(33.35641))
C1SQ = float(np.float32(np.float32(15.633302) * np.float32(15.633302)))
TIE = float(np.float32(1e-10))


def listed():
    return [
        # one q-point of the smallest commensurate cell: the shortest call, all latency
        {"name": "point_28_fp64", "kind": "solve", "m": 1, "nq": 1, "mixed": False, "vel": True, "vectors": False,
         "il": 0, "iu": 0},
        # a band structure without velocities: 64 q-points of the 9.43 degree cell, plain FP64 form
        {"name": "bands_148_fp64", "kind": "solve", "m": 3, "nq": 64, "mixed": False, "vel": False,
         "vectors": False, "il": 0, "iu": 0},
        # frequencies and group velocities of the 6.01 degree cell kept on the device
        {"name": "path_364_mixed", "kind": "device", "m": 5, "nq": 16, "mixed": True, "vel": True,
         "vectors": False},
        # all eigenvectors and velocities in the plain FP64 form
        {"name": "vectors_364_fp64", "kind": "device", "m": 5, "nq": 4, "mixed": False, "vel": True,
         "vectors": True},
        # all eigenvectors and velocities of the 3.89 degree cell, mixed form
        {"name": "vectors_868_mixed", "kind": "device", "m": 8, "nq": 4, "mixed": True, "vel": True,
         "vectors": True},
        # the lowest 256 modes with eigenvectors and velocities in host memory (what the driver writes to its file)
        {"name": "lowest_868_mixed", "kind": "solve", "m": 8, "nq": 3, "mixed": True, "vel": True, "vectors": True,
         "il": 1, "iu": 256},
        # the plain FP64 form of a large cell, frequencies and velocities
        {"name": "path_868_fp64", "kind": "device", "m": 8, "nq": 2, "mixed": False, "vel": True,
         "vectors": False},
        # the headline workload: frequencies and velocities of the 2.88 degree cell, mixed form
        {"name": "path_1588_mixed", "kind": "device", "m": 11, "nq": 8, "mixed": True, "vel": True,
         "vectors": False},
        # q-points of three twist angles solved in shared batches
        {"name": "uneven_mixed", "kind": "multi", "m0": 3, "m1": 5, "m2": 8, "nq": 24, "mixed": True, "vel": True},
        # one step of fitting force constants to target frequencies: forward and backward
        {"name": "fit_364_mixed", "kind": "fit", "m": 5, "nq": 4, "mixed": True},
        # eigenvalues of a caller's own Hermitian matrix, no allocation
        {"name": "values_1092", "kind": "values", "m": 5, "lowest": 0},
        # density of states of a 32 x 32 q-grid of the 9.43 degree cell
        {"name": "dos_148", "kind": "dos", "grid": 32, "bands": 444, "energies": 1000, "weighted": False},
    ]


def _order(m):
    return 12 * (3 * m * m + 3 * m + 1)


def _cost(n, nq, mixed, vectors):
    """Cost of a solve in units of one mixed-form order^3."""
    return nq * float(n) ** 3 * (1.0 if mixed else 5.0) * (1.5 if vectors else 1.0)


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = _cost(_order(11), 7, True, False)

    def batch(n, mixed, vectors, cap=64):
        top = int(most / _cost(n, 1, mixed, vectors))
        return logint(1, max(1, min(cap, top)))

    kind = rng.choice(["solve", "solve", "device", "device", "device", "multi", "fit", "values", "dos"])
    mixed = rng.random() < 0.6
    if kind in ("solve", "device"):
        m = logint(1, 11)
        vel = rng.random() < 0.7
        vectors = rng.random() < 0.35 and m <= 8
        case = {"kind": kind, "m": m, "mixed": mixed, "vel": vel, "vectors": vectors}
        if kind == "solve":
            lo = 1 + rng.randrange(0, 40)
            some = vectors or rng.random() < 0.3
            case["il"], case["iu"] = (lo, min(_order(m), lo + logint(4, 300))) if some else (0, 0)
        # host eigenvectors of a whole spectrum are not among the listed ranges
        case["nq"] = batch(_order(m), mixed, vectors, 64 if not vectors else 12)
        return case
    if kind == "multi":
        a, b, c = (logint(1, 8) for _ in range(3))
        top = max(a, b, c)
        return {"kind": kind, "m0": a, "m1": b, "m2": c, "nq": 1 + batch(_order(top), mixed, False, 30),
                "mixed": mixed, "vel": rng.random() < 0.8}
    if kind == "fit":
        m = logint(1, 6)
        return {"kind": kind, "m": m, "nq": logint(1, 8), "mixed": mixed}
    if kind == "values":
        return {"kind": kind, "m": logint(1, 5), "lowest": rng.choice([0, 0, logint(3, 80)])}
    return {"kind": kind, "grid": rng.randrange(8, 33), "bands": logint(84, 600), "energies": logint(100, 1000),
            "weighted": rng.random() < 0.4}


# ---------------------------------------------------------------------------
# inputs
@functools.lru_cache(maxsize=None)
def _cell(m):
    """A cell and its force constants (the same for every seed, as for a user who varies the q-points)."""
    cell = synth.tblg_cell(m)
    return cell, synth.spring_force_constants(cell, seed=0)


def _qpoints(nq, seed):
    """q-points along a band path, each moved off its symmetry lines, so that modes cross nowhere exactly and single
    modes, their vectors and their velocities are determined."""
    rng = np.random.default_rng(1000 + seed)
    s = np.sort(rng.random(nq))
    path = synth.band_path(257)
    q = np.stack([np.interp(0.02 + 0.96 * s, np.linspace(0, 1, 257), path[:, k]) for k in range(3)], axis=1)
    q[:, :2] += rng.uniform(0.03, 0.08, (nq, 2))
    return q


def _reference(n, seed):
    """The vector that fixes the free phase of every eigenvector (a program that follows modes over q does this)."""
    rng = np.random.default_rng(5000 + seed)
    return rng.standard_normal(n) + 1j * rng.standard_normal(n)


def _prec(case):
    return api.PP_PREC_MIXED if case["mixed"] else api.PP_PREC_FP64


def _bands(case, seed):
    """Model bands over a uniform q-grid, their weights, triangles and energies."""
    rng = np.random.default_rng(9000 + seed)
    grid, nb = case["grid"], case["bands"]
    q = synth.uniform_grid(grid)
    base = np.sort(rng.uniform(5.0, 1600.0, nb))
    hop = rng.integers(-2, 3, (nb, 2))
    amp, phase = rng.uniform(2.0, 60.0, nb), rng.uniform(0, 2 * np.pi, nb)
    freq = base + amp * np.cos(2 * np.pi * (q[:, :2] @ hop.T) + phase) * np.minimum(1.0, base / 100.0)
    freq = np.sort(freq + rng.uniform(0, 0.3, freq.shape), axis=1)
    energy = np.linspace(-10.0, 1700.0, case["energies"])
    weight = rng.uniform(0.1, 3.0, freq.shape) if case["weighted"] else None
    rec = geometry.reciprocal_lattice(synth.tblg_cell(3).lat)
    return freq, weight, dos.triangulate(q, rec), energy


def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda")
    if kind == "dos":
        freq, weight, tri, energy = _bands(case, seed)
        return {"case": case, "freq": torch.tensor(freq, device=dev), "tri": torch.tensor(tri, device=dev),
                "energy": torch.tensor(energy, device=dev),
                "weight": None if weight is None else torch.tensor(weight, device=dev)}
    if kind == "multi":
        cells = [_cell(case[k]) for k in ("m0", "m1", "m2")]
        ctxs = [api.PhononContext.from_cell(c, phi) for c, phi in cells]
        which = np.arange(case["nq"], dtype=np.int64) % 3
        return {"case": case, "ctxs": ctxs, "cell": which, "q": _qpoints(case["nq"], seed),
                "opts": api.EigOpts(jobz="N", vel=case["vel"], precision=_prec(case))}
    cell, phi = _cell(case["m"])
    n = cell.n
    if kind == "values":
        with api.PhononContext.from_cell(cell, phi) as ctx:
            d = ctx.dynamical_matrix(_qpoints(1, seed)[0])
        a = torch.tensor(np.ascontiguousarray(d.T), device=dev)   # row-major transpose: column-major D
        return {"case": case, "n": n, "a": a, "work": torch.empty_like(a),
                "w": torch.zeros(n, dtype=torch.float64, device=dev),
                "m": torch.zeros(1, dtype=torch.int64, device=dev),
                "info": torch.zeros(1, dtype=torch.int64, device=dev)}
    q = _qpoints(case["nq"], seed)
    if kind == "fit":
        return {"case": case, "spec": autograd.PhononSpectrum.from_cell(cell, precision=_prec(case)),
                "q": torch.tensor(q, device=dev, requires_grad=True),
                "phi": torch.tensor(phi, device=dev, requires_grad=True),
                "target": torch.tensor(_targets(n, case["nq"], seed), device=dev)}
    ctx = api.PhononContext.from_cell(cell, phi)
    jobz = "V" if case["vectors"] else "N"
    if kind == "solve":
        opts = api.EigOpts(jobz=jobz, vel=case["vel"], precision=_prec(case))
        if case["il"]:
            opts.range, opts.il, opts.iu = "I", case["il"], case["iu"]
        return {"case": case, "ctx": ctx, "q": q, "opts": opts, "ref": _reference(n, seed)}
    nq = case["nq"]

    def zeros(shape, dtype):
        return torch.zeros(shape, dtype=dtype, device=dev)
    return {"case": case, "ctx": ctx, "opts": api.EigOpts(jobz=jobz, vel=case["vel"], precision=_prec(case)),
            "q": torch.tensor(np.asfortranarray(q).ravel(order="F"), device=dev),
            "w": zeros((nq, n), torch.float64), "m": zeros(nq, torch.int64), "nz": zeros(nq, torch.int64),
            "info": zeros(nq, torch.int64), "vel": zeros((nq, n, 3), torch.float64) if case["vel"] else None,
            "z": zeros((nq, n, n), torch.complex128) if case["vectors"] else None,
            "ref": torch.tensor(_reference(n, seed), device=dev)}


def _targets(n, nq, seed):
    rng = np.random.default_rng(7000 + seed)
    return np.sort(rng.uniform(1.0, 1600.0, (nq, n)), axis=1)


# ---------------------------------------------------------------------------
# one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        r = state["ctx"].solve(state["q"], state["opts"], want_z=case["vectors"])
        out = {"m": r.m, "info": r.info, "w": r.w}
        if case["vel"]:
            out["vel"] = r.vel
        if case["vectors"]:
            out["z"] = _fix_phase(r.z, state["ref"])
        return out
    if kind == "device":
        state["ctx"].solve_device(state["q"], state["opts"], state["w"], state["m"], state["nz"], state["info"],
                                  vel_dev=state["vel"], z_dev=state["z"])
        out = {"m": state["m"], "info": state["info"], "w": state["w"]}
        if case["vel"]:
            out["vel"] = state["vel"]
        if case["vectors"]:
            z = state["z"]                       # z[t, j, r]: component r of eigenvector j
            ph = z.conj() @ state["ref"]
            out["z"] = z * (ph / ph.abs())[..., None]
        return out
    if kind == "multi":
        r = api.solve_multi(state["ctxs"], state["cell"], state["q"], state["opts"], want_z=False)
        out = {"m": r.m, "info": r.info, "w": r.w}
        if case["vel"]:
            out["vel"] = r.vel
        return out
    if kind == "fit":
        w = state["spec"].frequencies(state["q"], state["phi"])
        loss = ((w - state["target"]) ** 2).sum()
        gq, gphi = torch.autograd.grad(loss, (state["q"], state["phi"]))
        return {"w": w.detach(), "grad_q": gq, "grad_phi": gphi}
    if kind == "values":
        n = state["n"]
        state["work"].copy_(state["a"])          # the entry point overwrites its matrix
        lowest = case["lowest"]
        rc = api.heevx_values_noalloc(state["work"].data_ptr(), n, n, state["w"].data_ptr(), state["m"].data_ptr(),
                                      state["info"].data_ptr(), range="I" if lowest else "A", il=1,
                                      iu=lowest if lowest else n,
                                      stream=torch.cuda.current_stream().cuda_stream)
        if rc:
            raise api.PPError(rc, "pp_heevx_values_noalloc")
        return {"w": state["w"][:lowest] if lowest else state["w"], "m": state["m"], "info": state["info"]}
    d, nd = dos.linear_triangulation_device(state["freq"], state["tri"], state["energy"], func_dev=state["weight"])
    return {"dos": d, "nd": nd}


def _fix_phase(z, ref):
    """Every eigenvector (column) times the phase that makes its overlap with `ref` real and positive."""
    ph = ref.conj() @ z
    return z * (ph.conj() / np.abs(ph))[:, None, :]


# ---------------------------------------------------------------------------
# what a pass cannot do without
def _solve_work(n, nq, mm, vecs, vel, zout):
    flops = nq * (16.0 / 3.0 * n ** 3 + (8.0 * n * n * mm if vecs else 0.0))
    byts = 8.0 * n * n + nq * mm * (8.0 + (24.0 if vel else 0.0) + (16.0 * n if zout else 0.0))
    return flops, byts


def work(case):
    kind = case["kind"]
    if kind == "dos":
        nk, nb, ne = case["grid"] ** 2, case["bands"], case["energies"]
        # every triangle and band contributes over the energies its three vertices span: about one in twenty
        flops = 2.0 * nk * nb * ne * 40.0 / 20.0
        return {"bytes": 8.0 * nk * nb * (2 if case["weighted"] else 1) + 24.0 * 2 * nk + 24.0 * ne, "flops": flops}
    if kind == "multi":
        flops = byts = 0.0
        for k in range(3):
            nq = len(range(k, case["nq"], 3))
            n = _order(case["m%d" % k])
            f, b = _solve_work(n, nq, n, case["vel"], case["vel"], False)
            flops, byts = flops + f, byts + b
        return {"bytes": byts, "flops": flops}
    n = _order(case["m"])
    if kind == "values":
        return {"bytes": 16.0 * n * n + 8.0 * n, "flops": 16.0 / 3.0 * n ** 3}
    if kind == "fit":
        nq = case["nq"]
        f, b = _solve_work(n, nq, n, True, False, False)
        return {"bytes": b + 8.0 * n * n + 16.0 * nq * n, "flops": f + nq * 4.0 * n ** 3}
    mm = case["iu"] - case["il"] + 1 if case.get("il") else n
    f, b = _solve_work(n, case["nq"], mm, case["vectors"] or case["vel"], case["vel"], case["vectors"])
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch
class _Model:
    """D(q) and its boundary blocks of one cell from its geometry and force constants."""

    def __init__(self, m):
        dev = torch.device("cuda")
        cell, phi = _cell(m)
        self.n, self.N = cell.n, cell.natom
        self.lat = torch.tensor(cell.lat, device=dev)
        self.crys = torch.tensor(geometry.crys_from_positions(cell.lat, cell.real_pos), device=dev)
        pos = torch.tensor(cell.real_pos, device=dev)
        mass = torch.tensor(cell.masses, device=dev)[torch.tensor(cell.at_types - 1, device=dev)]
        self.phi = torch.tensor(phi, device=dev)
        self.rec = torch.tensor(geometry.reciprocal_lattice(cell.lat), device=dev)
        self.shifts = [(i, j) for i in (-1, 0, 1) for j in (-1, 0, 1)]
        dist = []
        for i, j in self.shifts:
            img = (self.crys + torch.tensor([i, j, 0.0], device=dev, dtype=torch.float64)) @ self.lat
            dist.append((pos[:, None, :] - img[None, :, :]).square().sum(-1).sqrt())
        dist = torch.stack(dist)
        tie = dist < dist.min(dim=0).values + TIE
        upper = torch.ones(self.N, self.N, device=dev).triu().bool()
        self.tie = torch.where(upper, tie, tie.transpose(1, 2).flip(0))   # an (I > J) block mirrors (J, I)
        self.scale = 1.0 / (self.tie.sum(0) * (mass[:, None] * mass[None, :]).sqrt())
        away = self.tie.clone()
        away[4] = False
        block = (self.phi.view(self.N, 3, self.N, 3) != 0).any(3).any(1)
        self.pairs = (away.any(0) & block & upper).nonzero()

    def angle(self, q, s, rows=None, cols=None):
        cr = self.crys if rows is None else self.crys[rows]
        cc = self.crys if cols is None else self.crys[cols]
        shift = torch.tensor([self.shifts[s][0], self.shifts[s][1], 0.0], device=q.device, dtype=torch.float64)
        d = cc[None, :, :] + shift - cr[:, None, :] if rows is None else cc + shift - cr
        return -2.0 * PI_F * (d * q).sum(-1)

    def factor(self, q):
        """p(I, J): the mean phase over the tie set and the masses."""
        p = torch.zeros(self.N, self.N, dtype=torch.complex128, device=q.device)
        for s in range(9):
            p = p + torch.polar(self.tie[s].double(), self.angle(q, s))
        p = p * self.scale
        up = p.triu(1)
        return up + up.conj().T + torch.diag(p.diagonal().real).to(p.dtype)

    def matrix(self, q, phi=None):
        p = self.factor(q)
        big = p[:, None, :, None].expand(self.N, 3, self.N, 3).reshape(self.n, self.n)
        return (self.phi if phi is None else phi) * big

    def velocities(self, q, w, z):
        I, J = self.pairs[:, 0], self.pairs[:, 1]
        raw = torch.zeros(z.shape[1], 3, dtype=torch.float64, device=q.device)
        zb = z.view(self.N, 3, -1)
        for k in range(0, len(I), 256):
            i, j = I[k:k + 256], J[k:k + 256]
            block = self.phi.view(self.N, 3, self.N, 3)[i, :, j, :].to(z.dtype)
            h = (zb[i].conj() * torch.bmm(block, zb[j])).sum(1)                 # (pairs, modes)
            g = torch.zeros(len(i), 3, dtype=z.dtype, device=q.device)
            for s, (a, b) in enumerate(self.shifts):
                if (a, b) == (0, 0):
                    continue
                t = a * self.lat[0] + b * self.lat[1]
                e = torch.polar(self.tie[s][i, j].double(), self.angle(q, s, i, j))
                g += -1j * e[:, None] * t[None, :].to(z.dtype)
            g = g * self.scale[i, j][:, None]
            raw += 2.0 * torch.einsum("pk,pm->mk", g, h).real
        f = C2 * C1SQ * 100.0 * 2.0 * PI_F
        return raw / (2.0 * w.abs()).clamp_min(1e-3)[:, None] * f


@functools.lru_cache(maxsize=4)
def _model(m):
    return _Model(m)


def _freq(lam):
    return lam.sign() * lam.abs().sqrt() * (C1 * C2)


def _spectrum(model, q, vel, vecs):
    q = torch.as_tensor(q, device="cuda")
    D = model.matrix(q)
    if not (vel or vecs):
        return _freq(torch.linalg.eigvalsh(D)), None, None
    lam, z = torch.linalg.eigh(D)
    w = _freq(lam)
    return w, (model.velocities(q, w, z) if vel else None), z


def exact(case, seed):
    kind = case["kind"]
    if kind == "dos":
        return _exact_dos(case, seed)
    if kind == "values":
        lam = torch.linalg.eigvalsh(_model(case["m"]).matrix(torch.as_tensor(_qpoints(1, seed)[0], device="cuda")))
        return {"w": lam[:case["lowest"]] if case["lowest"] else lam, "m": None, "info": None}
    q = _qpoints(case["nq"], seed)
    if kind == "fit":
        mo = _model(case["m"])
        target = torch.tensor(_targets(mo.n, case["nq"], seed), device="cuda")
        qt = torch.tensor(q, device="cuda", requires_grad=True)
        phi = mo.phi.clone().requires_grad_(True)
        ws = []
        gq, gphi = torch.zeros_like(qt), torch.zeros_like(phi)
        for t in range(case["nq"]):
            w = _freq(torch.linalg.eigvalsh(mo.matrix(qt[t], phi)))
            g = torch.autograd.grad(((w - target[t]) ** 2).sum(), (qt, phi))
            gq, gphi = gq + g[0], gphi + g[1]
            ws.append(w.detach())
        # the force constants are symmetric: half of a pair's derivative on each of its two entries
        return {"w": torch.stack(ws), "grad_q": gq, "grad_phi": 0.5 * (gphi + gphi.T)}
    if kind == "multi":
        ms = [case[k] for k in ("m0", "m1", "m2")]
        nmax = max(_order(m) for m in ms)
        w = torch.zeros(case["nq"], nmax, dtype=torch.float64)
        v = torch.zeros(case["nq"], nmax, 3, dtype=torch.float64)
        for t in range(case["nq"]):
            mo = _model(ms[t % 3])
            wt, vt, _ = _spectrum(mo, q[t], case["vel"], False)
            w[t, :mo.n] = wt.cpu()
            if case["vel"]:
                v[t, :mo.n] = vt.cpu()
        out = {"m": None, "info": None, "w": w}
        if case["vel"]:
            out["vel"] = v
        return out
    mo = _model(case["m"])
    n = mo.n
    lo, hi = (case["il"] - 1, case["iu"]) if case.get("il") else (0, n)
    w = torch.zeros(case["nq"], n, dtype=torch.float64)
    v = torch.zeros(case["nq"], n, 3, dtype=torch.float64)
    zs = []
    for t in range(case["nq"]):
        wt, vt, z = _spectrum(mo, q[t], case["vel"], case["vectors"])
        w[t, :hi - lo] = wt[lo:hi].cpu()
        if case["vel"]:
            v[t, :hi - lo] = vt[lo:hi].cpu()
        if case["vectors"]:
            z = z[:, lo:hi]
            ph = torch.tensor(_reference(n, seed), device="cuda").conj() @ z
            z = z * (ph.conj() / ph.abs())[None, :]
            zs.append((z if kind == "solve" else z.T).cpu())
    out = {"m": None, "info": None, "w": w}
    if case["vel"]:
        out["vel"] = v
    if case["vectors"]:
        out["z"] = np.stack([x.numpy() for x in zs]) if kind == "solve" else torch.stack(zs)
    return out


def _exact_dos(case, seed):
    freq, weight, tri, energy = (None if x is None else torch.as_tensor(x, device="cuda") for x in _bands(case, seed))
    f = torch.ones_like(freq) if weight is None else weight
    e, order = torch.sort(freq[tri], dim=1)           # (triangles, 3, bands)
    f = torch.gather(f[tri], 1, order)
    (e0, e1, e2), (f0, f1, f2) = e.unbind(1), f.unbind(1)
    full = f0 + f1 + f2
    dos_, nd_ = torch.zeros_like(energy), torch.zeros_like(energy)
    for k, E in enumerate(energy):
        a, b = (E - e0) / (e1 - e0), (E - e0) / (e2 - e0)
        da, db = 1 / (e1 - e0), 1 / (e2 - e0)
        s = (3 - a - b) * f0 + a * f1 + b * f2
        low_n = s * a * b
        low_d = (da * b + a * db) * s + a * b * ((-da - db) * f0 + da * f1 + db * f2)
        c, d = (e2 - E) / (e2 - e0), (e2 - E) / (e2 - e1)
        dc, dd = -1 / (e2 - e0), -1 / (e2 - e1)
        up_n = (1 - d * c * c) * f0 + (1 - c * d * d) * f1 + (1 - 3 * c * d + d * c * c + c * d * d) * f2
        up_d = (-2 * c * dc * d - dd * c * c) * f0 + (-dc * d * d - 2 * c * d * dd) * f1 + \
            (-3 * d * dc - 3 * c * dd + 2 * c * d * dc + dd * c * c + 2 * c * d * dd + dc * d * d) * f2
        zero = torch.zeros_like(full)
        nd_[k] = torch.where(E < e0, zero, torch.where(E < e1, low_n, torch.where(E < e2, up_n, full))).sum()
        dos_[k] = torch.where((E < e0) | (E >= e2), zero, torch.where(E < e1, low_d, up_d)).sum()
    return {"dos": dos_, "nd": nd_}
