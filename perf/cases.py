"""
Timed cases: what programs have this package compute, through its public calls.

A case is one call of a user's loop on inputs that are on the GPU already:
an energy, energies with forces, a parameter-fit step, or the properties of
the D4 model, for one structure or a zero-padded batch.  Structures follow
the package's workload generators (uniform atoms in a cube at 0.01 atoms per
cubic Bohr, no two closer than 1.8 Bohr, the twelve-element mix; H/C/N/O for
single small molecules).  The dtype of the positions selects the method, as
in ``dftd4``: float64 the plain FP64 kernels, float32 the precision form.

``exact`` restates the model in float64 torch, one structure at a time.
"""

from __future__ import annotations

import functools
import importlib
import math
from pathlib import Path

import numpy as np
import torch

d4 = importlib.import_module("tad-dftd4_gb300")

ROOT = Path(__file__).resolve().parents[1]
DENSITY = 0.01  # atoms / Bohr^3
DMIN = 1.8      # Bohr
PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.40, "a2": 5.0, "s9": 1.0}
HCNO = ((1, 0.5), (6, 0.3), (7, 0.1), (8, 0.1))
MIX12 = ((1, 0.45), (6, 0.30)) + tuple((z, 0.025) for z in (5, 7, 8, 9, 14, 15, 16, 17, 35, 53))
NO_EXACT_FROM = 1600  # atoms: the dense float64 triples of a larger structure take too long


def _case(name=None, **kw):
    """A case with its defaults: ``nmin``..``nmax`` atoms per structure, padded to ``nmax``."""
    c = {"call": "forces", "dtype": "float32", "model": "d4", "batch": 1, "nmin": 32, "nmax": 32,
         "charged": False, "disp2": 60.0, "disp3": 40.0}
    c.update(kw)
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # one small molecule, energy only, in the default precision: the
        # smallest call (a dispersion correction added to a single point)
        _case("molecule32_f64_energy", call="energy", dtype="float64", nmin=32, nmax=32),
        # one molecule per step with forces: geometry optimisation, MD
        _case("molecule57_f64_forces", dtype="float64", nmin=57, nmax=57),
        # one molecular crystal cell or host-guest complex in double precision
        _case("complex301_f64_forces", dtype="float64", nmin=301, nmax=301, charged=True),
        # the displaced geometries of one 30-atom molecule (a numerical Hessian)
        _case("displaced360_f64_fused", call="fused", dtype="float64", batch=360, nmin=30, nmax=30),
        # a mixed batch in double precision (a benchmark set, reference data)
        _case("batch64_f64_forces", dtype="float64", batch=64, nmin=8, nmax=200, charged=True),
        # CN, charges, C6 and polarisabilities of a set of molecules
        _case("props64_f64", call="properties", dtype="float64", batch=64, nmin=8, nmax=150,
              charged=True),
        # the repository's headline: 512 structures of 8-200 atoms, energies and forces
        _case("batch512_f32_forces", batch=512, nmin=8, nmax=200, charged=True),
        # screening: energies of many small molecules
        _case("screen1000_f32_energy", call="energy", batch=1000, nmin=5, nmax=60, charged=True),
        # a fit of the damping parameters: energies, forces and parameter gradients
        _case("fit256_f32", call="fit", batch=256, nmin=20, nmax=150),
        # the same sizes with the pairwise-weighted model
        _case("d4s96_f32_forces", model="d4s", batch=96, nmin=20, nmax=147),
        # one protein-sized structure
        _case("protein997_f32_forces", nmin=997, nmax=997),
        # the largest: one 16000-atom structure with shortened cutoffs
        _case("large16k_f32_forces", nmin=16000, nmax=16000, disp2=50.0, disp3=25.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.randrange(6)
    if kind == 0:  # one molecule, double precision
        n = _log(rng, 5, 320)
        return _case(call=rng.choice(["energy", "forces"]), dtype="float64", nmin=n, nmax=n,
                     charged=rng.random() < 0.3)
    if kind == 1:  # a batch in double precision
        nmax = rng.randrange(12, 201)
        batch = max(2, min(_log(rng, 2, 400), int(4e8 / nmax ** 3)))
        return _case(call=rng.choice(["energy", "forces", "fused", "fit"]), dtype="float64",
                     batch=batch, nmin=rng.randrange(5, nmax + 1), nmax=nmax,
                     charged=rng.random() < 0.5)
    if kind == 2:  # a batch in the precision form
        nmax = rng.randrange(12, 221)
        return _case(call=rng.choice(["energy", "forces", "forces", "fused", "fit"]),
                     batch=max(2, min(_log(rng, 2, 1024), int(4e9 / nmax ** 3))),
                     nmin=rng.randrange(5, nmax + 1), nmax=nmax, charged=rng.random() < 0.5)
    if kind == 3:  # D4S batches
        nmax = rng.randrange(12, 151)
        return _case(call=rng.choice(["energy", "forces"]), model="d4s", dtype="float32",
                     batch=_log(rng, 1, 96), nmin=rng.randrange(5, nmax + 1), nmax=nmax)
    if kind == 4:  # properties
        nmax = rng.randrange(12, 201)
        return _case(call="properties", dtype="float64", batch=_log(rng, 1, 100),
                     nmin=rng.randrange(5, nmax + 1), nmax=nmax, charged=rng.random() < 0.5)
    n = _log(rng, 200, 16000)  # one structure in the precision form
    short = n > 1500
    return _case(call=rng.choice(["energy", "forces", "forces"]), nmin=n, nmax=n,
                 disp2=50.0 if short else 60.0, disp3=25.0 if short else 40.0)


# ---------------------------------------------------------------- inputs


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _too_close(pos, size):
    """(B, N) flags of the atoms nearer than DMIN to an earlier atom of their structure."""
    B, N, _ = pos.shape
    idx = torch.arange(N, device=pos.device)
    out = torch.zeros((B, N), dtype=torch.bool, device=pos.device)
    rows = max(1, int(3e7 / (B * N)))
    for a in range(0, N, rows):
        b = min(N, a + rows)
        d = pos[:, a:b, None, :] - pos[:, None, :, :]
        near = (d * d).sum(-1) < DMIN * DMIN
        near &= (idx[None, :] < idx[a:b, None])[None]
        out[:, a:b] = near.any(-1)
    return out & (idx[None, :] < size[:, None])


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    B, N = case["batch"], case["nmax"]
    size = rng.integers(case["nmin"], N + 1, size=B)
    table = HCNO if B == 1 and N < 100 else MIX12
    p = np.array([w for _, w in table])
    z = rng.choice(np.array([e for e, _ in table], dtype=np.int64), size=(B, N), p=p / p.sum())
    z[np.arange(N)[None, :] >= size[:, None]] = 0
    side = (size / DENSITY) ** (1.0 / 3.0)
    pos = rng.uniform(0.0, 1.0, (B, N, 3)) * side[:, None, None]
    dev = _device()
    dsize = torch.from_numpy(size).to(dev)
    for _ in range(400):
        bad = _too_close(torch.from_numpy(pos).to(dev), dsize).cpu().numpy()
        if not bad.any():
            break
        b, i = np.nonzero(bad)
        pos[b, i] = rng.uniform(0.0, 1.0, (len(b), 3)) * side[b, None]
    pos[z == 0] = 0.0
    charge = rng.integers(-1, 2, size=B).astype(np.float64) if case["charged"] else np.zeros(B)
    return z, pos, charge


def _tensors(case, seed):
    z, pos, charge = _inputs(case, seed)
    dev, dtype = _device(), getattr(torch, case["dtype"])
    return (torch.from_numpy(z).to(dev), torch.from_numpy(pos).to(dev, dtype),
            torch.from_numpy(charge).to(dev, dtype))


def prepare(case, seed):
    numbers, positions, charge = _tensors(case, seed)
    param = dict(PARAM)
    if case["call"] == "fit":
        param = {k: torch.tensor(v, dtype=positions.dtype, device=positions.device,
                                 requires_grad=True) for k, v in PARAM.items()}
    if case["call"] in ("forces", "fit"):
        positions.requires_grad_(True)
    cutoff = None
    if (case["disp2"], case["disp3"]) != (60.0, 40.0):
        cutoff = d4.Cutoff(disp2=case["disp2"], disp3=case["disp3"])
    return {"call": case["call"], "model": case["model"], "numbers": numbers,
            "positions": positions, "charge": charge, "param": param, "cutoff": cutoff}


def run(state):
    numbers, positions, charge = state["numbers"], state["positions"], state["charge"]
    param, call = state["param"], state["call"]
    if call == "properties":
        cn, q, c6, alpha = d4.get_properties(numbers, positions, charge)
        return {"cn": cn, "charges": q, "c6": c6, "alpha": alpha}
    kw = {"model": state["model"], "cutoff": state["cutoff"]}
    if call == "fused":
        energy, grad = d4.dispersion_energy_gradient(numbers, positions, charge, param, **kw)
        return {"energy": energy, "gradient": grad}
    energy = d4.dftd4(numbers, positions, charge, param, **kw)
    if call == "energy":
        return {"energy": energy}
    if call == "forces":
        (grad,) = torch.autograd.grad(energy.sum(), positions)
        return {"energy": energy.detach(), "gradient": grad}
    leaves = [positions, *param.values()]
    grads = torch.autograd.grad(energy.sum(), leaves)
    return {"energy": energy.detach(), "gradient": grads[0],
            "param_gradient": dict(zip(param, grads[1:]))}


# ---------------------------------------------------------------- work


def _within(t):
    """Share of the pairs of a cube of side 1 that are nearer than t."""
    if t >= 1.0:
        return 1.0
    return 4.0 / 3.0 * math.pi * t ** 3 - 1.5 * math.pi * t ** 4 + 1.6 * t ** 5 - t ** 6 / 6.0


def work(case):
    """Bytes of the inputs and outputs; operations of the expected sizes (transcendentals count
    one): CN 20 and BJ energy with two C6 122 per pair, EEQ n^3 / 3 + 4 n^2, ATM 60 per triple
    with at least two sides inside its cutoff; twice that again for the adjoint of all but
    the EEQ (which reuses its factor)."""
    real = 4 if case["dtype"] == "float32" else 8
    sizes = range(case["nmin"], case["nmax"] + 1)
    B, N = case["batch"], case["nmax"]
    atoms = pairs = near = triples = eeq = 0.0
    for n in sizes:
        side = (n / DENSITY) ** (1.0 / 3.0)
        f2, f3 = _within(case["disp2"] / side), _within(case["disp3"] / side)
        atoms += n
        pairs += n * (n - 1) / 2.0 * f2
        near += n * (n - 1) / 2.0 * _within(30.0 / side)
        triples += n * (n - 1) * (n - 2) / 6.0 * min(1.0, 2.06 * f3 * f3)
        eeq += n ** 3 / 3.0 + 4.0 * n * n
    scale = B / len(sizes)
    grad = case["call"] in ("forces", "fused", "fit")
    flops = 20.0 * near + 122.0 * pairs + 60.0 * triples
    byte = B * N * (8 + 3 * real) + B * real + B * N * real * (4 if grad else 1)
    if case["call"] == "properties":
        flops = 20.0 * near + 46.0 * pairs
        byte = B * N * (8 + 3 * real) + B * real + B * N * real * (3 + N)
    flops = flops * (3.0 if grad else 1.0) + eeq + (4.0 * atoms if grad else 0.0)
    return {"bytes": float(byte), "flops": float(flops * scale)}


# ---------------------------------------------------------------- float64 values


@functools.lru_cache(maxsize=1)
def _tables():
    with np.load(ROOT / "tad-dftd4_gb300" / "data" / "d4_tables.npz") as f:
        return {k: torch.from_numpy(np.array(f[k])).to(_device()) for k in f.files
                if k != "provenance"}


def _zeta(gam, qref, qmod):
    z = torch.exp(3.0 * (1.0 - torch.exp(gam * (1.0 - qref / (qmod - torch.finfo(qmod.dtype).eps)))))
    return torch.where(qmod > 0.0, z, math.exp(3.0))


def _ref_alpha(t, z):
    sysn = t["refsys"][z]
    zeff = t["zeff"][sysn].double()
    scale = torch.where(sysn > 0, _zeta(2.0 * t["gam"][sysn], zeff, t["clsh"][z] + zeff), 0.0)
    sec = t["secscale"][sysn][..., None] * t["secalpha"][sysn] * scale[..., None]
    return (t["refascale"][z][..., None]
            * (t["refalpha"][z] - t["refscount"][z][..., None] * sec)).clamp_min(0.0)


def _weights(t, z, cn, q, model):
    """Charge-scaled reference weights (1 or n partners, n, 7)."""
    refc = t["refc"][z]
    arg = -(cn[:, None] - t["refcovcn"][z]) ** 2
    wf = torch.full((1, len(z)), 6.0, dtype=cn.dtype, device=cn.device)
    if model == "d4s":
        wf = t["wfpair"][z[:, None], z[None, :]].transpose(0, 1)
    g = torch.exp(arg[None] * wf[..., None])
    g3 = g + g ** 2 + g ** 3
    g = torch.where(refc == 3, g3, torch.where(refc == 1, g, torch.exp(arg)[None]
                                               if model == "d4" else g))
    g = torch.where(refc > 0, g, 0.0)
    norm = g.sum(-1, keepdim=True)
    last = (t["refcovcn"][z] == t["refcovcn"][z].amax(-1, keepdim=True)).double()
    some = norm > 0.0
    g = torch.where(some, g / torch.where(some, norm, 1.0), last)
    zeff = t["zeff"][z].double()[:, None]
    zet = _zeta(2.0 * t["gam"][z][:, None], t["clsq"][z] + zeff, q[:, None] + zeff)
    return torch.where(refc > 0, zet, 0.0) * g


def _c6(t, gw, alpha):
    fw = 3.0 / math.pi * t["freq_weights"]
    if gw.shape[0] == 1:
        a = torch.einsum("nr,nrw->nw", gw[0], alpha)
        return (a * fw) @ a.T
    p = torch.einsum("mnr,nrw->mnw", gw, alpha)  # [partner, atom]
    return torch.einsum("mnw,nmw,w->nm", p, p, fw)


def _safe(r2, eye):
    return torch.where(eye, 1.0, r2)


def _model(z, pos, charge, model):
    """Pair distances, CN, charges and both C6 matrices of one structure (n >= 1 atoms)."""
    t = _tables()
    n = len(z)
    eye = torch.eye(n, dtype=torch.bool, device=pos.device)
    d = pos[:, None] - pos[None]
    r2 = (d * d).sum(-1)
    r = torch.sqrt(_safe(r2, eye))
    rc = t["cov_d3"][z][:, None] + t["cov_d3"][z][None]
    cf = 0.5 * torch.erfc(7.5 * (r / rc - 1.0))
    en = t["en"][z]
    den = 4.10451 * torch.exp(-((en[:, None] - en[None]).abs() + 19.08857) ** 2
                              / (2.0 * 11.28174 ** 2))
    cn = torch.where(~eye & (r <= 30.0), den * cf, 0.0).sum(-1)
    cq = torch.where(~eye & (r <= 25.0), cf, 0.0).sum(-1)
    cq = torch.log1p(torch.expm1(cq) / (1.0 + torch.exp(cq - 8.0)))
    some = cq > 0.0
    root = torch.where(some, torch.sqrt(torch.where(some, cq, 1.0)), 0.0)
    rad = t["eeq_rad"][z]
    gam = 1.0 / torch.sqrt(rad[:, None] ** 2 + rad[None] ** 2)
    amat = torch.where(eye, 0.0, torch.erf(gam * r) / r) + torch.diag(
        t["eeq_eta"][z] + math.sqrt(2.0 / math.pi) / rad)
    rhs = torch.stack([-t["eeq_chi"][z] + t["eeq_kcn"][z] * root, torch.ones_like(rad)], dim=1)
    chol = torch.linalg.cholesky(amat)
    sol = torch.cholesky_solve(rhs, chol)
    q = sol[:, 0] - sol[:, 1] * ((sol[:, 0].sum() - charge) / sol[:, 1].sum())
    alpha = _ref_alpha(t, z)
    return (r2, r, eye, cn, q, alpha, _weights(t, z, cn, q, model),
            _weights(t, z, cn, torch.zeros_like(q), model))


def _triples(r2, root, radii, s9, cut, grad):
    """ATM energies per atom, and d(their sum) / d(r2, root, radii, s9), row blocks at a time."""
    n = len(r2)
    leaves = [x.detach().requires_grad_(grad) for x in (r2, root, radii, s9)]
    r2, root, radii, s9 = leaves
    off = ~torch.eye(n, dtype=torch.bool, device=r2.device)
    energy, total = [], [torch.zeros_like(x) for x in leaves]
    rows = max(1, int(2.5e7 / (n * n)))
    for a in range(0, n, rows):
        s = slice(a, min(n, a + rows))
        ok = off[s, :, None] & off[s, None, :] & off[None]
        ok &= (r2[s, :, None] <= cut * cut) & (r2[None] <= cut * cut)
        x, y, w = r2[s, :, None], r2[s, None, :], r2[None]
        prod = torch.where(ok, x * y * w, 1.0)
        r1 = torch.sqrt(prod)
        rr = radii[s, :, None] * radii[s, None, :] * radii[None]
        damp = 1.0 / (1.0 + 6.0 * (rr / r1) ** (16.0 / 3.0))
        ang = (0.375 * (x + w - y) * (x - w + y) * (w + y - x) / prod + 1.0) / (r1 * prod)
        e = torch.where(ok, ang * damp * root[s, :, None] * root[s, None, :] * root[None], 0.0)
        e = s9 / 6.0 * e.sum((-2, -1))
        energy.append(e.detach())
        if grad:
            for k, g in enumerate(torch.autograd.grad(e.sum(), leaves)):
                total[k] += g
    return torch.cat(energy), total


def _exact_one(case, z, pos, charge, param):
    t, call, n = _tables(), case["call"], len(z)
    grad = call in ("forces", "fused", "fit")
    pos = pos.clone().requires_grad_(grad)
    r2, r, eye, cn, q, alpha, gw, gw0 = _model(z, pos, charge, case["model"])
    c6 = _c6(t, gw, alpha)
    if call == "properties":
        a0 = torch.einsum("nr,nr->n", gw[0], alpha[..., 0])
        return {"cn": cn, "charges": q, "c6": c6, "alpha": a0}
    c60 = _c6(t, gw0, alpha)
    r4 = t["r4r2"][z]
    qq = 3.0 * r4[:, None] * r4[None]
    radii = param["a1"] * torch.sqrt(qq) + param["a2"]
    f6, f8 = 1.0 / (r ** 6 + radii ** 6), 1.0 / (r ** 8 + radii ** 8)
    inside = ~eye & (r <= case["disp2"])
    e2 = -0.5 * torch.where(inside, c6 * (param["s6"] * f6 + param["s8"] * qq * f8), 0.0).sum(-1)
    r2 = _safe(r2, eye)
    root = torch.sqrt(c60.abs())
    s9 = torch.as_tensor(param["s9"], dtype=torch.float64, device=pos.device)
    e3, g = _triples(r2, root, radii, s9, case["disp3"], grad)
    out = {"energy": (e2 + e3).detach()}
    if grad:
        leaves = [pos] + ([param[k] for k in PARAM] if call == "fit" else [])
        total = e2.sum() + sum((a.detach() * b).sum() for a, b in zip(g, (r2, root, radii, s9)))
        got = torch.autograd.grad(total, leaves)
        out["gradient"] = got[0]
        if call == "fit":
            out["param_gradient"] = dict(zip(PARAM, got[1:]))
    return out


def exact(case, seed):
    if case["nmax"] >= NO_EXACT_FROM:
        return None
    numbers, positions, charge = _tensors(case, seed)
    B, N = numbers.shape
    param = {k: torch.tensor(v, dtype=positions.dtype, device=positions.device).double()
             for k, v in PARAM.items()} if case["call"] == "fit" else dict(PARAM)
    if case["call"] == "fit":
        param = {k: v.requires_grad_(True) for k, v in param.items()}
    out = {}
    for b in range(B):
        n = int((numbers[b] != 0).sum())
        one = _exact_one(case, numbers[b, :n], positions[b, :n].double(), charge[b].double(),
                         param)
        for key, v in one.items():
            if key == "param_gradient":
                acc = out.setdefault(key, {k: torch.zeros_like(x) for k, x in v.items()})
                for k, x in v.items():
                    acc[k] += x
                continue
            shape = (B, N, N) if key == "c6" else (B, N, 3) if key == "gradient" else (B, N)
            full = out.setdefault(key, torch.zeros(shape, dtype=torch.float64, device=v.device))
            full[(b, slice(0, n), slice(0, n)) if key == "c6" else (b, slice(0, n))] = v.detach()
    return out
