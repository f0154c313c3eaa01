"""The workloads by which this library's speed is followed.

Each case is one call (or the short chain of calls) that a GW/BSE program makes
through the public entry points, on seeded synthetic tensors of the
distributions of ``quasix_b200.synth``: occupied energies uniform in
[-1.2, -0.3] Ha, virtual ones in [0.05, 3.0] Ha, B symmetric and normal,
rescaled to a given ||Pi(0)||_2.  The tensors live on the GPU, as the output of
a density-fitting step does; energies are host arrays.  The sizes span
the library's own workloads: nmo 24 / naux 84 (the smallest G0W0), nmo 40-400
(batches), nmo 200 / naux 700 (gradients) and nmo 300 / naux 1000 (evGW).

Kinds:
  evgw       run_evgw_blocks, one iteration over every orbital (AC, Pade, linearized QP)
  sigma      get_sigma_diag of the 2 k orbitals around the gap, or of all of them (k = 0),
             which is one evGW step up to the Pade fit
  cd         g0w0_cd (contour deformation, linearized QP) of those orbitals
  batch      g0w0_cd_batch over systems of different sizes
  grad       the adjoint of the CD QP energies of HOMO and LUMO, given the roots
  bse_apply  BSE-TDA Hamiltonian times a block of vectors
  bse_solve  BSE-TDA kernel set-up and lowest roots (Davidson)
"""
import math

import numpy as np
import torch

import quasix_b200 as qx
from quasix_b200 import bse as qbse
from quasix_b200 import grad as qgrad
from quasix_b200 import gw as qgw

DEV = "cuda:0"
F8 = torch.float64


# ---------------------------------------------------------------------------
# The cases.
# ---------------------------------------------------------------------------
def _case(kind, nocc, nvir, naux, nw=32, k=2, precision="fp64", pi_norm=2.0, **more):
    return dict(kind=kind, nocc=nocc, nvir=nvir, naux=naux, nw=nw, k=k, precision=precision, pi_norm=pi_norm, **more)


def listed():
    def named(name, *a, **kw):
        return dict(_case(*a, **kw), name=name)

    return [
        # A small molecule's frontier levels by contour deformation: latency and launches.
        named("cd_nmo24", "cd", 5, 19, 84, nw=16, k=2),
        # A small molecule's Sigma_c(iw) of two levels each side of the gap, odd sizes.
        named("sigma_nmo40", "sigma", 7, 33, 139, nw=24, k=2),
        # G0W0 (the first evGW iteration) of a mid-sized molecule, every orbital, in
        # plain FP64, the default precision.
        named("evgw_nmo121", "evgw", 20, 101, 423, nw=32, pi_norm=1.5),
        # An evGW step of a large molecule in FP64 and in the FP16 split form.
        named("sigma_nmo300_all", "sigma", 40, 260, 1000, nw=32, k=0, pi_norm=4.0),
        named("sigma_nmo300_all_fp16x3", "sigma", 40, 260, 1000, nw=32, k=0, precision="fp16x3", pi_norm=4.0),
        # G0W0 of the frontier levels only, where P0 and the inversion dominate.
        named("sigma_nmo300_frontier", "sigma", 40, 260, 1000, nw=32, k=2, pi_norm=4.0),
        # The reference's default grid (100 points) in the BF16 split form, ragged sizes.
        named("sigma_nmo201_bf16x3", "sigma", 31, 170, 703, nw=100, k=5, precision="bf16x3"),
        # Screening runs over several molecules of uneven sizes in one call.
        named("batch_fp64", "batch", 0, 0, 0, nw=24, k=3, systems=8, nmo_lo=40, nmo_hi=200),
        named("batch_fp16x3", "batch", 0, 0, 0, nw=24, k=3, systems=8, nmo_lo=40, nmo_hi=400, precision="fp16x3"),
        # Gradients of HOMO and LUMO with respect to the energies and the whole tensor.
        named("grad_nmo200", "grad", 30, 170, 700, nw=24),
        # A caller's own eigensolver on the BSE Hamiltonian: blocks of ten vectors.
        named("bse_apply_dim10400", "bse_apply", 40, 260, 1000, vectors=10, pi_norm=4.0),
        # Optical spectrum of a mid-sized molecule: kernel set-up and five roots.
        named("bse_solve_dim3264", "bse_solve", 24, 136, 560, roots=5, pi_norm=3.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """(nocc, nvir, naux) of a molecule of lo..hi orbitals, as the listed ones."""
    nmo = _log_int(rng, lo, hi)
    nocc = max(3, int(round(nmo * rng.uniform(0.13, 0.21))))
    naux = max(8, min(1000, int(round(nmo * rng.uniform(3.2, 3.6))) + rng.randint(-3, 3)))
    return nocc, nmo - nocc, naux


def draw(rng):
    kind = rng.choice(["cd", "sigma", "sigma", "evgw", "evgw", "batch", "grad", "bse_apply", "bse_solve"])
    split = rng.choice(["fp64", "fp64", "fp16x3", "bf16x3"])
    pi = round(rng.uniform(1.0, 4.0), 2)
    if kind == "cd":
        return _case(kind, *_size(rng, 24, 300), nw=rng.randint(16, 32), k=rng.randint(1, 3), precision=split,
                     pi_norm=pi)
    if kind == "sigma":
        k = rng.choice([0, 0, 1, 2, 3])
        return _case(kind, *_size(rng, 24, 290), nw=rng.randint(16, 100 if k else 32), k=k, precision=split,
                     pi_norm=pi)
    if kind == "evgw":
        return _case(kind, *_size(rng, 24, 200), nw=rng.randint(18, 32), pi_norm=round(rng.uniform(1.0, 2.0), 2))
    if kind == "batch":
        return _case(kind, 0, 0, 0, nw=rng.randint(16, 24), k=rng.randint(1, 3), systems=rng.randint(3, 10),
                     nmo_lo=rng.randint(30, 60), nmo_hi=rng.randint(100, 200),
                     precision=rng.choice(["fp64", "fp16x3"]))
    if kind == "grad":
        return _case(kind, *_size(rng, 60, 200), nw=rng.randint(16, 24), pi_norm=round(rng.uniform(1.0, 2.0), 2))
    if kind == "bse_apply":
        nocc, nvir, naux = _size(rng, 60, 290)
        prec = rng.choice(["fp64", "fp64", "fp16x3"])
        if prec != "fp64":
            naux += naux % 2  # the split BSE kernels take an even naux
        return _case(kind, nocc, nvir, naux, vectors=rng.randint(1, 12), precision=prec, pi_norm=pi)
    return _case(kind, *_size(rng, 60, 140), roots=rng.randint(3, 6), pi_norm=pi)


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _system(nocc, nvir, naux, pi_norm, seed):
    """(energies [nmo], lpq [naux, nmo, nmo]) on the GPU."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    nmo = nocc + nvir
    kw = dict(generator=g, device=DEV, dtype=F8)
    e = torch.cat([torch.sort(torch.rand(nocc, **kw) * 0.9 - 1.2).values,
                   torch.sort(torch.rand(nvir, **kw) * 2.95 + 0.05).values])
    lpq = torch.randn(naux, nmo, nmo, **kw) * 0.05
    lpq = torch.triu(lpq) + torch.triu(lpq, 1).transpose(1, 2)
    bov = lpq[:, :nocc, nocc:].reshape(naux, -1)
    w = 4.0 / (e[None, nocc:] - e[:nocc, None]).reshape(-1)
    x = torch.ones(naux, dtype=F8, device=DEV)
    norm = None
    for _ in range(40):  # the largest eigenvalue of -Pi(0) by power iteration
        x = bov @ (w * (bov.T @ x))
        norm = x.norm()
        x = x / norm
    return e, (lpq * torch.sqrt(pi_norm / norm)).contiguous()


def _exchange(lpq, nocc):
    return -(lpq[:, :, :nocc] ** 2).sum(dim=(0, 2))


def _targets(nocc, nmo, k):
    return list(range(max(0, nocc - k), min(nmo, nocc + k)))


def _batch_shapes(case, seed):
    rng = np.random.default_rng(seed)
    shapes = []
    for i in range(case["systems"]):
        # The sizes follow from the case and the index, the values from the seed.
        lo, hi = case["nmo_lo"], case["nmo_hi"]
        nmo = int(round(lo + (hi - lo) * ((i * 0.6180339887 + 0.43) % 1.0)))
        shapes.append((int(round(nmo / 6)), nmo - int(round(nmo / 6)), int(round(3.5 * nmo)),
                       float(rng.uniform(1.0, 4.0)), seed * 1009 + i))
    return shapes


def _bse_inputs(case, seed):
    nocc, nvir, naux = case["nocc"], case["nvir"], case["naux"]
    e, lpq = _system(nocc, nvir, naux, case["pi_norm"], seed)
    dia, dij, dab = qgrad.bse_blocks_t(lpq, nocc)
    c = 4.0 / (e[None, nocc:] - e[:nocc, None]).reshape(-1)
    eps0 = torch.eye(naux, dtype=F8, device=DEV) + dia.T @ (c[:, None] * dia)
    w0 = torch.linalg.inv(0.5 * (eps0 + eps0.T))
    w0 = (0.5 * (w0 + w0.T)).contiguous()
    delta = (e[None, nocc:] - e[:nocc, None]).reshape(-1).contiguous()
    return delta, dia, dij, dab, w0


def _vectors(case, seed):
    return np.random.default_rng(seed + 17).normal(size=(case["nocc"] * case["nvir"], case["vectors"]))


def _grad_inputs(case, seed):
    """Energies, lpq, targets and QP roots 0.05 Ha inside the gap (a fixed Vxc puts them there)."""
    nocc = case["nocc"]
    e, lpq = _system(nocc, case["nvir"], case["naux"], case["pi_norm"], seed)
    return e, lpq, [nocc - 1, nocc], torch.stack([e[nocc - 1] + 0.05, e[nocc] - 0.05])


def prepare(case, seed):
    kind, s = case["kind"], dict(case)
    if kind in ("evgw", "sigma", "cd"):
        e, lpq = _system(case["nocc"], case["nvir"], case["naux"], case["pi_norm"], seed)
        s.update(e=e.cpu().numpy(), lpq=lpq, vxc=_exchange(lpq, case["nocc"]).cpu().numpy(),
                 targets=_targets(case["nocc"], case["nocc"] + case["nvir"], case["k"] or case["nocc"] + case["nvir"]))
    elif kind == "batch":
        s["list"] = []
        for nocc, nvir, naux, pin, sd in _batch_shapes(case, seed):
            e, lpq = _system(nocc, nvir, naux, pin, sd)
            s["list"].append(dict(mo_energy=e.cpu().numpy(), lpq=lpq, vxc=_exchange(lpq, nocc).cpu().numpy(),
                                  nocc=nocc, targets=_targets(nocc, nocc + nvir, case["k"])))
    elif kind == "grad":
        e, lpq, tg, qp = _grad_inputs(case, seed)
        s.update(e=e, lpq=lpq, targets=tg, qp=qp.cpu().numpy())
    else:
        s["in"] = _bse_inputs(case, seed)
        if kind == "bse_apply":
            s["kernel"] = qbse.BSETDAKernel(case["nocc"], case["nvir"], case["naux"], *s["in"],
                                            precision=case["precision"])
            s["in"] = None
            s["x"] = _vectors(case, seed)
    return s


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------
_CD_KEYS = ("qp_energies", "z_factors", "sigma_c", "sigma_x")


def run(s):
    kind = s["kind"]
    if kind == "evgw":
        r = qx.run_evgw_blocks(s["e"], s["lpq"], s["vxc"], s["nocc"], fixed_iterations=1, nfreq=s["nw"],
                               precision=s["precision"])
        return {k: r[k] for k in ("qp_energies", "z_factors", "sigma_x", "sigma_c", "energies")}
    if kind == "sigma":
        return qgw.get_sigma_diag(s["e"], s["lpq"], s["targets"], s["nocc"], nw=s["nw"], precision=s["precision"])
    if kind == "cd":
        r = qgw.g0w0_cd(s["e"], s["lpq"], s["nocc"], s["targets"], nw=s["nw"], vxc=s["vxc"], qp_solver="linearized",
                        precision=s["precision"])
        return {k: r[k] for k in _CD_KEYS}
    if kind == "batch":
        rs = qgw.g0w0_cd_batch(s["list"], nw=s["nw"], qp_solver="linearized", precision=s["precision"])
        return [np.stack([r[k] for k in _CD_KEYS]) for r in rs]
    if kind == "grad":
        return qgrad.g0w0_cd_grad(s["e"], s["lpq"], s["nocc"], s["targets"], s["qp"], [1.0, 1.0], nw=s["nw"],
                                  precision=s["precision"])
    if kind == "bse_apply":
        return s["kernel"].apply_hamiltonian_batch(s["x"])
    kernel = qbse.BSETDAKernel(s["nocc"], s["nvir"], s["naux"], *s["in"], precision=s["precision"])
    r = kernel.solve_davidson(n_roots=s["roots"], max_iter=300, tol_residual=1e-10)
    kernel.close()
    v = r["eigenvectors"]  # of either sign: fixed by the largest component
    return r["eigenvalues"], v * np.sign(v[np.abs(v).argmax(0), np.arange(v.shape[1])])


# ---------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------
def _gw_work(nocc, nvir, naux, nw, npair):
    """P0 (half of a symmetric product), inversion, b^T W b over half of W."""
    nov = nocc * nvir
    flops = nw * (float(nov) * naux * (naux + 1) + float(naux) ** 3 + float(npair) * naux * (naux + 1))
    return flops, 8.0 * naux * (nov + npair)


def work(case):
    kind, nocc, nvir, naux, nw = (case[k] for k in ("kind", "nocc", "nvir", "naux", "nw"))
    nmo = nocc + nvir
    if kind == "batch":
        flops = byt = 0.0
        for o, v, x, _, _ in _batch_shapes(case, 0):
            f, b = _gw_work(o, v, x, nw, 2 * case["k"] * (o + v))
            flops, byt = flops + f, byt + b
    elif kind == "evgw":
        flops, byt = _gw_work(nocc, nvir, naux, nw, nmo * (nmo + 1) // 2)
    elif kind in ("sigma", "cd"):
        flops, byt = _gw_work(nocc, nvir, naux, nw, 2 * case["k"] * nmo or nmo * (nmo + 1) // 2)
    elif kind == "grad":
        # P0, the inversion and W b, then G and G B_ov.
        flops, byt = _gw_work(nocc, nvir, naux, nw, 2 * nmo)
        flops += 2.0 * nw * (float(nocc * nvir) * naux * naux + 2.0 * nmo * naux * naux)
        byt += 8.0 * naux * nmo * nmo
    else:
        nov = float(nocc * nvir)
        nvec = case["vectors"] if kind == "bse_apply" else 4 * case["roots"]
        # Direct term through T[a][j][Q], exchange through Z[Q], per vector.
        flops = nvec * (2.0 * nov * nvir * naux + 2.0 * nov * nocc * naux + 4.0 * nov * naux)
        byt = 8.0 * naux * (nov + nocc * nocc + float(nvir) * nvir)
    return {"bytes": byt, "flops": flops}


# ---------------------------------------------------------------------------
# The same results in plain 64-bit torch.
# ---------------------------------------------------------------------------
def _grid(nw, x0=0.5):
    t, w = np.polynomial.legendre.leggauss(nw)
    f, wt = x0 * (1 + t) / (1 - t), w * 2 * x0 / (1 - t) ** 2
    return torch.tensor(f, device=DEV), torch.tensor(wt, device=DEV)


def _wc(e, bov, nocc, f, real=False):
    """eps^-1 - I at one imaginary (or real) frequency."""
    d = (e[None, nocc:] - e[:nocc, None]).reshape(-1)
    c = 4.0 * d / (d * d - f * f) if real else 4.0 * d / (d * d + f * f)
    one = torch.eye(bov.shape[0], dtype=F8, device=DEV)
    return torch.linalg.inv(one + (bov * c) @ bov.T) - one


def _bov(lpq, nocc):
    return lpq[:, :nocc, nocc:].reshape(lpq.shape[0], -1)


def _wmat(e, lpq, nocc, orbs, freqs):
    """v[w][t][m] = b_tm^T Wc(i f_w) b_tm."""
    naux, nmo = lpq.shape[0], lpq.shape[1]
    b = lpq[:, orbs, :].permute(1, 2, 0).reshape(-1, naux).contiguous()
    bov = _bov(lpq, nocc)
    return torch.stack([((b @ _wc(e, bov, nocc, f)) * b).sum(1).reshape(len(orbs), nmo) for f in freqs])


def _gap_sigma(e, lpq, nocc, tg, om, freqs, wts):
    """Sigma_c of the levels tg at energies om inside the gap (no residues)."""
    v = _wmat(e, lpq, nocc, tg, freqs)
    x = om[:, None] - e[None, :]
    return -(v * (wts[:, None, None] * x / (x * x + (freqs ** 2)[:, None, None]))).sum(dim=(0, 2)) / math.pi


def _sigma_iw(e, lpq, nocc, orbs, nw):
    freqs, wts = _grid(nw)
    v = _wmat(e, lpq, nocc, orbs, freqs)
    iw = torch.cat([torch.zeros(1, dtype=F8, device=DEV), freqs[freqs < 5.0]])
    ef = 0.5 * (e[nocc - 1] + e[nocc])
    sgn = torch.tensor([-1.0 if n < nocc else 1.0 for n in orbs], dtype=F8, device=DEV)
    om = 1j * sgn[:, None] * iw[None, :]
    sig = torch.zeros(len(orbs), iw.numel(), dtype=torch.complex128, device=DEV)
    for k in range(iw.numel()):
        z = om[:, k][:, None] + (ef - e)[None, :]
        g = z[None] / (z[None] ** 2 + (freqs ** 2)[:, None, None])
        sig[:, k] = -(v * wts[:, None, None] * g).sum(dim=(0, 2)) / math.pi
    return sig.cpu().numpy(), om.cpu().numpy()


def _pade_points(n):
    a = list(range(1, min(40, n), 6))
    a += list(range(a[-1] + 4, n, 4)) if a else []
    return a[: len(a) // 2 * 2]


def _thiele(z, f):
    a = f.copy()
    for j in range(1, len(z)):
        a[j:] = (a[j - 1] - a[j:]) / ((z[j:] - z[j - 1]) * a[j:])
    return a


def _continued(w, z, a):
    x = 0.0
    for i in range(len(z) - 1, 0, -1):
        x = a[i] * (w - z[i - 1]) / (1.0 + x)
    return a[0] / (1.0 + x)


def _exact_evgw(case, e, lpq):
    nocc, nmo = case["nocc"], case["nocc"] + case["nvir"]
    e0 = e.cpu().numpy()
    sig, om = _sigma_iw(e, lpq, nocc, list(range(nmo)), case["nw"])
    pts, ef = _pade_points(sig.shape[1]), 0.5 * (e0[nocc - 1] + e0[nocc])
    sc = np.array([_continued(e0[n] - ef, om[n, pts], _thiele(om[n, pts], sig[n, pts])) for n in range(nmo)])
    # Z, and with it the QP energies, carry a finite difference's own error: no exact value.
    return dict(qp_energies=None, z_factors=None, sigma_x=_exchange(lpq, nocc).cpu().numpy(), sigma_c=sc,
                energies=[None])


def _exact_cd(case, nocc, e, lpq, targets):
    """qp, z, Sigma_c and Sigma_x of the linearized contour-deformation G0W0, Vxc = diag(Sigma_x)."""
    freqs, wts = _grid(case["nw"])
    v, bov = _wmat(e, lpq, nocc, targets, freqs), _bov(lpq, nocc)
    om = e[targets]
    x, f2 = om[:, None] - e[None, :], (freqs ** 2)[:, None, None]
    vw = v * wts[:, None, None]
    sig = -(vw * (x / (x * x + f2))).sum(dim=(0, 2)) / math.pi
    ds = -(vw * ((f2 - x * x) / (x * x + f2) ** 2)).sum(dim=(0, 2)) / math.pi
    d = (e[None, nocc:] - e[:nocc, None]).reshape(-1)
    for i, n in enumerate(targets):
        for m in range(lpq.shape[1]):
            occ = m < nocc
            if (occ and e[m] > om[i]) or (not occ and e[m] < om[i]):
                w = (e[m] - om[i]).abs()
                b = lpq[:, n, m]
                y = b + _wc(e, bov, nocc, w, real=True) @ b
                sig[i] += (-1.0 if occ else 1.0) * (b @ (y - b))
                t = bov.T @ y
                ds[i] -= (4.0 * d * 2.0 * w / (d * d - w * w) ** 2 * t * t).sum()
    z = torch.clamp(1.0 / (1.0 - ds), 0.1, 0.999)
    return {"qp_energies": om + z * sig, "z_factors": z, "sigma_c": sig, "sigma_x": _exchange(lpq, nocc)[targets]}


def _exact_grad(case, seed):
    nocc, nw = case["nocc"], case["nw"]
    e, lpq, tg, qp = _grad_inputs(case, seed)
    freqs, wts = _grid(nw)
    v = _wmat(e, lpq, nocc, tg, freqs)
    x, f2 = qp[:, None] - e[None, :], (freqs ** 2)[:, None, None]
    ds = -(v * wts[:, None, None] * ((f2 - x * x) / (x * x + f2) ** 2)).sum(dim=(0, 2)) / math.pi
    mu = 1.0 / (1.0 - ds)
    e, lpq = e.requires_grad_(True), lpq.requires_grad_(True)
    ge, gl = torch.autograd.grad((mu * (e[tg] + _exchange(lpq, nocc)[tg])).sum(), (e, lpq))
    for k in range(nw):
        s = (mu * _gap_sigma(e, lpq, nocc, tg, qp, freqs[k:k + 1], wts[k:k + 1])).sum()
        a, b = torch.autograd.grad(s, (e, lpq))
        ge, gl = ge + a, gl + b
    return ge, 0.5 * (gl + gl.transpose(1, 2)), mu


def exact(case, seed):
    kind, nocc, nvir = case["kind"], case["nocc"], case["nvir"]
    if kind in ("evgw", "sigma", "cd"):
        e, lpq = _system(nocc, nvir, case["naux"], case["pi_norm"], seed)
        if kind == "evgw":
            return _exact_evgw(case, e, lpq)
        tg = _targets(nocc, nocc + nvir, case["k"] or nocc + nvir)
        return _sigma_iw(e, lpq, nocc, tg, case["nw"]) if kind == "sigma" else _exact_cd(case, nocc, e, lpq, tg)
    if kind == "batch":
        out = []
        for o, v, x, pin, sd in _batch_shapes(case, seed):
            e, lpq = _system(o, v, x, pin, sd)
            r = _exact_cd(case, o, e, lpq, _targets(o, o + v, case["k"]))
            out.append(torch.stack([r[k] for k in _CD_KEYS]).cpu().numpy())
        return out
    if kind == "grad":
        return _exact_grad(case, seed)
    delta, dia, dij, dab, w0 = _bse_inputs(case, seed)
    ijw = dij @ w0
    if kind == "bse_apply":
        x = torch.tensor(_vectors(case, seed), device=DEV)
        y = delta[:, None] * x + 2.0 * dia @ (dia.T @ x)
        bab = dab.reshape(nvir, nvir, -1)
        for c in range(x.shape[1]):
            t = torch.einsum("abq,jb->ajq", bab, x[:, c].reshape(nocc, nvir))
            y[:, c] -= (ijw.reshape(nocc, -1) @ t.reshape(nvir, -1).T).reshape(-1)
        return y.cpu().numpy()
    kd = (ijw @ dab.T).reshape(nocc, nocc, nvir, nvir).permute(0, 2, 1, 3).reshape(nocc * nvir, -1)
    h = torch.diag(delta) + 2.0 * dia @ dia.T - kd
    ev, v = torch.linalg.eigh(0.5 * (h + h.T))
    v = v[:, : case["roots"]].cpu().numpy()
    return ev[: case["roots"]].cpu().numpy(), v * np.sign(v[np.abs(v).argmax(0), np.arange(v.shape[1])])
