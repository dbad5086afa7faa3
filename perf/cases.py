"""Workloads of the per-Fermi-orbital SIC path, timed through its public entry points.

Each case is one thing a host code asks of the library in an SCF iteration:
a whole SIC cycle after new orbitals (set_orbitals + cycle), a batch of
molecules, one pass of a chunked cycle, the basis-space derivatives at
converged potentials, the DFT density and potential, and GETVLXC on device
buffers.  The systems are those of publicrelease_2020_b200.workloads (water,
benzene, alkanes, the 40-atom synthetic system, C60), whose orbitals are drawn
on a coarse mesh and whose mesh is then replaced by one of the wanted size.
Every input follows from the seed.
"""
import dataclasses
import math

import numpy as np
import torch

from publicrelease_2020_b200 import sic as S
from publicrelease_2020_b200 import workloads as W
from publicrelease_2020_b200.batch import Batch

LDA, PBE, SCAN = "LDA-PW91*LDA-PW91", "GGA-PBE*GGA-PBE", "MGGA-SCAN*MGGA-SCAN"


def listed():
    return [
        # the smallest whole call: water in the reference's default basis on a coarse mesh
        dict(name="water_lda", kind="cycle", system="water", nrad=10, functional=LDA, precision="fp64", density="phi2"),
        # an ordinary molecule in the default basis, the drop-in precision and the mixed one
        dict(name="benzene_lda", kind="cycle", system="benzene", nrad=24, functional=LDA, precision="fp64",
             density="phi2"),
        dict(name="benzene_lda_mixed", kind="cycle", system="benzene", nrad=24, functional=LDA, precision="mixed",
             density="phi2"),
        # a meta-GGA cycle of a ring, 24 FOs of each spin (no multiple of any tile)
        dict(name="ring_scan", kind="cycle", system="ring", ncarbon=6, nrad=14, functional=SCAN, precision="fp64",
             density="phi2"),
        # the 40-atom, 512-function, 128-FO system on a part of its million points
        dict(name="c2_pbe", kind="cycle", system="synthetic", natoms=40, nbasis=512, nfo=128, nmsh=100_003,
             functional=PBE, precision="fp64", density="phi2"),
        dict(name="c2_pbe_mixed", kind="cycle", system="synthetic", natoms=40, nbasis=512, nfo=128, nmsh=150_000,
             functional=PBE, precision="mixed", density="phi2"),
        # the reference's own pair-route FO density
        dict(name="pairs_pbe", kind="cycle", system="synthetic", natoms=20, nbasis=256, nfo=64, nmsh=50_021,
             functional=PBE, precision="fp64", density="pairs"),
        # uneven molecules in one batched launch
        dict(name="batch_lda", kind="batch", count=6, max_carbons=4, nrad=10, functional=LDA, precision="fp64"),
        # one pass of a chunked cycle, 37 + 37 FOs
        dict(name="chain_scan_chunk", kind="chunk", system="chain", ncarbon=9, nrad=20, chunks=2, functional=SCAN,
             precision="fp64"),
        # backward: dE/dC, FOD gradient, atomic force terms and SIC Hamiltonian at cached potentials
        dict(name="benzene_grad", kind="grad", system="benzene", nrad=24, functional=LDA),
        # the DFT side of an iteration at 900 functions and 180 + 180 orbitals
        dict(name="c60_dft", kind="dft", system="c60", nrad=2, functional=SCAN),
        # GETVLXC alone on the caller's device buffers, the smallest call
        dict(name="getvlxc_pbe", kind="xc", npts=20_011, functional=PBE),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cycle", "cycle", "cycle", "cycle", "batch", "chunk", "grad", "dft", "xc"])
    prec = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "xc":
        return dict(kind="xc", npts=_log(rng, 1000, 1_000_000), functional=rng.choice([LDA, PBE]))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(2, 7), max_carbons=rng.randint(2, 4), nrad=rng.randint(6, 11),
                    functional=LDA, precision=prec)
    if kind == "chunk":
        return dict(kind="chunk", system=rng.choice(["chain", "ring"]), ncarbon=rng.randint(3, 8),
                    nrad=rng.randint(8, 20), chunks=rng.randint(2, 4), functional=rng.choice([LDA, SCAN]), precision=prec)
    if kind in ("grad", "dft"):
        system = rng.choice(["water", "benzene", "chain"])
        c = dict(kind=kind, system=system, nrad=rng.randint(8, 24 if kind == "grad" else 16),
                 functional=rng.choice([LDA, PBE]))
        return c if system != "chain" else dict(c, ncarbon=rng.randint(1, 4))
    system = rng.choice(["water", "benzene", "chain", "ring", "synthetic"])
    c = dict(kind="cycle", system=system, functional=rng.choice([LDA, PBE, SCAN]), precision=prec, density="phi2")
    if system == "synthetic":
        natoms = rng.randint(6, 40)
        nbasis = int(12.8 * natoms)
        return dict(c, natoms=natoms, nbasis=nbasis, nfo=max(2, min(128, int(natoms * rng.uniform(1.0, 3.2)))),
                    nmsh=_log(rng, 4_000, 90_000), functional=rng.choice([LDA, PBE]),
                    density=rng.choice(["phi2", "phi2", "pairs"]) if natoms <= 20 else "phi2")
    if system == "water":
        return dict(c, nrad=rng.randint(6, 40))
    if system == "benzene":
        return dict(c, nrad=rng.randint(6, 24), functional=rng.choice([LDA, PBE]))
    return dict(c, ncarbon=rng.randint(3 if system == "ring" else 1, 6), nrad=rng.randint(6, 14))


# ---------------------------------------------------------------------------
# systems
# ---------------------------------------------------------------------------
def _system(case, seed):
    kind, f = case["system"], case["functional"]
    if kind == "synthetic":
        box = 12.0 * (case["natoms"] / 40) ** (1 / 3)
        s = W.synthetic(natoms=case["natoms"], nbasis=case["nbasis"], nmsh=6000, nfo=1, box_ang=box, seed=seed,
                        functional=f)
        rng = np.random.default_rng(seed + 1)
        psi = W.orthonormal_orbitals(s, case["nfo"], rng)
        s = dataclasses.replace(s, psi=psi, nwfs=(case["nfo"], 0), fods=[_fods(s, psi, rng)])
        n, side = case["nmsh"], box * W.BOHR_PER_ANG
        n1 = math.ceil(n ** (1 / 3) - 1e-9)
        idx = np.stack(np.meshgrid(*[np.arange(n1)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        rmsh = (idx + 0.5 + rng.uniform(-0.35, 0.35, idx.shape)) * (side / n1)
        wmsh = rng.uniform(0.5, 1.5, n)
        return dataclasses.replace(s, rmsh=rmsh, wmsh=wmsh * (side ** 3 / wmsh.sum()))
    if kind == "c60":
        return W.c60(seed=seed, nrad=case["nrad"], functional=f)
    if kind == "water":
        s, scale = W.water(seed=seed, nrad=6, functional=f, basis="default"), [0.7, 0.5, 0.5]
    elif kind == "benzene":
        s, scale = W.benzene(seed=seed, nrad=4, functional=f, basis="default"), [0.7] * 6 + [0.5] * 6
    else:
        nc = case["ncarbon"]
        s = W.alkane(nc, ring=kind == "ring", seed=seed, nrad=4, functional=f)
        scale = [0.7] * nc + [0.5] * (s.natoms - nc)
    rmsh, wmsh = W.atom_centred_mesh(s.rat, nrad=case["nrad"], rscale=scale, seed=seed + 1)
    # the cut-off of small weights leaves a count that depends on the seed: keep a fixed one
    n = min(len(wmsh), _points(s.natoms, case["nrad"]))
    keep = np.sort(np.random.default_rng(seed + 2).permutation(len(wmsh))[:n])
    return dataclasses.replace(s, rmsh=np.ascontiguousarray(rmsh[keep]), wmsh=wmsh[keep] * (len(wmsh) / n))


def _fods(s, psi, rng):
    """One FOD per orbital near the atoms: of many random positions those whose normalised orbital
    values (the rows of the Fermi transformation) are the most independent, one after another."""
    cand = np.repeat(s.rat, math.ceil(6 * len(psi) / s.natoms), axis=0)
    cand = cand + rng.normal(0, 0.6, cand.shape)
    t = W.basis_values(s, cand) @ psi.T
    t /= np.linalg.norm(t, axis=1)[:, None]
    picked = []
    for _ in range(len(psi)):
        left = (t * t).sum(1)
        left[picked] = -1.0
        picked.append(int(np.argmax(left)))
        q = t[picked[-1]] / np.linalg.norm(t[picked[-1]])
        t -= np.outer(t @ q, q)
    return cand[picked]


def _points(natoms, nrad):
    return int(0.9 * natoms * nrad * 146)


def _fo_density(n, seed):
    """RHOG (10, n) of an FO-like density, the square of three Gaussians, with its derivatives."""
    g = torch.Generator().manual_seed(seed)
    r = (torch.randn(n, 3, generator=g, dtype=torch.float64) * 2.5).cuda()
    cen = (torch.randn(3, 3, generator=g, dtype=torch.float64) * 0.8).cuda()
    alp = torch.rand(3, generator=g, dtype=torch.float64).cuda() * 2.0 + 0.15
    cof = torch.rand(3, generator=g, dtype=torch.float64).cuda() + 0.2
    d = r[:, None, :] - cen
    e = cof * torch.exp(-alp * (d * d).sum(-1))
    phi = e.sum(1)
    g1 = -2 * (alp[None, :, None] * e[..., None] * d).sum(1)
    rho = torch.empty(10, n, dtype=torch.float64, device="cuda")
    rho[0] = phi * phi
    rho[1:4] = 2 * phi * g1.T
    for q, (i, j) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
        h = (e * (4 * alp ** 2 * d[..., i] * d[..., j] - (2 * alp if i == j else 0 * alp))).sum(1)
        rho[4 + q] = 2 * (g1[:, i] * g1[:, j] + phi * h)
    w = (torch.rand(n, generator=g, dtype=torch.float64) + 0.5).cuda() * (2.0 / n)
    return rho, w


def _molecules(case):
    """The chains and rings of a batch; they depend on the case alone, so that each seed asks for the same work."""
    out = []
    for i in range(case["count"]):
        ring = i % 2 == 1 and case["max_carbons"] >= 3
        nc = 3 + i % (case["max_carbons"] - 2) if ring else 1 + i % case["max_carbons"]
        out.append(dict(system="ring" if ring else "chain", ncarbon=nc, nrad=case["nrad"] - i % 3,
                        functional=case["functional"]))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "xc":
        ctx = S.FlosicSIC()
        ctx.set_geometry(W.small_synthetic(functional=case["functional"]))
        rho, w = _fo_density(case["npts"], seed)
        v = torch.empty(2 * case["npts"], dtype=torch.float64, device="cuda")
        return dict(kind=kind, ctx=ctx, rho=rho, w=w, v=v, n=case["npts"])
    if kind == "batch":
        mols = [_system(m, seed + 10 * i) for i, m in enumerate(_molecules(case))]
        return dict(kind=kind, batch=Batch(mols, precision=case["precision"]))
    sysm = _system(case, seed)
    ctx = S.FlosicSIC()
    if kind == "chunk":
        ctx.set_shard(0, case["chunks"])
    ctx.set_geometry(sysm)
    ctx.set_precision(case.get("precision", "fp64"))
    ctx.set_density_mode(case.get("density", "phi2"))
    st = dict(kind=kind, ctx=ctx, sysm=sysm)
    if kind != "cycle":
        ctx.set_orbitals(sysm.psi, sysm.nwfs, sysm.fods)
    if kind == "chunk":
        st["part"] = torch.zeros(ctx.partial_size(), dtype=torch.float64, device="cuda")
        st["chunks"] = case["chunks"]
    if kind == "grad":
        ctx.cycle()
    return st


def run(st):
    kind = st["kind"]
    if kind == "xc":
        n, v = st["n"], st["v"]
        ergs = st["ctx"].getvlxc_device(n, st["rho"].data_ptr(), n, st["w"].data_ptr(), v.data_ptr())
        return dict(up=v[:n], down=v[n:], ergs=ergs)
    if kind == "batch":
        return st["batch"].cycle()
    ctx, sysm = st["ctx"], st["sysm"]
    if kind == "cycle":  # an SCF iteration hands over its new orbitals and takes the SIC block's results
        ctx.set_orbitals(sysm.psi, sysm.nwfs, sysm.fods)
        return ctx.cycle()
    if kind == "chunk":  # one pass of shard.chunked_cycle
        ctx.set_orbitals(sysm.psi, sysm.nwfs, sysm.fods)
        ctx.cycle_partial(st["part"].data_ptr())
        return st["part"]
    if kind == "grad":
        spins = range(1, sysm.nspn + 1)
        return dict(adjoint=[ctx.adjoint(s) for s in spins], fod=[ctx.adjoint_fod(s) for s in spins],
                    dersic=ctx.siclag_der(), ham=[ctx.sicham(s) for s in spins])
    rhog, phig = ctx.densold(10)
    return dict(rho=rhog[:, 0], grad=rhog[:, 1:4], hess=rhog[:, 4:], phig=phig, coulomb=ctx.coupot1())


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
# Per FO and mesh point, the reference's POISSON1 work in these systems as the
# library counts it: near Gaussian-pair evaluations (92 flops each) and kept
# multipole terms (2 flops each).  It hardly depends on the mesh's density.
def _poisson(system, n):
    """Both counts; n: carbon atoms of a chain or ring, atoms of the synthetic system."""
    return dict(water=(144, 600), benzene=(1412, 11300), c60=(12500, 131000), chain=(165 * n ** 1.25, 944 * n ** 1.48),
                ring=(74 * n ** 1.63, 422 * n ** 1.85), synthetic=(1433 * (n / 40) ** 1.9, 25200 * (n / 40) ** 1.28))[system]


def _shape(case):
    """(mesh points, basis functions, FOs of both spins, near, kept terms)"""
    kind = case["system"]
    if kind == "synthetic":
        return (case["nmsh"], case["nbasis"], case["nfo"]) + _poisson(kind, case["natoms"])
    nc = case.get("ncarbon", 0)
    nh = 2 * nc + (2 if kind == "chain" else 0)
    nat, nb, nfo = dict(water=(3, 73, 10), benzene=(12, 324, 42), c60=(60, 900, 360)).get(
        kind, (nc + nh, 15 * nc + 5 * nh, 6 * nc + nh))
    p = nat * case["nrad"] * 146 if kind == "c60" else _points(nat, case["nrad"])
    return (p, nb, nfo) + _poisson(kind, nc)


def work(case):
    kind = case["kind"]
    if kind == "xc":
        n = case["npts"]
        ch = 1 if case["functional"] == LDA else 10
        return dict(bytes=8 * n * (ch + 1 + 2), flops=(100 if ch == 1 else 400) * n)
    if kind == "batch":
        each = [work(dict(m, kind="cycle")) for m in _molecules(case)]
        return dict(bytes=sum(w["bytes"] for w in each), flops=sum(w["flops"] for w in each))
    p, nb, nfo, near, terms = _shape(case)
    nch = {LDA: 1, PBE: 10, SCAN: 4}[case["functional"]]
    if kind == "grad":  # basis values against Y: adjoint, DERSIC (3 gradient channels), the two halves of SICHAM
        ch = 4 if case["functional"] == SCAN else 1
        return dict(bytes=8 * p * (4 + 2 * nfo), flops=2 * p * nb * nfo * (2 * ch + 3 + 2))
    if kind == "dft":   # orbital values in 10 channels; one density's Coulomb potential
        return dict(bytes=8 * p * (4 + 2 * 11 + 1), flops=2 * p * nb * nfo * nch + p * (92 * near + 2 * terms))
    if kind == "chunk":
        p //= case["chunks"]
    flops = p * nfo * (92 * near + 2 * terms) + 2 * p * nb * nfo * nch + 2 * p * nfo * nfo + 400 * p * nfo
    if case.get("density") == "pairs":
        flops += p * nfo * near * 2 * (155 if nch == 10 else 35)
    return dict(bytes=8 * (4 * p + nb * nfo + nfo * nfo), flops=flops)


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _xc_exact(case, seed):
    """The functional of a fully polarised density and its functional derivative
    dF/dn - div dF/d(grad n), by automatic differentiation."""
    rho, w = (t.cpu() for t in _fo_density(case["npts"], seed))
    gga = case["functional"] == PBE
    n = rho[0].clone().requires_grad_()
    gv = rho[1:4].clone().requires_grad_()
    third = 1.0 / 3.0
    fx = -0.75 * (3 / math.pi) ** third * (2 * n) ** third        # per particle, of the doubled density
    rs = (3 / (4 * math.pi * n)) ** third
    rt = rs.sqrt()
    q1 = 2 * 0.01554535 * rt * (14.1189 + rt * (6.1977 + rt * (3.3662 + rt * 0.62517)))
    ec = -2 * 0.01554535 * (1 + 0.20548 * rs) * torch.log1p(1 / q1)
    parts = [n * fx, None, n * ec, None]
    if gga:
        g2 = (gv * gv).sum(0)
        s2 = 4 * g2 / (4 * (3 * math.pi ** 2) ** (2 * third) * (2 * n) ** (8 * third))
        kap, mu = 0.804, 0.2195149727645171
        parts[1] = n * fx * (kap - kap / (1 + mu / kap * s2))
        gam, bet = (1 - math.log(2)) / math.pi ** 2, 0.06672455060314922
        phi = 2 ** (-third)
        ks2 = 4 * (3 * math.pi ** 2 * n) ** third / math.pi
        t2 = g2 / (4 * phi ** 2 * ks2 * n * n)
        a = bet / gam / torch.expm1(-ec / (gam * phi ** 3))
        parts[3] = n * gam * phi ** 3 * torch.log1p(bet / gam * t2 * (1 + a * t2) / (1 + a * t2 + (a * t2) ** 2))
    tot = sum(p for p in parts if p is not None)
    if gga:
        fn, fg = torch.autograd.grad(tot.sum(), (n, gv), create_graph=True)
        v = fn.detach().clone()
        hess = {(0, 0): 4, (1, 1): 5, (2, 2): 6, (0, 1): 7, (0, 2): 8, (1, 2): 9}
        for i in range(3):
            dn, dg = torch.autograd.grad(fg[i].sum(), (n, gv), retain_graph=True)
            v -= dn * rho[1 + i]
            for j in range(3):
                v -= dg[j] * rho[hess[min(i, j), max(i, j)]]
    else:
        v = torch.autograd.grad(tot.sum(), n)[0]
    keep = rho[0] >= 1e-20   # the functional is evaluated above this density
    ergs = [float((torch.where(keep, p.detach(), 0.0) * w).sum()) if p is not None else 0.0 for p in parts]
    # ERGXL, ERGXN, ERGCL, ERGCN; without gradients the PW91 non-local parts vanish.  The unoccupied
    # spin's potential is regularised by the functional's own cut-offs and has no plain value.
    return dict(up=torch.where(keep, v, 0.0).numpy(), down=None, ergs=np.array(ergs))


def _dft_exact(case, seed):
    """Density, gradient and sum |grad psi|^2 of the occupied orbitals (no value for the
    Coulomb potential, which the reference defines with its multipole far field)."""
    s = _system(case, seed)
    pw = [[(0, 0, 0)], [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
          [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)]]
    out = []
    psi = torch.from_numpy(np.where(np.abs(s.psi) > 1e-10, s.psi, 0.0))
    for c0 in range(0, s.nmsh, 20000):
        x = torch.from_numpy(s.rmsh[c0:c0 + 20000])
        cols = [[], [], [], []]
        for a in range(s.natoms):
            t = int(s.atom_type[a])
            nb = int(s.n_bare[t])
            alp = torch.from_numpy(s.bfalp[t, :nb])
            d = x - torch.from_numpy(s.rat[a])
            arg = (d * d).sum(1)[:, None] * alp
            e = torch.where(arg < 40.0, torch.exp(-arg), 0.0)
            for l in range(3):
                con = torch.from_numpy(s.bfcon[t, l, :int(s.n_con[t, l]), :nb]).T.contiguous()
                r0, r1 = e @ con, (e * (-2 * alp)) @ con
                for p in pw[l]:
                    mono = [d[:, i] ** p[i] for i in range(3)]
                    ang = mono[0] * mono[1] * mono[2]
                    cols[0].append(ang[:, None] * r0)
                    for i in range(3):
                        da = p[i] * d[:, i] ** max(p[i] - 1, 0) * mono[(i + 1) % 3] * mono[(i + 2) % 3]
                        cols[1 + i].append(da[:, None] * r0 + (ang * d[:, i])[:, None] * r1)
        v = [torch.cat(c, 1) @ psi.T for c in cols]
        both = []
        for sp in range(2):
            q = [t[:, sp * s.nwfs[0]:sp * s.nwfs[0] + s.nwfs[sp]] for t in v]
            both.append(torch.stack([(q[0] ** 2).sum(1)] + [2 * (q[0] * q[i]).sum(1) for i in (1, 2, 3)]
                                    + [sum((q[i] ** 2).sum(1) for i in (1, 2, 3))]))
        out.append(torch.stack(both))
    r = torch.cat(out, 2).numpy()
    return dict(rho=r[:, 0], grad=r[:, 1:4], hess=None, phig=r[:, 4], coulomb=None)


def exact(case, seed):
    if case["kind"] == "xc":
        return _xc_exact(case, seed)
    if case["kind"] == "dft":
        return _dft_exact(case, seed)
    # The other paths contain the FOs' Coulomb potentials, which are not the integrals themselves: the
    # reference's batches, cut-off spheres and L <= 6 multipoles define them to a part in a million.
    return None
