"""The work that is timed: H|psi>, its batched, spinor, adjoint and drop-in forms and the eigensolver.

A case is one call that an electronic-structure program makes through this package's public entry
points, with the crystal, plane-wave basis, potential and projectors that the call needs:

* ``hk``      H|psi> of one k-point on device blocks (``Context.hk_psi``), in the three precision forms;
* ``kbatch``  H|psi> of the k-points of one crystal in one call (``KBatch.hk_psi``);
* ``spin``    H|psi> of two-component spinors with a non-collinear potential (``Context.hk_psi_spin``);
* ``adjoint`` the backward direction: density, local and Kleinman-Bylander force terms (``HFSystem``);
* ``dropin``  the reference's own call with host arrays (``hk_psi_c16``);
* ``eig``     a whole block eigensolve (``eigensolve``).

Crystals come from ``configs`` (silicon and zincblende supercells) or, for the ``box`` cells, are
orthorhombic cells of randomly placed atoms at silicon's density whose FFT box has any of the
reference's sizes per direction. The case fixes the k-points, and with them the plane-wave counts; a
seed fixes the atomic displacements and the wavefunctions.
"""
import math

import numpy as np
import torch

from cpw2000_b200 import configs, crystal, pseudo
from cpw2000_b200 import ditsp as E
from cpw2000_b200 import forces as F
from cpw2000_b200 import hk_psi as H
from cpw2000_b200 import kbatch as KB

PRECISION = {"fp64": H.FP64, "mixed": H.MIXED, "mixed_tc": H.MIXED_TC}
DELQ, NQ = 0.01, 4000
BOHR_PER_POINT = 20.52 / 96            # mesh spacing of the silicon supercells (96 points, 144 points)
ATOM_VOLUME = 10.26 ** 3 / 8           # bohr^3 per atom of silicon


def listed():
    return [
        # the smallest call: the primitive cell of an SCF loop over k-points, a handful of bands
        dict(name="hk_si2_fp64", path="hk", cell="si2", bands=8, precision="fp64"),
        # an ordinary supercell, all its bands at once, as the drop-in computes it
        dict(name="hk_si64_fp64", path="hk", cell="si64", bands=160, precision="fp64"),
        # the same in the mixed form meant for production
        dict(name="hk_si64_tc", path="hk", cell="si64", bands=160, precision="mixed_tc"),
        # the benchmark's cell: the largest basis, box, projector and band counts
        dict(name="hk_si216_fp64", path="hk", cell="si216", bands=480, precision="fp64"),
        dict(name="hk_si216_tc", path="hk", cell="si216", bands=480, precision="mixed_tc"),
        # the unconverged remainder of a block late in a solve, in a cell whose three box lengths
        # differ and are none of the cubic benchmark sizes
        dict(name="hk_ragged_fp64", path="hk", cell="box", n1=72, n2=80, n3=108, bands=37, precision="fp64"),
        # a slab-like cell in the mixed form with FP64 projector products
        dict(name="hk_ragged_mixed", path="hk", cell="box", n1=64, n2=50, n3=128, bands=91, precision="mixed"),
        # every k-point of a small crystal in one call
        dict(name="kbatch_si8_tc", path="kbatch", nk=64, bands=40, uneven=False, precision="mixed_tc"),
        # spin-orbit: spinors in a four-component potential with spinor projectors
        dict(name="spin4_si8_fp64", path="spin", nsp=4, bands=80, precision="fp64"),
        # forces of a two-species supercell from its occupied bands
        dict(name="adjoint_zb64", path="adjoint", cell="zb64", bands=128),
        # the reference's call with host arrays: copies in, H|psi>, copies out
        dict(name="dropin_si64", path="dropin", cell="si64", bands=160),
        # one k-point's whole eigensolve from the small dense start to convergence
        dict(name="eig_si8_fp64", path="eig", bands=40, ecut=20.0),
    ]


# FFT lengths the reference's size_fft returns for cells of this kind
BOXES = (24, 32, 36, 40, 48, 50, 54, 64, 72, 80, 96, 100, 108, 128, 144)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("hk", "hk", "hk", "hk", "kbatch", "spin", "adjoint", "dropin", "eig"))
    if kind == "kbatch":
        return dict(path="kbatch", nk=_log_int(rng, 2, 64), bands=rng.randint(9, 40), uneven=rng.random() < 0.7,
                    precision=rng.choice(tuple(PRECISION)))
    if kind == "spin":
        return dict(path="spin", nsp=rng.choice((1, 2, 4, 4)), bands=_log_int(rng, 4, 80),
                    precision=rng.choice(("fp64", "fp64", "mixed")))
    if kind == "eig":
        return dict(path="eig", bands=rng.randint(12, 40), ecut=round(rng.uniform(10.0, 20.0), 2))
    most = 108 if kind in ("adjoint", "dropin") else 144
    while True:
        # lengths over the whole range, the shortest at least a third of the longest
        n = [rng.choice([b for b in BOXES if b <= most]) for _ in range(3)]
        if max(n) <= 3 * min(n):
            break
    # bands between a few and the occupied bands of the cell with a quarter more
    natom = _natom(n)
    bands = _log_int(rng, 3, max(4, min(480, int(2.5 * natom))))
    case = dict(path=kind, cell="box", n1=n[0], n2=n[1], n3=n[2], bands=bands)
    if kind == "hk":
        case["precision"] = rng.choice(("fp64", "fp64", "mixed", "mixed_tc", "mixed_tc"))
    return case


# ---------------------------------------------------------------- crystals and their inputs

def _natom(n):
    return max(1, round(n[0] * n[1] * n[2] * BOHR_PER_POINT ** 3 / ATOM_VOLUME))


def _workload(case, seed):
    """The crystal and its k-points (configs.Workload)."""
    rng = np.random.default_rng(seed)
    if case["path"] in ("kbatch", "spin", "eig"):
        w = configs.si8_cubic_kbatch(nk=case.get("nk", 1))
        w.ecut = case.get("ecut", w.ecut)
        return _displaced(w, rng)
    cell = case["cell"]
    if cell == "si2":
        w = configs.si2_fcc()
        w.kpoints = w.kpoints[3:4]
        return _displaced(w, rng)
    if cell in ("si64", "zb64", "si216"):
        return {"si64": configs.si64_cubic, "zb64": configs.zb64_cubic, "si216": configs.si216_cubic}[cell](seed)
    n = (case["n1"], case["n2"], case["n3"])
    a = np.array(n) * BOHR_PER_POINT
    sp = pseudo.Species(v0=4.0, sigma=0.8, ekb=(2.0, -1.5), sigma_kb=1.0, rat=rng.uniform(0, 1, (_natom(n), 3)))
    return configs.Workload("box", np.diag(a * a), [sp], 16.0, n, np.array([[0.17, -0.31, 0.42]]), case["bands"])


def _displaced(w, rng):
    """The cell with its atoms moved by about 0.02 bohr, as in the supercells."""
    for sp in w.species:
        sp.rat = sp.rat + rng.normal(0.0, 0.02 / math.sqrt(w.adot[0, 0]), sp.rat.shape)
    return w


def _crystal(w):
    """What all k-points of a crystal share: G vectors, potential on the box, radial tables."""
    _, bvec = crystal.adot_to_avec(w.adot)
    kmax = max(float(np.linalg.norm(bvec @ k)) for k in w.kpoints)
    kgv = crystal.gspace(w.adot, math.sqrt(2 * w.ecut) + kmax + 0.5)
    vscr, veffr1 = pseudo.local_potential_box(w.species, w.adot, w.box, w.idpad)
    vkb, nkb = pseudo.kb_tables(w.species, DELQ, NQ)
    n1, n2, n3 = w.box
    kmscr = np.array([(n1 - 1) // 2, (n2 - 1) // 2, (n3 - 1) // 2, n1, n2, n3, w.ident], dtype=np.int32)
    return dict(kgv=kgv, ng=int(kgv.shape[1]), vscr=vscr, veffr1=veffr1, vkb=vkb, nkb=nkb, kmscr=kmscr)


def _basis(w, shared, ik=0):
    """The arrays of one k-point, without the projectors."""
    rk = np.asarray(w.kpoints[ik], dtype=np.float64)
    mtxd, isort, qmod, ekpg = crystal.hamilt_struct(w.ecut, rk, shared["kgv"], w.adot)
    return dict(shared, mtxd=mtxd, isort=isort, qmod=qmod, ekpg=ekpg, rkpt=rk)


def _host_projectors(w, d):
    x, xnl = pseudo.proj_nl_kb(d["rkpt"], d["isort"], d["kgv"], w.species, d["vkb"], d["nkb"], w.adot, DELQ, NQ)
    return dict(d, anlga=np.asfortranarray(x), xnlkb=xnl, nanl=int(xnl.size))


def _context(w, d, precision):
    """A context with the k-point, the potential and the projectors built on the device."""
    ctx = H.Context(0, precision=precision)
    ctx.set_kpoint(d["mtxd"], d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    ctx.set_potential(d["vscr"])
    ctx.proj_nl_kb(d["rkpt"], w.species, d["vkb"], d["nkb"], w.adot, DELQ, NQ)
    return ctx


def _waves(ekpg, nb, seed, rows_per_wave=1):
    """(rows, nb) column-major wavefunctions: random phases, amplitudes that fall with the kinetic
    energy as those of smooth bands do, norm 1."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    ek = torch.from_numpy(np.repeat(np.asarray(ekpg), rows_per_wave)).cuda()
    x = torch.randn((nb, ek.numel()), dtype=torch.complex128, device="cuda", generator=g) / (1 + ek) ** 2
    return (x / torch.linalg.vector_norm(x, dim=1, keepdim=True)).t()


def _spin_inputs(w, d, case, seed):
    """Four potential components (the magnetic ones a tenth of the scalar one) and spinor projectors:
    every scalar projector with two orthogonal spin directions."""
    rng = np.random.default_rng(seed + 1)
    nsp = case["nsp"]
    v = np.asfortranarray(np.stack([d["vscr"]] + [0.1 * rng.uniform(-1, 1) * np.roll(d["vscr"], 7 * j)
                                                  for j in range(1, nsp)], axis=1))
    x = d["anlga"]
    m, na = x.shape
    th = rng.uniform(0, math.pi, na)
    ph = np.exp(1j * rng.uniform(0, 2 * math.pi, na))
    a = np.zeros((2 * m, 2 * na), np.complex128, order="F")
    a[0::2, :na], a[1::2, :na] = x * np.cos(th / 2), x * (np.sin(th / 2) * ph)
    a[0::2, na:], a[1::2, na:] = x * (-np.sin(th / 2) * ph.conj()), x * np.cos(th / 2)
    return v, a, np.concatenate([d["xnlkb"], 0.8 * d["xnlkb"]])


def _occupations(case):
    nb = case["bands"]
    return np.where(np.arange(nb) < 0.9 * nb, 2.0, 0.5)


def _pinned(shape):
    return torch.zeros(shape, dtype=torch.complex128, pin_memory=True).numpy().T


def _inputs(case, seed):
    """(workload, arrays) of the cases with one k-point."""
    w = _workload(case, seed)
    return w, _basis(w, _crystal(w))


# ---------------------------------------------------------------- prepare and run

def prepare(case, seed):
    path, nb = case["path"], case["bands"]
    if path == "hk":
        w, d = _inputs(case, seed)
        psi = _waves(d["ekpg"], nb, seed)
        return dict(path=path, ctx=_context(w, d, PRECISION[case["precision"]]), psi=psi,
                    hpsi=torch.zeros_like(psi))
    if path == "kbatch":
        w = _workload(case, seed)
        shared = _crystal(w)
        ks = [_host_projectors(w, _basis(w, shared, k)) for k in range(case["nk"])]
        ctx = H.Context(0, precision=PRECISION[case["precision"]]).setup(ks[0])
        nbs = _band_counts(case)
        flat = [torch.zeros(sum(n * d["mtxd"] for n, d in zip(nbs, ks)), dtype=torch.complex128, device="cuda")
                for _ in range(2)]
        blocks, at = ([], []), 0
        for k, (n, d) in enumerate(zip(nbs, ks)):
            size = n * d["mtxd"]
            for buf, out in zip(flat, blocks):
                out.append(buf[at:at + size].view(n, d["mtxd"]).t())
            blocks[0][k].copy_(_waves(d["ekpg"], n, seed * 1000 + k))
            at += size
        return dict(path=path, ctx=ctx, kb=KB.KBatch(ctx, ks), psi=blocks[0], hpsi=blocks[1], out=flat[1])
    if path == "spin":
        w, d = _inputs(case, seed)
        d = _host_projectors(w, d)
        v, a, x = _spin_inputs(w, d, case, seed)
        ctx = H.Context(0, precision=PRECISION[case["precision"]])
        ctx.set_kpoint(d["mtxd"], d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
        ctx.set_potential_spin(v, case["nsp"])
        ctx.set_projectors_spin(a, x)
        psi = _waves(d["ekpg"], nb, seed, 2)
        return dict(path=path, ctx=ctx, psi=psi, hpsi=torch.zeros_like(psi))
    if path == "adjoint":
        w, d = _inputs(case, seed)
        s = F.HFSystem(w, d, _waves(d["ekpg"], nb, seed), _occupations(case))
        s.ctx.proj_nl_kb(d["rkpt"], w.species, d["vkb"], d["nkb"], w.adot, DELQ, NQ)
        return dict(path=path, system=s, tau=s.tau0().numpy(), points=math.prod(s.box))
    if path == "dropin":
        # the crystal of an SCF program stays; its wavefunctions change from call to call
        w, d = _inputs(case, 0)
        d = _host_projectors(w, d)
        psi, hpsi = _pinned((nb, d["mtxd"])), _pinned((nb, d["mtxd"]))
        psi[:] = _waves(d["ekpg"], nb, seed).cpu().numpy()
        return dict(path=path, d=d, nb=nb, psi=psi, hpsi=hpsi)
    w = _workload(case, seed)
    d = configs.kpoint_inputs(w, 0, nbands=nb, with_hamsm=True)
    ctx = H.Context(0).setup(d)
    psi = torch.zeros((nb, d["mtxd"]), dtype=torch.complex128, device="cuda").t()
    return dict(path=path, ctx=ctx, d=d, nb=nb, psi=psi, hpsi=torch.zeros_like(psi))


def _band_counts(case):
    return [max(1, case["bands"] - (3 * k) % 7) if case["uneven"] else case["bands"] for k in range(case["nk"])]


def run(state):
    path = state["path"]
    if path == "hk":
        return state["ctx"].hk_psi(state["psi"], state["hpsi"])
    if path == "kbatch":
        state["kb"].hk_psi(state["psi"], state["hpsi"])
        return state["out"]
    if path == "spin":
        state["ctx"].hk_psi_spin(state["psi"], state["hpsi"])
        return state["hpsi"]
    if path == "adjoint":
        s = state["system"]
        rho = s.density()
        return dict(density=rho, local=s.structure_grad(rho / state["points"], state["tau"]), kb=s.nl_grad())
    if path == "dropin":
        d, nb, m = state["d"], state["nb"], state["d"]["mtxd"]
        hpsi, _ = H.hk_psi_c16(m, nb, state["psi"], state["hpsi"], False, d["ng"], d["kgv"], d["ekpg"], d["isort"],
                               d["vscr"], d["kmscr"], d["anlga"], d["xnlkb"], d["nanl"], m, nb, d["nanl"], d["ng"],
                               d["vscr"].size)
        return hpsi
    d, nb = state["d"], state["nb"]
    r = E.eigensolve(state["ctx"], state["psi"], state["hpsi"], nb, d["mtxds"], d["hamsm"], d["hdiag"], epspsi=1e-5,
                     icmax=60)
    return dict(ei=r["ei"], psi=state["psi"])


# ---------------------------------------------------------------- work

def _sizes(case):
    """(plane waves, projectors, box, kept half-widths) of one k-point, from the cell alone."""
    path = case["path"]
    if path in ("kbatch", "spin", "eig"):
        n, a, na, ecut = (40, 40, 40), (10.26,) * 3, 32, case.get("ecut", 20.0)
    elif case["cell"] == "box":
        n = (case["n1"], case["n2"], case["n3"])
        a, na, ecut = [v * BOHR_PER_POINT for v in n], 4 * _natom(n), 16.0
    else:
        size, length, atoms = {"si2": (32, 7.255, 2), "si64": (96, 20.52, 64), "zb64": (96, 21.0, 64),
                               "si216": (144, 30.78, 216)}[case["cell"]]
        n, a, na, ecut = (size,) * 3, (length,) * 3, 4 * atoms, 16.0
    g = math.sqrt(2 * ecut)
    vol = 10.26 ** 3 / 4 if case.get("cell") == "si2" else math.prod(a)
    m = vol * g ** 3 / (6 * math.pi ** 2)
    kd = [g * v / (2 * math.pi) for v in a]
    return m, na, n, kd


def _fft_flops(n, kd):
    """One pruned transform between the sphere and the box: x lines on the kept rows of the kept
    planes, y lines on the kept planes, z lines on every column."""
    n1, n2, n3 = n
    y, z = 2 * kd[1] + 1, 2 * kd[2] + 1

    def line(k):
        return 5 * k * math.log2(k)

    return y * z * line(n1) + n1 * z * line(n2) + n1 * n2 * line(n3)


def work(case):
    """Each input read once, each output written once; the pruned transforms and the projector products."""
    path, nb = case["path"], case["bands"]
    m, na, n, kd = _sizes(case)
    box = math.prod(n)
    h_flops = 2 * _fft_flops(n, kd) + 16 * m * na            # one band of H|psi>
    if path == "kbatch":
        bands = sum(_band_counts(case))
        return dict(bytes=32 * m * bands + case["nk"] * 16 * m * na + 8 * box, flops=bands * h_flops)
    if path == "spin":
        flops = nb * (2 * 2 * _fft_flops(n, kd) + 16 * 2 * m * 2 * na)
        return dict(bytes=64 * m * nb + 16 * 2 * m * 2 * na + 8 * box * case["nsp"], flops=flops)
    if path == "adjoint":
        # density, one transform of the whole box, structure factors, P = X^H psi and X^H (G psi)
        flops = nb * (_fft_flops(n, kd) + 3 * box) + 15 * box * math.log2(box) / 3 + 20 * box * na / 4 + 32 * m * na * nb
        return dict(bytes=16 * m * nb + 16 * m * na + 8 * 3 * box, flops=flops)
    if path == "eig":
        # about ten applications of H to every band, as many block orthogonalisations and rotations
        return dict(bytes=32 * m * nb + 16 * m * na + 8 * box, flops=10 * nb * (h_flops + 8 * m * 3 * nb))
    return dict(bytes=32 * m * nb + 16 * m * na + 8 * box, flops=nb * h_flops)


# ---------------------------------------------------------------- exact: plain torch in 64 bits

def _solid_harmonics(q):
    """(l, value) of the s and p projectors in the order of the columns: 1; y, z, x."""
    return [(0, torch.ones_like(q[0])), (1, q[1]), (1, q[2]), (1, q[0])]


def _exact_projectors(w, d):
    """X (mtxd, nanl) and its signs: phase, solid harmonic and interpolated radial table."""
    _, bvec = crystal.adot_to_avec(w.adot)
    vcell = math.sqrt(np.linalg.det(w.adot))
    g = torch.from_numpy(d["kgv"][:, d["isort"] - 1].astype(np.float64)).cuda()
    q = torch.from_numpy(bvec).cuda() @ (g + torch.from_numpy(d["rkpt"]).cuda()[:, None])
    xq = torch.sqrt((q * q).sum(0)) / DELQ
    ni = torch.round(xq).long().clamp(min=0)
    xi = xq - ni
    cols, sign = [], []
    for t, sp in enumerate(w.species):
        phase = torch.exp(-2j * math.pi * (torch.from_numpy(sp.rat).cuda() @ g))
        for l, ylm in _solid_harmonics(q):
            tab = torch.from_numpy(np.ascontiguousarray(d["vkb"][t, l])).cuda()
            v0, vp, vm = tab[ni + 2], tab[ni + 3], tab[ni + 1]
            radial = v0 * (1 + xi) * (1 - xi) + 0.5 * (vp * (1 + xi) - vm * (1 - xi)) * xi
            cols.append((phase * (ylm * radial / math.sqrt(vcell) * 1j ** l)).t())
            sign += [float(d["nkb"][t, l])] * sp.natom
    return torch.cat(cols, 1), torch.tensor(sign, dtype=torch.float64, device="cuda")


def _box_index(d):
    """Position of every plane wave in the flattened (n3, n2, n1) box."""
    n1, n2, n3 = (int(v) for v in d["kmscr"][3:6])
    g = torch.from_numpy(d["kgv"][:, d["isort"] - 1].astype(np.int64)).cuda()
    return (g[2] % n3) * (n2 * n1) + (g[1] % n2) * n1 + g[0] % n1


def _to_mesh(psi, d):
    """psi(r) of a few bands, (bands, n3, n2, n1), unscaled."""
    n1, n2, n3 = (int(v) for v in d["kmscr"][3:6])
    box = torch.zeros((psi.shape[1], n1 * n2 * n3), dtype=torch.complex128, device="cuda")
    box[:, _box_index(d)] = psi.t()
    return torch.fft.ifftn(box.view(-1, n3, n2, n1), dim=(1, 2, 3)) * (n1 * n2 * n3)


def _to_waves(box, d):
    n = math.prod(box.shape[1:])
    return (torch.fft.fftn(box, dim=(1, 2, 3)).reshape(box.shape[0], -1)[:, _box_index(d)] / n).t()


def _mesh(v, d):
    n1, n2, n3 = (int(x) for x in d["kmscr"][3:6])
    return torch.from_numpy(np.ascontiguousarray(v).reshape(n3, n2, int(d["kmscr"][6]))[:, :, :n1].copy()).cuda()


def _chunks(nb, d, most=2 ** 26):
    step = max(1, most // math.prod(int(v) for v in d["kmscr"][3:6]))
    return [slice(b, min(nb, b + step)) for b in range(0, nb, step)]


def _exact_h(psi, d, x, sign):
    v = _mesh(d["vscr"], d)
    out = torch.from_numpy(d["ekpg"]).cuda()[:, None] * psi + x @ (sign[:, None] * (x.conj().t() @ psi))
    for b in _chunks(psi.shape[1], d):
        out[:, b] += _to_waves(_to_mesh(psi[:, b], d) * v, d)
    return out


def exact(case, seed):
    path, nb = case["path"], case["bands"]
    if path == "kbatch":
        w = _workload(case, seed)
        shared = _crystal(w)
        out = []
        for k, n in enumerate(_band_counts(case)):
            d = _basis(w, shared, k)
            out.append(_exact_h(_waves(d["ekpg"], n, seed * 1000 + k), d, *_exact_projectors(w, d)).t().reshape(-1))
        return torch.cat(out)
    if path == "eig":
        w, d = _inputs(case, seed)
        x, sign = _exact_projectors(w, d)
        n1, n2, n3 = (int(v) for v in d["kmscr"][3:6])
        vg = torch.fft.fftn(_mesh(d["vscr"], d)) / (n1 * n2 * n3)
        g = torch.from_numpy(d["kgv"][:, d["isort"] - 1].astype(np.int64)).cuda()
        h = (x * sign) @ x.conj().t() + torch.diag(torch.from_numpy(d["ekpg"]).cuda())
        dg = [(g[j][:, None] - g[j][None, :]) % n for j, n in enumerate((n1, n2, n3))]
        h += vg[dg[2], dg[1], dg[0]]
        return dict(ei=torch.linalg.eigvalsh(h)[:nb].cpu().numpy(), psi=None)
    w, d = _inputs(case, 0 if path == "dropin" else seed)
    if path == "spin":
        d = _host_projectors(w, d)
        v, a, xnl = _spin_inputs(w, d, case, seed)
        psi = _waves(d["ekpg"], nb, seed, 2)
        vs = [_mesh(v[:, j], d) for j in range(case["nsp"])] + [0.0] * (4 - case["nsp"])
        out = torch.from_numpy(np.repeat(d["ekpg"], 2)).cuda()[:, None] * psi
        a, xnl = torch.from_numpy(a).cuda(), torch.from_numpy(xnl).cuda()
        out += a @ (xnl[:, None] * (a.conj().t() @ psi))
        for b in _chunks(nb, d):
            u, s = _to_mesh(psi[0::2, b], d), _to_mesh(psi[1::2, b], d)
            out[0::2, b] += _to_waves((vs[0] + vs[1]) * u + (vs[2] - 1j * vs[3]) * s, d)
            out[1::2, b] += _to_waves((vs[0] - vs[1]) * s + (vs[2] + 1j * vs[3]) * u, d)
        return out
    psi = _waves(d["ekpg"], nb, seed)
    x, sign = _exact_projectors(w, d)
    if path == "adjoint":
        return _exact_adjoint(w, d, psi, torch.from_numpy(_occupations(case)).cuda(), x, sign)
    out = _exact_h(psi, d, x, sign)
    return out.cpu().numpy() if path == "dropin" else out


def _exact_adjoint(w, d, psi, f, x, sign):
    n1, n2, n3 = (int(v) for v in d["kmscr"][3:6])
    rho = torch.zeros((n3, n2, n1), dtype=torch.float64, device="cuda")
    for b in _chunks(psi.shape[1], d):
        rho += (f[b, None, None, None] * _to_mesh(psi[:, b], d).abs() ** 2).sum(0)
    # dE/dtau of sum_r rho V / N, V(G) = sum_a exp(-2 pi i G.tau_a) v_t(G)
    rg = torch.fft.fftn(rho) / (n1 * n2 * n3)
    vt = torch.from_numpy(pseudo.local_form_factors_box(w.species, w.adot, w.box)).cuda()
    m = [torch.from_numpy(np.fft.fftfreq(n, 1.0 / n)).cuda() for n in (n3, n2, n1)]
    local = []
    for t, sp in enumerate(w.species):
        c = vt[t] * rg.conj()
        for tau in sp.rat:
            ph = [torch.exp(-2j * math.pi * m[j] * float(tau[2 - j])) for j in range(3)]
            z = torch.einsum("abc,a,b,c->abc", c, ph[0], ph[1], ph[2])
            local.append([float((2 * math.pi * m[2 - j].view([-1 if k == 2 - j else 1 for k in range(3)]) * z.imag).sum())
                          for j in range(3)])
    # KB term: -4 pi sum_n f_n sum_a xnlkb Im(conj(P) X^H (G psi))
    g = torch.from_numpy(d["kgv"][:, d["isort"] - 1].astype(np.float64)).cuda()
    p = x.conj().t() @ psi
    atom = torch.from_numpy(pseudo.proj_atom_map(w.species, d["nkb"])).long().cuda()
    kb = torch.zeros((len(local), 3), dtype=torch.float64, device="cuda")
    for j in range(3):
        c = ((p.conj() * (x.conj().t() @ (g[j][:, None] * psi))).imag * f).sum(1)
        kb[:, j].index_add_(0, atom, -4 * math.pi * sign * c)
    return dict(density=rho, local=np.array(local), kb=kb.cpu().numpy())
