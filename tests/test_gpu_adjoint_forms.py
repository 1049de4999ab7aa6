"""The z stages of the density and of non-collinear spinors for every compiled line length, and the tiled
structure gradient, against numpy and the oracle.

Line lengths and half-widths as in the H|psi> line tests: just inside the outer quarters of the line
(compiled forms) and just beyond (run-time forms). Structure gradient: atom counts around the tile of 32,
several species of uneven size, boxes whose rows do not fill a chunk of 32, the longest rows.
All sides are FP64 transforms or sums of like length, phases of up to 128 turns (800 ulp = 1e-13 in the
reference): 1e-12 of the largest value; FP32 spinor stage 2e-5.
"""
import ctypes as C

import numpy as np
import pytest

from cpw2000_b200 import _lib
from cpw2000_b200 import hk_psi as H
from oracle import hk_psi as O
from tests.test_gpu_line_forms import SPLITS, _case, _limit

pytestmark = pytest.mark.gpu


def _kd3(n3, inside):
    kd = _limit(n3) - 1 if inside else _limit(n3)
    if kd > (n3 - 1) // 2:
        pytest.skip("the quarters cover the whole line")
    return kd


def _dev(cuda, a):
    import torch
    t = torch.empty_strided(a.shape, (1, a.shape[0]), dtype=torch.complex128, device=cuda)
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("n3", sorted(SPLITS))
@pytest.mark.parametrize("inside", [True, False])
def test_density(cuda, n3, inside):
    _density(cuda, (10, 9, n3), (2, 2, _kd3(n3, inside)), H.FP64)


@pytest.mark.parametrize("box,kd", [((40, 256, 16), (2, 54, 2)), ((144, 144, 16), (2, 34, 2))])
def test_density_wide_plane_of_a_mixed_context(cuda, box, kd):
    # a y tile of 40 columns fits the shared memory in FP32, one of 32 in FP64; one of 32 in FP32, one of 16 in FP64
    _density(cuda, box, kd, H.MIXED)


def _density(cuda, box, kd, prec):
    import torch
    n1, n2, n3 = box
    d, psi = _case(box, kd, 7, n3)
    occ = np.linspace(2.0, 0.3, 7)
    ctx = H.Context(0, precision=prec)
    ctx.set_kpoint(d["mtxd"], d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    x = _dev(cuda, psi)
    rho = torch.empty((n3, n2, n1), dtype=torch.float64, device=cuda)
    _lib.check(_lib.lib().cpw_b200_density_device(ctx.handle, 7, C.c_void_p(x.data_ptr()), d["mtxd"], _lib.dptr(occ),
                                                  C.c_void_p(rho.data_ptr()), None))
    g = d["kgv"] % np.array(box)[:, None]
    ref = np.zeros((n3, n2, n1))
    for n in range(7):
        b = np.zeros((n3, n2, n1), np.complex128)
        b[g[2], g[1], g[0]] = psi[:, n]
        ref += occ[n] * np.abs(np.fft.ifftn(b) * b.size) ** 2
    assert np.abs(rho.cpu().numpy() - ref).max() < 1e-12 * ref.max()
    ctx.close()


@pytest.mark.parametrize("prec,tol", [(H.FP64, 1e-12), (H.MIXED, 2e-5)])
@pytest.mark.parametrize("n3", sorted(SPLITS))
@pytest.mark.parametrize("inside", [True, False])
def test_noncollinear_stage(cuda, n3, inside, prec, tol):
    box = (10, 9, n3)
    d, _ = _case(box, (2, 2, _kd3(n3, inside)), 1, n3)
    m, rng = d["mtxd"], np.random.default_rng(n3)
    psi = rng.standard_normal((2 * m, 5)) + 1j * rng.standard_normal((2 * m, 5))
    v = np.asfortranarray(rng.standard_normal((d["vscr"].size, 4)))
    ctx = H.Context(0, precision=prec)
    ctx.set_kpoint(m, d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    ctx.set_potential_spin(v, 4)
    x, y = _dev(cuda, psi), _dev(cuda, psi)
    ctx.hk_psi_spin(x, y)
    ctx.synchronize()
    ref = O.hk_psi_spin_c16(m, 5, psi, d["ekpg"], d["isort"], v, d["kmscr"], d["kgv"], 4,
                            np.zeros((2 * m, 0), np.complex128), np.zeros(0))
    assert np.abs(y.cpu().numpy() - ref).max() < tol * np.abs(ref).max()
    ctx.close()


@pytest.mark.parametrize("box,counts", [((10, 9, 16), (1,)), ((12, 8, 20), (32, 1, 33)), ((9, 5, 18), (0, 5, 70)),
                                        ((20, 25, 24), (31,)), ((256, 3, 4), (3, 40))])
def test_structure_gradient(cuda, box, counts):
    import torch
    n1, n2, n3 = box
    d, _ = _case(box, (1, 1, 1), 1, 2)
    rng = np.random.default_rng(sum(counts))
    kind = rng.permutation(np.repeat(np.arange(len(counts)), counts)).astype(np.int32)
    tau = np.ascontiguousarray(rng.uniform(-1, 1, (kind.size, 3)))
    g, vt = rng.standard_normal((n3, n2, n1)), rng.standard_normal((len(counts), n3, n2, n1))
    ctx = H.Context(0)
    ctx.set_kpoint(d["mtxd"], d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    gd, vd = torch.from_numpy(g).to(cuda), torch.from_numpy(vt).to(cuda)
    out = np.zeros((kind.size, 3))
    _lib.check(_lib.lib().cpw_b200_structure_grad_device(ctx.handle, C.c_void_p(gd.data_ptr()), kind.size,
                                                         _lib.iptr(kind), _lib.dptr(tau), len(counts),
                                                         C.c_void_p(vd.data_ptr()), _lib.dptr(out), None))
    m = [np.where(np.arange(n) <= (n - 1) // 2, np.arange(n), np.arange(n) - n) for n in (n1, n2, n3)]
    fg = np.fft.fftn(g).conj()
    ref = np.zeros_like(out)
    for a, t in enumerate(tau):
        ph = [np.exp(-2j * np.pi * m[j] * t[j]) for j in range(3)]
        w = (vt[kind[a]] * fg * ph[2][:, None, None] * ph[1][None, :, None] * ph[0]).imag
        ref[a] = 2 * np.pi * np.array([(w * m[0]).sum(), (w * m[1][:, None]).sum(), (w * m[2][:, None, None]).sum()])
    assert np.abs(out - ref).max() < 1e-12 * np.abs(ref).max()
    ctx.close()


@pytest.mark.parametrize("na,nb", [(1, 3), (64, 1), (65, 4), (900, 2), (7400, 1)])
def test_projector_gradient_over_slices(cuda, na, nb):
    """One projector (16 slices of plane waves), more projectors than CTAs, and two blocks of projectors (7,400 on
    4,613 plane waves are 546 MB), against numpy: FP64 sums, 1e-12 of the largest product's scale."""
    import torch
    from cpw2000_b200 import configs
    d = configs.kpoint_inputs(configs.si8_cubic_kbatch(nk=1), 0)
    m, natom = d["mtxd"], 3
    rng = np.random.default_rng(na)
    x = np.resize(rng.standard_normal((1 << 20) - 3), 2 * m * na).view(np.complex128).reshape(na, m).T
    xnl, occ = rng.choice((-1.0, 1.0), na), np.linspace(2.0, 0.5, nb)
    atom = rng.integers(0, natom, na).astype(np.int32)
    psi = rng.standard_normal((m, nb)) + 1j * rng.standard_normal((m, nb))
    ctx = H.Context(0)
    ctx.set_kpoint(m, d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    ctx.set_potential(d["vscr"])
    ctx.set_projectors(x, xnl)
    p, out = _dev(cuda, psi), np.zeros((natom, 3))
    _lib.check(_lib.lib().cpw_b200_nl_grad_device(ctx.handle, nb, C.c_void_p(p.data_ptr()), m, _lib.dptr(occ),
                                                  _lib.iptr(atom), natom, _lib.dptr(out), None))
    g = d["kgv"][:, d["isort"] - 1].astype(float)
    pr = x.conj().T @ psi
    ref = np.zeros((natom, 3))
    for j in range(3):
        q = x.conj().T @ (g[j][:, None] * psi)
        np.add.at(ref[:, j], atom, -4 * np.pi * xnl * ((pr.conj() * q).imag @ occ))
    assert np.abs(out - ref).max() < 1e-12 * np.abs(pr).max() ** 2 * np.abs(g).max() * na
    ctx.close()
