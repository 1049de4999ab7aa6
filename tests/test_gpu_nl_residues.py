"""Projector products as residue GEMMs (csrc/crt.cu) against an extended-precision product on the CPU.

With V = 0 and no kinetic term H|psi> is X diag(xnlkb) X^H psi alone. The rows of the operands are rounded
to 2^-57 (FP64 form) or 2^-34 (MIXED_TC) of their 2-norms or better, so an element of P is off by at
most ~2^-56 |x| |psi|, sqrt(2 m) 2^-56 of a typical element, and the expansion adds sqrt(2 nanl) 2^-56:
below 1e-14 and 1e-7 of the result's maximum for the sizes here (sqrt(2 m) <= 41).
"""
import numpy as np
import pytest

from cpw2000_b200 import configs
from cpw2000_b200 import hk_psi as H

pytestmark = pytest.mark.gpu
TOL = {H.FP64: 1e-14, H.MIXED: 1e-14, H.MIXED_TC: 1e-7}


@pytest.fixture(autouse=True)
def residues(monkeypatch):
    monkeypatch.setenv("CPW_B200_NL_CRT", "1")


def _basis(name):
    return configs.kpoint_inputs(configs.WORKLOADS[name](), 1)


def _context(d, prec, x, xnl):
    ctx = H.Context(0, precision=prec)
    ctx.set_kpoint(d["mtxd"], d["isort"], d["kgv"], 0 * d["ekpg"], d["kmscr"])
    ctx.set_potential(0 * d["vscr"])
    ctx.set_projectors(x, xnl)
    return ctx


def _apply(cuda, ctx, psi):
    import torch
    # strides given outright: a transposed single column may report any
    p, h = (torch.empty_strided(psi.shape, (1, psi.shape[0]), dtype=torch.complex128, device=cuda) for _ in range(2))
    p.copy_(torch.from_numpy(psi))
    before = ctx.form_counts()
    ctx.hk_psi(p, h)
    ctx.synchronize()
    assert {k: n - before[k] for k, n in ctx.form_counts().items() if n != before[k]} == {"residues": 1}
    return h.cpu().numpy()


def _exact(x, xnl, psi):
    x, psi = x.astype(np.clongdouble), psi.astype(np.clongdouble)
    return x @ (xnl.astype(np.longdouble)[:, None] * (x.conj().T @ psi))


def _random(m, na, nb, seed):
    rng = np.random.default_rng(seed)
    x = np.asfortranarray((rng.standard_normal((m, na)) + 1j * rng.standard_normal((m, na)))
                          * np.exp(-rng.uniform(0, 4, (m, 1))))
    return x, rng.choice((-1.0, 1.0), na), rng.standard_normal((m, nb)) + 1j * rng.standard_normal((m, nb))


# edges: one row or column, one more or less than a tile (128 rows, 16 columns, 4 bands, 256 columns),
# one K block and a remainder of one
@pytest.mark.parametrize("prec", [H.FP64, H.MIXED, H.MIXED_TC])
@pytest.mark.parametrize("cell,na,nb", [("small", 1, 1), ("small", 129, 5), ("si2", 127, 16), ("si2", 128, 17),
                                        ("si2", 257, 3), ("si2", 8, 255), ("si2", 33, 258)])
def test_matches_extended_precision(cuda, prec, cell, na, nb):
    d = _basis(cell)
    x, xnl, psi = _random(d["mtxd"], na, nb, na + nb)
    ctx = _context(d, prec, x, xnl)
    ref = _exact(x, xnl, psi)
    err = float(np.abs(_apply(cuda, ctx, psi) - ref).max() / np.abs(ref).max())
    assert err < TOL[prec]
    ctx.close()


@pytest.mark.parametrize("prec", [H.FP64, H.MIXED_TC])
def test_bands_that_avoid_the_large_projector_elements(cuda, prec):
    """Projectors that fall off by ten orders of magnitude over the plane waves, bands that live on the smallest rows
    alone: the result is as accurate relative to its own size as for any other band (bounds as above: sums over
    the 60 rows and 60 rows of X to 57 or 34 bits of like numbers)."""
    d = _basis("si2")
    m, na = d["mtxd"], 40
    x, xnl, psi = _random(m, na, 5, 9)
    x = np.asfortranarray(x * np.logspace(0, -10, m)[:, None])
    psi[:-60] = 0.0
    x[-7] = 0.0                             # a plane wave that no projector sees
    ctx = _context(d, prec, x, xnl)
    got, ref = _apply(cuda, ctx, psi), _exact(x, xnl, psi)
    err = np.abs(got - ref).max(axis=1) / np.abs(ref).max(axis=1).clip(1e-300)      # row by row
    assert float(err.max()) < TOL[prec]
    ctx.close()


def test_scales_and_non_finite_bands(cuda):
    """A band of tiny or huge numbers keeps its relative accuracy; a NaN or an infinity makes its own band
    NaN and leaves the others as they are, to the bit."""
    d = _basis("si2")
    m = d["mtxd"]
    x, xnl, psi = _random(m, 24, 7, 5)
    ctx = _context(d, H.FP64, x, xnl)
    clean = _apply(cuda, ctx, psi)
    psi[:, 1] *= 2.0 ** -700
    psi[:, 2] *= 2.0 ** 700
    psi[:, 3] = 0.0
    psi[m // 2, 4] = np.nan
    psi[0, 5] = np.inf
    got = _apply(cuda, ctx, psi)
    assert np.array_equal(got[:, [0, 6]], clean[:, [0, 6]])
    for band, e in ((1, 700), (2, -700)):
        assert np.array_equal(got[:, band] * 2.0 ** e, clean[:, band])
    assert np.all(got[:, 3] == 0)
    assert np.isnan(got[:, 4]).all() and np.isnan(got[:, 5]).all()
    ctx.close()


def test_new_projectors_and_precision_replace_the_planes(cuda):
    d = _basis("si2")
    x, xnl, psi = _random(d["mtxd"], 20, 6, 7)
    x2, xnl2, _ = _random(d["mtxd"], 31, 6, 8)
    x3, xnl3, _ = _random(d["mtxd"], 31, 6, 9)
    ctx = _context(d, H.MIXED, x, xnl)
    _apply(cuda, ctx, psi)
    ctx.set_projectors(x2, xnl2)
    ref = _exact(x2, xnl2, psi)
    assert float(np.abs(_apply(cuda, ctx, psi) - ref).max() / np.abs(ref).max()) < TOL[H.MIXED]
    ctx.set_precision(H.MIXED_TC)         # 9 moduli on the same projectors, then 15 again
    nine = _apply(cuda, ctx, psi)
    assert float(np.abs(nine - ref).max() / np.abs(ref).max()) < TOL[H.MIXED_TC]
    ctx.set_precision(H.MIXED)
    fifteen = _apply(cuda, ctx, psi)
    assert float(np.abs(fifteen - ref).max() / np.abs(ref).max()) < TOL[H.MIXED]
    assert not np.array_equal(nine, fifteen)
    ctx.set_projectors(x3, xnl3)          # the same shape
    ref = _exact(x3, xnl3, psi)
    assert float(np.abs(_apply(cuda, ctx, psi) - ref).max() / np.abs(ref).max()) < TOL[H.MIXED]
    ctx.close()


@pytest.mark.parametrize("nb,chunks", [(15, 1), (40, 3), (97, 4), (97, 6)])
def test_drop_in_chunks(cuda, nb, chunks, monkeypatch):
    """The drop-in's band chunks (one; three, four and six with half-size ends) with residue products, and again with
    other projectors and waves, against the oracle (1e-12, the drop-in's tolerance). Residues everywhere take
    four chunks by themselves."""
    if chunks == 6:
        monkeypatch.setenv("CPW_B200_DROPIN_CHUNKS", "6")
    _drop_in(nb, lambda n: n == {"residues": chunks})


def _drop_in(nb, forms):
    from oracle import hk_psi as O
    d = _basis("si2")
    m = d["mtxd"]
    for seed, na in ((nb, 20), (nb + 1, 33)):
        x, xnl, _ = _random(m, na, 1, seed)
        psi = configs.random_psi(m, nb, seed)
        hpsi = np.zeros((m, nb), dtype=np.complex128, order="F")
        before = H.form_counts()
        H.hk_psi_c16(m, nb, psi, hpsi, False, d["ng"], np.asfortranarray(d["kgv"]), d["ekpg"], d["isort"], d["vscr"],
                     d["kmscr"], x, xnl, na, m, nb, na, d["ng"], d["vscr"].size)
        assert forms({k: n - before[k] for k, n in H.form_counts().items() if n != before[k]})
        ref = O.hk_psi_c16(m, nb, psi, d["ekpg"], d["isort"], d["vscr"], d["kmscr"], d["kgv"], x, xnl)
        assert np.abs(hpsi - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("prec", [H.FP64, H.MIXED_TC])
def test_first_call_on_new_projectors_does_not_wait(cuda, prec):
    """The conversion of new projectors is queued like the rest of the call: hk_psi returns while earlier work of
    its stream still runs."""
    import torch
    d = _basis("si2")
    x, xnl, psi = _random(d["mtxd"], 40, 6, 11)
    ctx = _context(d, prec, x, xnl)
    _apply(cuda, ctx, psi)                 # sizes the buffers
    ctx.set_projectors(x[:, ::-1], xnl[::-1].copy())
    p, h = (torch.zeros((6, d["mtxd"]), dtype=torch.complex128, device=cuda).t() for _ in range(2))
    p.copy_(torch.from_numpy(psi))
    torch.cuda.synchronize()
    busy = torch.cuda.Event()
    torch.cuda._sleep(10 ** 9)             # about half a second
    busy.record()
    ctx.hk_psi(p, h)
    assert not busy.query()
    ctx.synchronize()
    ref = _exact(x, xnl, psi)
    assert float(np.abs(h.cpu().numpy() - ref).max() / np.abs(ref).max()) < TOL[prec]
    ctx.close()


@pytest.mark.parametrize("prec", [H.FP64, H.MIXED_TC])
def test_several_accumulations_along_the_plane_waves(cuda, prec):
    """70,000 plane waves: more than the 512 K blocks of 128 that one int32 accumulation holds. Sums of 2 x 70,000
    products of operands held to 2^-57 and 2^-34 of their norms: sqrt(140,000) 2^-56 = 5.2e-15 and 4.4e-8 of a
    typical element, a few of these for the largest of 5 x 3 and 70,000 x 3."""
    k = np.arange(-23, 24)
    g = np.stack([a.ravel() for a in np.meshgrid(k, k, k, indexing="ij")])
    g = np.asfortranarray(g[:, np.argsort((g * g).sum(0), kind="stable")[:70000]].astype(np.int32))
    m = 70000
    d = dict(mtxd=m, isort=np.arange(1, m + 1, dtype=np.int32), kgv=g, ekpg=np.zeros(m), vscr=np.zeros(49 * 48 * 48),
             kmscr=np.array([23, 23, 23, 48, 48, 48, 49], dtype=np.int32))
    x, xnl, psi = _random(m, 5, 3, 12)
    ctx = _context(d, prec, x, xnl)
    got, ref = _apply(cuda, ctx, psi), _exact(x, xnl, psi)
    assert float(np.abs(got - ref).max() / np.abs(ref).max()) < {H.FP64: 3e-14, H.MIXED_TC: 3e-7}[prec]
    ctx.close()
