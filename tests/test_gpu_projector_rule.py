"""Which form the projector products of H|psi> take, by the shape of the call (no forcing variable).

Random projectors of the wanted number on a small cell; only the forms taken are looked at, apart from the
drop-in, whose result is compared with the oracle (1e-12, the drop-in's tolerance).
"""
import numpy as np
import pytest

from cpw2000_b200 import configs
from cpw2000_b200 import ditsp as E
from cpw2000_b200 import hk_psi as H
from cpw2000_b200._lib import CpwB200Error

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def by_rule(monkeypatch):
    monkeypatch.delenv("CPW_B200_NL_CRT", raising=False)


def _projectors(m, na, seed=1):
    rng = np.random.default_rng(seed)
    v = np.resize(rng.standard_normal(1 << 20), 2 * m * na)
    return v.view(np.complex128).reshape(na, m).T / np.sqrt(m), rng.choice((-1.0, 1.0), na)


def _context(d, prec, na):
    ctx = H.Context(0, precision=prec)
    ctx.set_kpoint(d["mtxd"], d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    ctx.set_potential(d["vscr"])
    ctx.set_projectors(*_projectors(d["mtxd"], na))
    return ctx


def _taken(before, after):
    return {k for k, n in after.items() if n != before[k] and not k.startswith("mgs")}


def test_a_mixed_solve_keeps_one_form(cuda):
    """130 bands of 4,613 plane waves and 3,600 projectors: a call of its own takes residues, the blocks of a
    MIXED_TC solve, large and small, all take split TF32."""
    import torch
    w = configs.si8_cubic_kbatch(nk=1)
    nb = 130
    d = configs.kpoint_inputs(w, 0, nbands=nb, with_hamsm=True)
    ctx = _context(d, H.MIXED_TC, 3600)
    psi = torch.randn((3 * nb, d["mtxd"]), dtype=torch.complex128, device=cuda).t()
    hpsi = torch.zeros_like(psi)
    start = ctx.form_counts()
    ctx.hk_psi(psi, hpsi, neig=nb)
    alone = ctx.form_counts()
    assert _taken(start, alone) == {"residues"}
    try:
        E.eigensolve(ctx, psi, hpsi, nb, d["mtxds"], d["hamsm"], d["hdiag"], epspsi=1e-5, icmax=2)
    except CpwB200Error:
        pass                                # the small matrix is another operator's: no convergence is asked for
    assert _taken(alone, ctx.form_counts()) == {"split_tf32"}
    ctx.close()


def _forms(cuda, ctx, m, nbs):
    import torch
    out = {}
    for nb in nbs:
        psi = torch.randn((nb, m), dtype=torch.complex128, device=cuda).t()
        before = ctx.form_counts()
        ctx.hk_psi(psi, torch.zeros_like(psi))
        (out[nb],) = _taken(before, ctx.form_counts())
    ctx.synchronize()
    ctx.close()
    return out


def test_split_tf32_of_a_residue_set(cuda, monkeypatch):
    """Its operands are made by the first block that takes them, and again after new projectors."""
    import torch
    d = configs.kpoint_inputs(configs.si8_cubic_kbatch(nk=1), 0)
    m, na, nb = d["mtxd"], 3600, 5
    ctx = _context(dict(d, ekpg=0 * d["ekpg"], vscr=0 * d["vscr"]), H.MIXED_TC, na)
    psi = torch.randn((nb, m), dtype=torch.complex128, device=cuda).t()
    out = {}
    for seed in (1, 2):
        x, xnl = _projectors(m, na, seed)
        ctx.set_projectors(x, xnl)
        for form, force in (("residues", None), ("split_tf32", "0"), ("residues", None)):
            monkeypatch.delenv("CPW_B200_NL_CRT", raising=False)
            if force:
                monkeypatch.setenv("CPW_B200_NL_CRT", force)
            h, before = torch.zeros_like(psi), ctx.form_counts()
            ctx.hk_psi(psi, h)
            ctx.synchronize()
            assert _taken(before, ctx.form_counts()) == {form}
            p = psi.cpu().numpy()
            ref = x @ (xnl[:, None] * (x.conj().T @ p))
            assert np.abs(h.cpu().numpy() - ref).max() < 2e-5 * np.abs(ref).max()
            out[seed, form] = h
        assert not torch.equal(out[seed, "residues"], out[seed, "split_tf32"])
    ctx.close()


def test_mixed_tc_form_follows_the_projector_set(cuda):
    """From 16 M elements of X on, residues for any number of bands; below, from 128 bands and 15 GFLOP."""
    d = configs.kpoint_inputs(configs.si8_cubic_kbatch(nk=1), 0)
    m = d["mtxd"]
    na = int(1.6e7 / m) + 1
    assert set(_forms(cuda, _context(d, H.MIXED_TC, na), m, (1, 60, 140)).values()) == {"residues"}
    assert _forms(cuda, _context(d, H.MIXED_TC, na - 1), m, (1, 127, 128)) == {1: "split_tf32", 127: "split_tf32",
                                                                             128: "residues"}
    assert _forms(cuda, _context(d, H.MIXED_TC, 1500), m, (128, 140)) == {128: "split_tf32", 140: "residues"}


@pytest.mark.parametrize("na,nb,form", [(700, 60, "zgemm"), (700, 200, "residues"), (32, 400, "zgemm"),
                                        (64, 600, "zgemm")])
def test_fp64_form_counts_the_conversion(cuda, na, nb, form):
    """The rule's sides, among them many bands on few projectors, which ZGEMMs do faster at any size."""
    d = configs.kpoint_inputs(configs.si8_cubic_kbatch(nk=1), 0)
    assert _forms(cuda, _context(d, H.FP64, na), d["mtxd"], (nb,)) == {nb: form}


def test_drop_in_with_both_forms_in_one_call(cuda):
    """831 plane waves, 4,200 projectors: six chunks whose four inner ones (96 bands) take residues and whose half-size
    ends take ZGEMMs."""
    from oracle import hk_psi as O
    d = configs.kpoint_inputs(configs.si2_fcc(), 1)
    m, na, nb = d["mtxd"], 4200, 480
    x, xnl = _projectors(m, na)
    x = np.asfortranarray(x)
    psi = configs.random_psi(m, nb, 5)
    hpsi = np.zeros((m, nb), dtype=np.complex128, order="F")
    before = H.form_counts()
    H.hk_psi_c16(m, nb, psi, hpsi, False, d["ng"], np.asfortranarray(d["kgv"]), d["ekpg"], d["isort"], d["vscr"],
                 d["kmscr"], x, xnl, na, m, nb, na, d["ng"], d["vscr"].size)
    after = H.form_counts()
    assert {k: after[k] - before[k] for k in _taken(before, after)} == {"residues": 4, "zgemm": 2}
    ref = O.hk_psi_c16(m, nb, psi, d["ekpg"], d["isort"], d["vscr"], d["kmscr"], d["kgv"], x, xnl)
    assert np.abs(hpsi - ref).max() < 1e-12 * np.abs(ref).max()


def test_planes_make_room(cuda, monkeypatch):
    """With the device nearly full, a call whose slab no longer fits takes the residue planes back and uses the other
    form; so does one on new projectors whose planes do not fit; there is room again, and they come back."""
    import torch
    d = configs.kpoint_inputs(configs.si8_cubic_kbatch(nk=1), 0)
    m, nb = d["mtxd"], 200
    ctx = _context(d, H.FP64, 1500)         # planes 620 MB; a slab of 200 bands 108 MB
    ctx.set_slab_budget(1 << 30)
    psi = torch.randn((nb, m), dtype=torch.complex128, device=cuda).t()
    few, full, again = torch.zeros_like(psi), torch.zeros_like(psi), torch.zeros_like(psi)
    ctx.hk_psi(psi, few, neig=40)
    before = ctx.form_counts()
    monkeypatch.setenv("CPW_B200_NL_CRT", "1")
    ctx.hk_psi(psi, few, neig=40)
    monkeypatch.delenv("CPW_B200_NL_CRT")
    assert _taken(before, ctx.form_counts()) == {"residues"}
    ctx.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (32 << 20), dtype=torch.uint8, device=cuda)
    before = ctx.form_counts()
    ctx.hk_psi(psi, full)
    ctx.synchronize()
    assert _taken(before, ctx.form_counts()) == {"zgemm"}
    ctx.set_projectors(*_projectors(m, 1500))
    before = ctx.form_counts()
    ctx.hk_psi(psi, again)
    ctx.synchronize()
    assert _taken(before, ctx.form_counts()) == {"zgemm"}
    assert torch.equal(again, full)
    del fill
    torch.cuda.empty_cache()
    ctx.set_projectors(*_projectors(m, 1500))
    before = ctx.form_counts()
    ctx.hk_psi(psi, again)
    ctx.synchronize()
    assert _taken(before, ctx.form_counts()) == {"residues"}
    assert float((again - full).abs().max() / full.abs().max()) < 1e-12
    ctx.close()
