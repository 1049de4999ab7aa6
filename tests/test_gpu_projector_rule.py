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
