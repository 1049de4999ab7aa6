"""Modified Gram-Schmidt by one cluster against the grid form it replaces.

Row counts at the edges of the rule (one block, two, the largest of each number of blocks to a CTA, the
first that goes back to the grid) and block counts that leave one, two or three blocks of the last CTA
without rows (9, 11, 13, 15 of 512 rows at two to a CTA; 17, 18, 19, 23, 30 at four), plane waves sorted by kinetic energy in a random potential. Both forms
add the same parts in the same order, so whole eigensolves agree bit for bit; the vectors are orthonormal
to rounding of sums of 16,385 products (1e-12).
"""
import numpy as np
import pytest

from cpw2000_b200 import ditsp as E
from cpw2000_b200 import hk_psi as H
from oracle import hk_psi as O

pytestmark = pytest.mark.gpu


def _case(m):
    n = 40
    k = np.arange(-19, 20)
    g = np.stack([a.ravel() for a in np.meshgrid(k, k, k, indexing="ij")])
    e = (g * g).sum(0)
    o = np.argsort(e, kind="stable")[:m]
    rng = np.random.default_rng(m)
    d = dict(mtxd=m, kgv=np.asfortranarray(g[:, o].astype(np.int32)), isort=np.arange(1, m + 1, dtype=np.int32),
             ekpg=0.3 * e[o] + 0.3 * rng.uniform(size=m), kmscr=np.array([19, 19, 19, n, n, n, n + 1], dtype=np.int32),
             vscr=0.5 * rng.standard_normal((n + 1) * n * n))
    d["mtxds"] = 60
    d["hamsm"] = np.asfortranarray(O.dense_h(60, d["ekpg"], d["isort"], d["vscr"], d["kmscr"], d["kgv"],
                                             np.zeros((60, 0), np.complex128), np.zeros(0)))
    return d


@pytest.mark.parametrize("m", [512, 513, 1024, 1025, 4096, 4097, 8192, 8193, 16384, 16385,
                               5600, 6600, 7680, 9100, 9700, 11700, 15300])
def test_cluster_and_grid_forms_agree(cuda, m, monkeypatch):
    import torch
    d, nb = _case(m), 12
    ctx = H.Context(0)
    ctx.set_kpoint(m, d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    ctx.set_potential(d["vscr"])
    out = []
    for grid in ("0", "1"):
        monkeypatch.setenv("CPW_B200_MGS_GRID", grid)
        psi = torch.zeros((3 * nb, m), dtype=torch.complex128, device=cuda).t()
        before = ctx.form_counts()
        r = E.eigensolve(ctx, psi, torch.zeros_like(psi), nb, 60, d["hamsm"], d["ekpg"] + d["vscr"].mean(), epspsi=1e-5)
        assert r["converged"]
        ran = {k for k, n in ctx.form_counts().items() if k.startswith("mgs") and n != before[k]}
        assert ran == {"mgs_cluster" if grid == "0" and 512 < m <= 16384 else "mgs_grid"}
        p = psi[:, :nb].cpu().numpy()
        assert np.abs(p.conj().T @ p - np.eye(nb)).max() < 1e-12
        out.append((r["ei"], p))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    ctx.close()
