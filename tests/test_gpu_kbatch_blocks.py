"""The batched projector products over the block shapes they accept, against a numpy product.

Blocks of 1 to 64 projectors and bands (edges of the 4 x 4 thread tiles, one tile, all 256), k-points
of one batch with different counts, one and several slices of plane waves. V = 0, so that H|psi> is the
kinetic term and X diag(xnlkb) X^H psi; both sides are FP64 sums of at most 836 products, 1e-13 of the
largest result.
"""
import numpy as np
import pytest

from cpw2000_b200 import configs
from cpw2000_b200 import hk_psi as H
from cpw2000_b200 import kbatch as KB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [[(1, 1)], [(3, 5), (4, 4), (64, 64)], [(5, 1), (1, 64), (0, 7), (64, 3)],
                                    [(32, 40)] * 5, [(63, 61), (17, 9)]])
def test_block_shapes(cuda, blocks):
    import torch
    w = configs.si2_fcc()
    rng = np.random.default_rng(len(blocks))
    ks = []
    for k, (na, nb) in enumerate(blocks):
        d = configs.kpoint_inputs(w, k)
        d["kgv"] = ks[0]["kgv"] if ks else d["kgv"]
        if k:                       # every k-point on the first one's G vectors: a basis of its leading ones
            d["mtxd"] = ks[0]["mtxd"] - 37 * k
            d["isort"], d["ekpg"] = ks[0]["isort"][:d["mtxd"]], ks[0]["ekpg"][:d["mtxd"]]
        m = d["mtxd"]
        d["anlga"] = np.asfortranarray(rng.standard_normal((m, na)) + 1j * rng.standard_normal((m, na)))
        d["xnlkb"] = rng.choice((-1.0, 1.0), na)
        d["vscr"] = 0 * d["vscr"]
        ks.append(d)
    ctx = H.Context(0).setup(ks[0])
    kb = KB.KBatch(ctx, ks)
    psi = [rng.standard_normal((d["mtxd"], nb)) + 1j * rng.standard_normal((d["mtxd"], nb))
           for d, (_, nb) in zip(ks, blocks)]
    x, y = ([torch.empty_strided(p.shape, (1, p.shape[0]), dtype=torch.complex128, device=cuda) for p in psi]
            for _ in range(2))
    for a, p in zip(x, psi):
        a.copy_(torch.from_numpy(p))
    for _ in range(2):              # the tuned call, then the replayed graph
        kb.hk_psi(x, y)
        kb.synchronize()
        for d, p, got in zip(ks, psi, y):
            ref = d["ekpg"][:, None] * p + d["anlga"] @ (d["xnlkb"][:, None] * (d["anlga"].conj().T @ p))
            assert np.abs(got.cpu().numpy() - ref).max() < 1e-13 * np.abs(ref).max()
    kb.close()
    ctx.close()
