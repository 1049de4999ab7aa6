"""The compiled z-line forms and the pruned first passes of the local kernels against the oracle.

Every line length with a compiled form, with the kept half-width just inside the outer quarters of the
line (the compiled, pruned forms) and just beyond them (the run-time, unpruned ones), on planes whose
column count is no multiple of the column tile and whose lengths are compiled or not. The basis is a
random set of G vectors in the kept block that includes its corners. Tolerances as for the other
H|psi> parity tests: rounding only.
"""
import numpy as np
import pytest

from cpw2000_b200 import hk_psi as H
from oracle import hk_psi as O

pytestmark = pytest.mark.gpu
TOL = {H.FP64: 1e-12, H.MIXED: 2e-5}

SPLITS = {16: (4, 4), 18: (3, 6), 20: (4, 5), 24: (4, 6), 32: (4, 8), 36: (6, 6), 40: (5, 8), 48: (6, 8), 50: (5, 10),
          54: (6, 9), 64: (8, 8), 72: (8, 9), 80: (8, 10), 96: (8, 12), 100: (10, 10), 108: (9, 12), 128: (8, 16),
          144: (12, 12), 160: (10, 16), 192: (12, 16), 256: (16, 16)}


def _limit(n):
    """The first half-width outside the outer quarters of a line of n points."""
    r1, r2 = SPLITS[n]
    return (r1 + 3) // 4 * r2


def _case(box, kd, nb, seed):
    rng = np.random.default_rng(seed)
    g = np.stack([rng.integers(-k, k + 1, 300) for k in kd])
    g[:, :8] = np.array([[a * kd[0], b * kd[1], c * kd[2]] for a in (-1, 1) for b in (-1, 1) for c in (-1, 1)]).T
    g = np.unique(g, axis=1).astype(np.int32)
    m = g.shape[1]
    n1, n2, n3 = box
    km = np.array([(n - 1) // 2 for n in box] + [n1, n2, n3, n1 + 1], dtype=np.int32)
    d = dict(mtxd=m, isort=np.arange(1, m + 1, dtype=np.int32), kgv=np.asfortranarray(g), ekpg=rng.uniform(0, 9, m),
             kmscr=km, vscr=rng.standard_normal((n1 + 1) * n2 * n3))
    return d, rng.standard_normal((m, nb)) + 1j * rng.standard_normal((m, nb))


def _check(cuda, box, kd, nb, prec, seed):
    import torch
    d, psi = _case(box, kd, nb, seed)
    ctx = H.Context(0, precision=prec)
    ctx.set_kpoint(d["mtxd"], d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    ctx.set_potential(d["vscr"])
    x, y = (torch.empty_strided(psi.shape, (1, psi.shape[0]), dtype=torch.complex128, device=cuda) for _ in range(2))
    x.copy_(torch.from_numpy(psi))
    ctx.hk_psi(x, y)
    torch.cuda.synchronize()
    ref = O.hk_psi_c16(d["mtxd"], nb, np.asfortranarray(psi), d["ekpg"], d["isort"], d["vscr"], d["kmscr"], d["kgv"],
                       np.zeros((d["mtxd"], 0), np.complex128), np.zeros(0))
    assert float(np.abs(y.cpu().numpy() - ref).max() / np.abs(ref).max()) < TOL[prec]
    ctx.close()


@pytest.mark.parametrize("prec", [H.FP64, H.MIXED])
@pytest.mark.parametrize("n3", sorted(SPLITS))
@pytest.mark.parametrize("inside", [True, False])
def test_line_lengths(cuda, n3, inside, prec):
    kd3 = _limit(n3) - 1 if inside else _limit(n3)
    if kd3 > (n3 - 1) // 2:
        pytest.skip("the quarters cover the whole line")
    _check(cuda, (10, 9, n3), (2, 2, kd3), 3, prec, n3)


@pytest.mark.parametrize("prec", [H.FP64, H.MIXED])
@pytest.mark.parametrize("n", [32, 40, 96, 144])
@pytest.mark.parametrize("kx,ky", [(0, 0), (-1, -1), (0, -1), (-1, 0)])
def test_square_planes(cuda, n, kx, ky, prec):
    lim = _limit(n)
    _check(cuda, (n, n, 12), (lim + kx, lim + ky, 3), 2, prec, n + kx)


@pytest.mark.parametrize("prec", [H.FP64, H.MIXED])
@pytest.mark.parametrize("box,kd", [((25, 15, 16), (5, 3, 3)), ((72, 50, 24), (13, 9, 4)), ((16, 256, 20), (3, 50, 4)),
                                    ((128, 18, 36), (24, 3, 11)), ((4, 6, 18), (1, 2, 5)), ((2, 2, 32), (0, 0, 7))])
def test_unequal_planes(cuda, box, kd, prec):
    _check(cuda, box, kd, 5, prec, sum(box))


def test_band_groups_and_chunks_do_not_change_a_bit(cuda):
    import torch
    d, psi = _case((24, 20, 54), (4, 3, 10), 37, 3)
    ctx = H.Context(0)
    ctx.set_kpoint(d["mtxd"], d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    ctx.set_potential(d["vscr"])
    x = torch.from_numpy(np.ascontiguousarray(psi.T)).to(cuda).t()
    whole, part = torch.zeros_like(x), torch.zeros_like(x)
    ctx.hk_psi(x, whole)
    ctx.set_slab_budget(1)          # one band at a time
    ctx.hk_psi(x, part)
    assert torch.equal(whole, part)
    ctx.close()


def test_line_that_fits_no_staging(cuda):
    # 255 kept planes of 256: two staging buffers exceed the shared memory of a CTA in FP64 (the plain form of B)
    _check(cuda, (10, 9, 256), (2, 2, 127), 3, H.FP64, 1)
