"""Failure detection on the GPU without a fault: bounded device waits that run out.

Every wait of the library's kernels on another party is bounded; when the limit
runs out the kernel records the failure and returns, the host reports
CPW_B200_TIMEOUT, and the context stays usable. Nothing here faults, traps or
hangs the GPU:

1. mbarrier wait (tensor-core GEMM roles): cpw_b200_wait_selftest runs the
   GEMMs' bounded wait on an mbarrier that nothing arrives at, with a 1 ms
   limit. cpw_b200_synchronize then returns CPW_B200_TIMEOUT, the next one 0,
   and a MIXED_TC H|psi> on the same context still matches the oracle.
2. grid barrier (the eigensolver's cooperative Gram-Schmidt kernel): with its
   poll limit set to 0, a CTA that reaches a grid barrier before the others
   gives up at its first poll, so the eigensolver call returns
   CPW_B200_TIMEOUT; with the default limit restored the same context solves
   to the dense eigenvalues.
3. the projector products' roles with a limit of 0 ns, and the eigensolver's status after one gave up.
"""
import numpy as np
import pytest

from cpw2000_b200 import _lib, configs
from cpw2000_b200 import ditsp as E
from cpw2000_b200 import hk_psi as H
from cpw2000_b200._lib import CpwB200Error
from oracle import hk_psi as O

pytestmark = pytest.mark.gpu

TIMEOUT = -4


def test_mbarrier_wait_runs_out_and_context_recovers(cuda):
    import torch
    w = configs.si2_fcc()
    d = configs.kpoint_inputs(w, 1)
    ctx = H.Context(0, precision=H.MIXED_TC).setup(d)
    L = _lib.lib()
    assert L.cpw_b200_wait_selftest(ctx.handle, 1_000_000, None) == 0
    assert L.cpw_b200_synchronize(ctx.handle) == TIMEOUT
    assert "gave up" in L.cpw_b200_last_error().decode()
    assert L.cpw_b200_synchronize(ctx.handle) == 0          # the flag is cleared once reported
    m, nb = d["mtxd"], 5
    psi_h = configs.random_psi(m, nb, 71)
    psi = torch.from_numpy(np.ascontiguousarray(psi_h.T)).to(cuda).t()
    out = torch.zeros((nb, m), dtype=torch.complex128, device=cuda).t()
    ctx.hk_psi(psi, out)
    ctx.synchronize()
    ref = O.hk_psi_c16(m, nb, psi_h, d["ekpg"], d["isort"], d["vscr"], d["kmscr"], d["kgv"], d["anlga"], d["xnlkb"])
    assert np.abs(out.cpu().numpy() - ref).max() / np.abs(ref).max() < 2e-5
    ctx.close()


@pytest.mark.parametrize("form", ["residues", "residues, 9 moduli", "split TF32", "int8 slices"])
def test_gemm_roles_with_no_time_to_wait(cuda, form, monkeypatch):
    """With a limit of 0 ns a role that has to wait at all may give up: the call then reports the time-out, and
    the next one on the same context is right. Blocks of several tiles per CTA, so that every role waits."""
    import torch
    monkeypatch.setenv("CPW_B200_NL_CRT", "1" if "residues" in form else "0")
    d = configs.kpoint_inputs(configs.si2_fcc(), 1)
    rng = np.random.default_rng(3)
    m, na, nb = d["mtxd"], 700, 300
    x = np.asfortranarray(rng.standard_normal((m, na)) + 1j * rng.standard_normal((m, na)))
    xnl = rng.choice((-1.0, 1.0), na)
    ctx = H.Context(0, precision=H.FP64 if _fp64(form) else H.MIXED_TC)
    ctx.set_kpoint(m, d["isort"], d["kgv"], 0 * d["ekpg"], d["kmscr"])
    ctx.set_potential(0 * d["vscr"])
    ctx.set_projectors(x, xnl)
    L = _lib.lib()
    if form == "int8 slices":
        assert L.cpw_b200_set_projector_slices(ctx.handle, 7) == 0
    psi = rng.standard_normal((m, nb)) + 1j * rng.standard_normal((m, nb))
    dev = torch.from_numpy(np.ascontiguousarray(psi.T)).to(cuda).t()
    out = torch.zeros((nb, m), dtype=torch.complex128, device=cuda).t()
    for limit in (0, -1, 0, 200, -1):           # -1: the default
        L.cpw_b200_set_wait_limits(ctx.handle, limit, -1)
        ctx.hk_psi(dev, out)
        status = L.cpw_b200_synchronize(ctx.handle)
        assert status in ((0, TIMEOUT) if limit >= 0 else (0,))
        if limit < 0:
            ref = x @ (xnl[:, None] * (x.conj().T @ psi))
            assert np.abs(out.cpu().numpy() - ref).max() < (1e-12 if _fp64(form) else 2e-5) * np.abs(ref).max()
    ctx.close()


def _fp64(form):
    return form in ("residues", "int8 slices")


@pytest.mark.parametrize("prec", [H.FP64, H.MIXED_TC])
def test_eigensolver_reports_a_wait_that_gave_up(cuda, prec, monkeypatch):
    """A tensor-core kernel that gave up leaves H|psi> incomplete: the solve that used it does not return success.
    The flag is that of the projector products; the self-test raises it as a product of the solve would."""
    import torch
    monkeypatch.setenv("CPW_B200_NL_CRT", "1")
    d = configs.kpoint_inputs(configs.si2_fcc(), 0, with_hamsm=True)
    nb, m = 8, d["mtxd"]
    ctx = H.Context(0, precision=prec).setup(d)

    def solve():
        psi = torch.zeros((3 * nb, m), dtype=torch.complex128, device=cuda).t()
        return E.eigensolve(ctx, psi, torch.zeros_like(psi), nb, d["mtxds"], d["hamsm"], d["hdiag"], epspsi=1e-5)

    assert _lib.lib().cpw_b200_wait_selftest(ctx.handle, 1_000_000, None) == 0
    with pytest.raises(CpwB200Error) as ei:
        solve()
    assert ei.value.status == TIMEOUT
    assert solve()["converged"]             # the flag is cleared once reported
    ctx.synchronize()
    ctx.close()


def test_selftest_rejects_limits_above_two_seconds(cuda):
    ctx = H.Context(0)
    L = _lib.lib()
    assert L.cpw_b200_wait_selftest(ctx.handle, 3_000_000_000, None) == 1
    ctx.close()


def test_grid_barrier_wait_runs_out_and_context_recovers(cuda):
    import torch
    w = configs.si2_fcc()
    d = configs.kpoint_inputs(w, 0, with_hamsm=True)
    nb = 8
    ctx = H.Context(0).setup(d)            # FP64: the reference's modified Gram-Schmidt on the device
    m = d["mtxd"]

    def solve():
        psi = torch.zeros((3 * nb, m), dtype=torch.complex128, device=cuda).t()
        hpsi = torch.zeros_like(psi)
        return E.eigensolve(ctx, psi, hpsi, nb, d["mtxds"], d["hamsm"], d["hdiag"], epspsi=1e-5)

    ctx.set_wait_limits(grid_polls=0)
    with pytest.raises(CpwB200Error) as ei:
        solve()
    assert ei.value.status == TIMEOUT and "grid barrier" in str(ei.value)
    ctx.set_wait_limits()                   # defaults again
    r = solve()
    assert r["converged"]
    dense = np.linalg.eigvalsh(O.dense_h(m, d["ekpg"], d["isort"], d["vscr"], d["kmscr"], d["kgv"], d["anlga"],
                                         d["xnlkb"]))
    assert np.abs(r["ei"] - dense[: r["neig"]]).max() < 1e-8
    ctx.close()
