"""A captured H|psi> replayed after new projectors of the same shape equals the eager call with them.

The default projector forms: FP64 ZGEMMs, split TF32 and residue products of both. Replay and eager call run the
same kernels on the same data: equal to the bit. In between, projectors of another shape are set and used.
"""
import numpy as np
import pytest

from cpw2000_b200 import configs
from cpw2000_b200 import hk_psi as H
from cpw2000_b200._lib import CpwB200Error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,crt", [(H.FP64, "0"), (H.FP64, "1"), (H.MIXED_TC, "0"), (H.MIXED_TC, "1")])
def test_replay_follows_the_projectors(cuda, prec, crt, monkeypatch):
    import torch
    monkeypatch.setenv("CPW_B200_NL_CRT", crt)
    d = configs.kpoint_inputs(configs.si2_fcc(), 1)
    m, na, nb = d["mtxd"], 150, 20
    rng = np.random.default_rng(7)
    sets = []
    for n in (na, na, na + 9):
        x = np.asfortranarray(rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n)))
        sets.append((x, rng.choice((-1.0, 1.0), n)))
    ctx = H.Context(0, precision=prec)
    ctx.set_kpoint(m, d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    ctx.set_potential(d["vscr"])
    ctx.set_projectors(*sets[2])
    psi = torch.randn((nb, m), dtype=torch.complex128, device=cuda).t()
    out, eager = torch.zeros_like(psi), torch.zeros_like(psi)
    ctx.hk_psi(psi, eager)                  # the largest buffers first
    ctx.set_projectors(*sets[0])
    ctx.hk_psi(psi, eager)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.hk_psi(psi, out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager)
    before = eager.clone()
    ctx.set_projectors(*sets[2])            # another shape, used
    ctx.hk_psi(psi, eager)
    torch.cuda.synchronize()
    ctx.set_projectors(*sets[1])            # the captured shape, other values: no eager call before the replay
    graph.replay()
    torch.cuda.synchronize()
    ctx.hk_psi(psi, eager)
    torch.cuda.synchronize()
    assert not torch.equal(eager, before)
    assert torch.equal(out, eager)
    graph.reset()
    ctx.close()


@pytest.mark.parametrize("prec,crt", [(H.FP64, "0"), (H.FP64, "1"), (H.MIXED_TC, "0"), (H.MIXED_TC, "1")])
def test_capture_before_any_eager_call_with_the_projectors(cuda, prec, crt, monkeypatch):
    """Buffers sized by other projectors of the shape; the first call with the present ones is the captured one. Eager
    calls between the capture and the replay see them too."""
    import torch
    monkeypatch.setenv("CPW_B200_NL_CRT", crt)
    d = configs.kpoint_inputs(configs.si2_fcc(), 1)
    m, na, nb = d["mtxd"], 150, 20
    rng = np.random.default_rng(8)
    sets = []
    for _ in range(3):
        x = np.asfortranarray(rng.standard_normal((m, na)) + 1j * rng.standard_normal((m, na)))
        sets.append((x, rng.choice((-1.0, 1.0), na)))
    ctx = H.Context(0, precision=prec)
    ctx.set_kpoint(m, d["isort"], d["kgv"], d["ekpg"], d["kmscr"])
    ctx.set_potential(d["vscr"])
    psi = torch.randn((nb, m), dtype=torch.complex128, device=cuda).t()
    out, eager = torch.zeros_like(psi), torch.zeros_like(psi)
    ctx.set_projectors(*sets[0])
    ctx.hk_psi(psi, out)
    ctx.set_projectors(*sets[1])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.hk_psi(psi, out)
    ctx.hk_psi(psi, eager)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager)
    ctx.set_projectors(*sets[2])
    graph.replay()
    torch.cuda.synchronize()
    ctx.hk_psi(psi, eager)
    torch.cuda.synchronize()
    assert torch.equal(out, eager)
    graph.reset()
    ctx.close()


@pytest.mark.parametrize("prec", [H.FP64, H.MIXED_TC])
def test_a_discarded_capture_leaves_no_planes_behind(cuda, prec, monkeypatch):
    """New projectors, then a captured call that needs more scratch than any eager call has sized, thrown away: what
    it recorded of the conversion never ran. The next eager call converts for itself."""
    import ctypes as C

    import torch
    rt = C.CDLL("libcudart.so.12")
    monkeypatch.setenv("CPW_B200_NL_CRT", "1")
    d = configs.kpoint_inputs(configs.si2_fcc(), 1)
    m, na, nb = d["mtxd"], 150, 300
    rng = np.random.default_rng(9)
    x = [np.asfortranarray(rng.standard_normal((m, na)) + 1j * rng.standard_normal((m, na))) for _ in range(2)]
    xnl = rng.choice((-1.0, 1.0), na)
    ctx = H.Context(0, precision=prec)
    ctx.set_kpoint(m, d["isort"], d["kgv"], 0 * d["ekpg"], d["kmscr"])
    ctx.set_potential(0 * d["vscr"])
    ctx.set_slab_budget(1)                  # one band at a time: the slab does not grow
    psi = torch.randn((nb, m), dtype=torch.complex128, device=cuda).t()
    out = torch.zeros_like(psi)
    ctx.set_projectors(x[0], xnl)
    ctx.hk_psi(psi, out, neig=20)
    ctx.set_projectors(x[1], xnl)
    torch.cuda.synchronize()
    st, graph = torch.cuda.Stream(), C.c_void_p()
    assert rt.cudaStreamBeginCapture(C.c_void_p(st.cuda_stream), 2) == 0        # relaxed: allocations may go on
    try:
        ctx.hk_psi(psi, out, stream=st.cuda_stream)
    except CpwB200Error:
        pass
    rt.cudaStreamEndCapture(C.c_void_p(st.cuda_stream), C.byref(graph))
    if graph:
        assert rt.cudaGraphDestroy(graph) == 0
    torch.cuda.synchronize()
    ctx.hk_psi(psi, out)
    ctx.synchronize()
    p = psi.cpu().numpy()
    ref = x[1] @ (xnl[:, None] * (x[1].conj().T @ p))
    assert np.abs(out.cpu().numpy() - ref).max() < (1e-12 if prec == H.FP64 else 1e-6) * np.abs(ref).max()
    ctx.close()
