"""The 2D time loop's workspace where device memory is short: SimTM2D then takes the
smallest size that runs the program, as it does where the fast path's extra would
leave the caller less than half of the free memory, and the results stay the same."""
import pytest
import torch

from simulation_gb300 import _lib, build
from simulation_gb300 import fd2d as G


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _sim(nx, ny, dft, device):
    return G.SimTM2D(nx, ny, pml=G.pmlparam(nx, ny, 8, device=device), lossy=True,
                     source=G.PointSource(nx // 2, ny // 2, ("gauss", 20, 6.0)), ns=64, device=device,
                     freq=[1e8, 4e8, 7e8] if dft else None)


# ragged rows run without any workspace, the DFT on whole rows with the passes' six fields
@pytest.mark.parametrize("nx,ny,dft,plain_slots", [(1101, 1003, False, 0), (1101, 1003, True, 0), (1024, 1536, True, 6)])
@pytest.mark.parametrize("how", ["out of memory", "little left"])
def test_falls_back_to_the_smallest_size(monkeypatch, nx, ny, dft, plain_slots, how):
    s = _sim(nx, ny, dft, "cpu")
    fast = _lib.lib().fdtd2d_fast_workspace_size(s._p, 0)
    plain = _lib.lib().fdtd2d_workspace_size(s._p, 0)
    assert plain == plain_slots * ((nx * ny * 4 + 255) // 256 * 256) < fast
    empty, tried = torch.empty, []

    def short(*a, **k):
        tried.append(a[0])
        if a[0] >= fast:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*a, **k)

    if how == "out of memory":
        monkeypatch.setattr(torch, "empty", short)
    else:
        monkeypatch.setattr(G, "WS_EXTRA_SMALL", 0)
        monkeypatch.setattr(G, "free_bytes", lambda device: 2 * (fast - plain) - 1)
    ws = s.workspace()
    assert (0 if ws is None else ws.numel()) == plain
    n = len(tried)
    assert s.workspace() is ws and len(tried) == n  # decided once
    monkeypatch.undo()
    assert _sim(nx, ny, dft, "cpu").workspace().numel() == fast


def test_out_of_memory_for_the_smallest_size_is_raised(monkeypatch):
    s = _sim(1024, 1536, True, "cpu")
    monkeypatch.setattr(torch, "empty", lambda *a, **k: (_ for _ in ()).throw(torch.cuda.OutOfMemoryError("none")))
    with pytest.raises(torch.cuda.OutOfMemoryError):
        s.workspace()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,dft", [(1101, 1003, False), (1501, 1203, True), (1400, 1536, True)])
def test_same_results_with_the_smallest_size(cuda_lib, monkeypatch, nx, ny, dft):
    a = _sim(nx, ny, dft, "cuda")
    assert a.workspace() is not None
    monkeypatch.setattr(G, "WS_EXTRA_SMALL", 0)
    monkeypatch.setattr(G, "free_bytes", lambda device: 0)
    b = _sim(nx, ny, dft, "cuda")
    for n in (9, 24):
        a.step(n)
        b.step(n)
    plain = _lib.lib().fdtd2d_workspace_size(b._p, 0)
    assert (0 if b._workspace is None else b._workspace.numel()) == plain < a._workspace.numel()
    torch.cuda.synchronize()
    for k in a.FIELDS:
        x, y = getattr(a, k), getattr(b, k)
        assert x is None or torch.equal(x, y), k
