"""Plane wave and running DFT in the chained passes and in the on-chip loop
against the per-function kernels, bitwise: sizes around the stripes and segments, the tiles and the
incident line's warps, box edges on stripe
borders, with and without layer and loss, frequency counts, either extra alone,
step counts that take every pass length, graph replay and the smallest
workspace."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sim(nx, ny, lossy, npml, tfsf, nf, ns=64):
    from simulation_gb300 import fd2d as G
    dt = 0.01 / 6e8
    naz = nbz = None
    if lossy:
        naz, nbz = G.dielectric(nx, ny, min(8, min(nx, ny) // 4), min(nx, ny) // 4, dt, 30.0, 0.3)
    s = G.SimTM2D(nx, ny, pml=G.pmlparam(nx, ny, npml) if npml else None, naz=naz, nbz=nbz, lossy=lossy,
                  tfsf_npml=tfsf, freq=np.linspace(1e8, 9e8, nf) if nf else None, dt=dt, ns=ns)
    i = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None]
    j = torch.arange(ny, device="cuda", dtype=torch.float64)[None, :]
    s.dz.copy_((0.1 * torch.cos(0.11 * i + 0.3) * torch.cos(0.07 * j + 0.1)).float())
    return s


def _equal(a, b, what):
    torch.cuda.synchronize()
    a.check()
    for k in list(a.FIELDS) + ["r_pt", "i_pt", "r_in", "i_in", "ezi", "hxi", "bc"]:
        x, y = getattr(a, k, None), getattr(b, k, None)
        if x is not None:
            assert torch.equal(x, y), f"{what}: {k} max {float((x - y).abs().max()):.3e}"


@pytest.mark.parametrize("nx,ny", [(1024, 1400), (1100, 1344), (8200, 132), (300, 4096), (1403, 1012), (1300, 1345), (1024, 1402)])
@pytest.mark.parametrize("lossy,npml,tfsf,nf", [(True, 8, 8, 3), (True, 12, 9, 1), (False, 8, 8, 6), (True, 0, 60, 2),
                                                (False, 8, 0, 4), (True, 8, 8, 0)])
def test_sizes(cuda_lib, nx, ny, lossy, npml, tfsf, nf):
    a, b = _sim(nx, ny, lossy, npml, tfsf, nf), _sim(nx, ny, lossy, npml, tfsf, nf)
    for n in (8, 21, 4, 16):
        a.step(n)
    b.step_per_function(49)
    _equal(a, b, f"{nx}x{ny}")


@pytest.mark.parametrize("nx,ny,tfsf", [(20, 17, 4), (100, 100, 8), (129, 127, 8), (250, 241, 60), (96, 385, 8),
                                        (1001, 61, 2), (513, 516, 8), (61, 3072, 9), (40, 3076, 9), (1024, 1024, 8),
                                        (1080, 960, 112)])
@pytest.mark.parametrize("lossy,npml,nf", [(True, 8, 3), (False, 4, 13), (True, 0, 1), (False, 0, 0)])
def test_on_chip(cuda_lib, nx, ny, tfsf, lossy, npml, nf):
    npml = min(npml, (min(nx, ny) - 1) // 2 - 1)
    a, b = _sim(nx, ny, lossy, npml, tfsf, nf, 128), _sim(nx, ny, lossy, npml, tfsf, nf, 128)
    for n in (4, 67, 9):
        a.step(n)
    b.step_per_function(80)
    _equal(a, b, f"{nx}x{ny}")


@pytest.mark.parametrize("nx,ny", [(1024, 1400), (400, 500)])
def test_graph_and_march(cuda_lib, nx, ny):
    mk = lambda: _sim(nx, ny, True, 8, 8, 3)  # noqa: E731
    a, c, g = mk(), mk(), mk()
    a.step(40)
    c.step(40, steps_per_pass=4)
    g.run_graph(20)
    g.run_graph(20)
    _equal(a, c, "march")
    _equal(a, g, "graph")
