"""The on-chip 2D time loop (grids whose tiles fit the SMs) against the
per-function kernels, bitwise: one tile and many, tile-edge and odd sizes, with
and without loss and absorbing layer, sources on tile borders, calls off the
exchange period, graph replay, and the march for the same grids."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sim(nx, ny, lossy, npml, src, kind="hard", wave=("gauss", 20, 6.0)):
    from simulation_gb300 import fd2d as G
    dt = 0.01 / 6e8
    naz = nbz = None
    if lossy:
        naz, nbz = G.dielectric(nx, ny, npml, min(nx, ny) // 4, dt, 30.0, 0.3)
    s = G.SimTM2D(nx, ny, pml=G.pmlparam(nx, ny, npml) if npml else None, naz=naz, nbz=nbz, lossy=lossy,
                  source=G.PointSource(*src, wave, kind) if src else None)
    i = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None]
    j = torch.arange(ny, device="cuda", dtype=torch.float64)[None, :]
    s.dz.copy_((0.1 * torch.cos(0.11 * i + 0.3) * torch.cos(0.07 * j + 0.1)).float())
    return s


def _equal(a, b, what):
    torch.cuda.synchronize()
    a.check()
    for k in a.FIELDS:
        x, y = getattr(a, k), getattr(b, k)
        if x is not None:
            assert torch.equal(x, y), f"{what}: {k} max {float((x - y).abs().max()):.3e}"


@pytest.mark.parametrize("nx,ny", [(5, 5), (9, 128), (16, 127), (33, 129), (100, 100), (121, 97), (250, 241),
                                   (300, 512), (1000, 60), (61, 1001), (513, 515), (1024, 1024), (1080, 960)])
@pytest.mark.parametrize("lossy,pml", [(False, False), (False, True), (True, False), (True, True)])
def test_sizes(cuda_lib, nx, ny, lossy, pml):
    npml = max(1, min(8, (min(nx, ny) - 1) // 2 - 1)) if pml else 0
    a = _sim(nx, ny, lossy, npml, (nx // 2, ny // 2))
    b = _sim(nx, ny, lossy, npml, (nx // 2, ny // 2))
    for n in (4, 17, 22):
        a.step(n)
    b.step_per_function(43)
    _equal(a, b, f"{nx}x{ny}")


@pytest.mark.parametrize("src", [(0, 0), (1, 5), (55, 119), (56, 120), (239, 240), (23, 511), (399, 3)])
@pytest.mark.parametrize("kind", ["hard", "soft"])
def test_sources_and_march(cuda_lib, src, kind):
    mk = lambda: _sim(400, 512, True, 12, src, kind, ("sin", 0.01, 9e8))  # noqa: E731
    a, b, c, g = mk(), mk(), mk(), mk()
    a.step(61)
    b.step_per_function(61)
    c.step(61, steps_per_pass=4)
    g.run_graph(30)
    g.run_graph(31)
    _equal(a, b, "per function")
    _equal(a, c, "march")
    _equal(a, g, "graph")


def test_nonfinite_and_two_streams(cuda_lib):
    from simulation_gb300 import _lib
    a = _sim(300, 300, True, 8, (150, 150))
    a.naz[10, 10] = float("nan")
    a.step(20)
    with pytest.raises(_lib.FdtdError):
        a.check()
    sims = [_sim(700, 700, False, 10, (350, 300 + q)) for q in range(2)]
    refs = [_sim(700, 700, False, 10, (350, 300 + q)) for q in range(2)]
    streams = [torch.cuda.Stream() for _ in sims]
    torch.cuda.synchronize()
    for _ in range(4):
        for s, st in zip(sims, streams):
            with torch.cuda.stream(st):
                s.step(25)
    for r in refs:
        r.step_per_function(100)
    for s, r in zip(sims, refs):
        _equal(s, r, "streams")


@pytest.mark.parametrize("lossy,npml", [(False, 0), (False, 12), (True, 12)])
def test_subnormal_fields(cuda_lib, lossy, npml):
    """fields around the smallest normal number: every product is rounded by itself"""
    mk = lambda: _sim(400, 512, lossy, npml, None)  # noqa: E731
    a, b = mk(), mk()
    for s in (a, b):
        s.dz.mul_(1e-37)
    a.step(24)
    b.step_per_function(24)
    _equal(a, b, "subnormal")


@pytest.mark.parametrize("nx,ny", [(100, 100), (250, 241), (700, 512)])
@pytest.mark.parametrize("lossy,npml", [(False, 0), (False, 8), (True, 8)])
@pytest.mark.parametrize("ext", [False, True])
def test_nonfinite_ez_of_the_last_cell(cuda_lib, nx, ny, lossy, npml, ext):
    """No H update reads ez of cell (nx-1, ny-1): an Inf or NaN there is in ez alone"""
    from simulation_gb300 import _lib
    from simulation_gb300 import fd2d as G
    for bad in (float("inf"), float("nan")):
        s = G.SimTM2D(nx, ny, pml=G.pmlparam(nx, ny, npml) if npml else None, lossy=lossy,
                      source=G.PointSource(nx // 2, ny // 2, ("gauss", 20, 6.0)), tfsf_npml=8 if ext else 0)
        s.step(12)
        s.check()
        s.naz[nx - 1, ny - 1] = bad
        s.step(12)
        assert not bool(torch.isfinite(s.ez[nx - 1, ny - 1]))
        with pytest.raises(_lib.FdtdError):
            s.check()
