"""The chunked 1D run against the per-function kernels, bitwise: line lengths
around the chunk, block and cluster edges of its layouts, the DFT of every cell
in registers (up to 4 and 8 frequencies) and in global memory, probes and
sources in the chunks' overlaps, and calls split off the exchange period."""
import numpy as np
import pytest
import torch

from tests.test_fd1d_gpu import _coeffs, _fused_vs_per_function

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [513, 700, 1023, 1985, 3841, 8191, 15361, 38001, 64604, 65535])
@pytest.mark.parametrize("form", ["cb", "cacb", "dform", "debye"])
def test_lengths(cuda_lib, nx, form):
    _fused_vs_per_function(nx, form, 150, src_kind="hard" if nx % 3 == 0 else "soft", src_k=nx // 2,
                           wave=("gauss", 20, 6.0), abc=nx % 4 != 3)


@pytest.mark.parametrize("nf", [1, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("nx,src_k", [(66, 0), (200, 47), (512, 95), (513, 512), (1301, 96)])
def test_every_cell_dft(cuda_lib, nx, src_k, nf):
    for form in ("cb", "dform", "debye"):
        _fused_vs_per_function(nx, form, 131, src_kind="soft", src_k=src_k, wave=("gauss", 20, 6.0),
                               freq=np.linspace(5e7, 9e8, nf), full_dft=True,
                               probes=(0, 1, 10, src_k, nx // 2, nx // 2 + 1, nx - 2, nx - 1))


@pytest.mark.parametrize("nx", [700, 5000])
def test_split_calls_and_initial_fields(cuda_lib, nx):
    from simulation_gb300 import fd1d as G
    kw = dict(src_kind="soft", src_k=97, wave=("gauss", 30, 8.0), freq=[1e8, 4e8, 7e8], probes=(2, 97, nx - 3),
              full_dft=True, **_coeffs(nx, "debye"))
    a, b = G.Sim1D(nx, "debye", **kw), G.Sim1D(nx, "debye", **kw)
    init = torch.sin(torch.arange(nx, dtype=torch.float32, device="cuda") * 0.1)
    for s in (a, b):
        for k in ("ex", "hy", "dx", "r_pt"):
            getattr(s, k).copy_(init.expand_as(getattr(s, k)))
    for n in (1, 31, 33, 64, 7, 90):
        a.step(n)
    b.step_per_function(226)
    torch.cuda.synchronize()
    for k in ("ex", "hy", "dx", "ix", "sx", "bc", "r_pt", "i_pt", "r_pr", "i_pr"):
        assert torch.equal(getattr(a, k), getattr(b, k)), f"nx={nx} {k}"


@pytest.mark.parametrize("nx,form,nf", [(513, "cb", 0), (700, "cacb", 0), (1184, "dform", 0), (800, "debye", 0),
                                        (66, "cb", 3), (300, "debye", 3), (688, "dform", 3), (130, "cb", 8)])
def test_many_calls_shorter_than_the_exchange_period(cuda_lib, nx, form, nf):
    """A call of 1 to 16 steps on a line that one block of several warps holds ends before
    the warps' first exchange: its stores must still come after every warp's loads.  Several
    hundred calls in a row, so that a warp that starts from later values shows."""
    from simulation_gb300 import fd1d as G
    kw = dict(src_kind="soft", src_k=nx // 3, wave=("gauss", 30, 8.0), **_coeffs(nx, form))
    if nf:
        kw.update(freq=np.linspace(5e7, 9e8, nf), full_dft=True, probes=(1, nx // 2, nx - 2))
    a, b = G.Sim1D(nx, form, **kw), G.Sim1D(nx, form, **kw)
    init = torch.sin(torch.arange(nx, dtype=torch.float32, device="cuda") * 0.1)
    for s in (a, b):
        s.ex.copy_(init)
        s.hy.copy_(init.flip(0))
    total = 0
    for n in (1, 2, 3, 5, 8, 13, 16) * 40:
        a.step(n)
        total += n
    b.step_per_function(total)
    torch.cuda.synchronize()
    for k in ("ex", "hy", "dx", "ix", "sx", "bc", "r_pt", "i_pt", "r_pr", "i_pr"):
        x, y = getattr(a, k), getattr(b, k)
        assert x is None or torch.equal(x, y), f"nx={nx} {form} nf={nf}: {k}"
