"""The chained passes of 4 and 8 steps (large grids; padded copies where ny is
no multiple of 4) against the per-function
kernels, bitwise: sizes around the stripes and segments, with and without loss
and absorbing layer, sources at stripe and segment borders, step counts that
take every pass length, and the march on the same grid."""
import pytest
import torch

from tests.test_fd2d_tile_gpu import _equal, _sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1024, 1400), (1100, 1344), (8200, 132), (70, 16384), (2049, 1012), (1500, 1504),
                                   (1501, 1203), (1300, 1345), (1024, 1402)])
@pytest.mark.parametrize("lossy,npml", [(False, 0), (False, 20), (True, 0), (True, 20)])
def test_sizes(cuda_lib, nx, ny, lossy, npml):
    mk = lambda: _sim(nx, ny, lossy, npml, (nx // 2, ny // 2))  # noqa: E731
    a, b = mk(), mk()
    for n in (8, 23, 4, 16):
        a.step(n)
    b.step_per_function(51)
    _equal(a, b, f"{nx}x{ny}")


@pytest.mark.parametrize("src", [(0, 0), (5, 111), (700, 112), (1023, 1399), (512, 119), (333, 1231)])
def test_sources_and_march(cuda_lib, src):
    mk = lambda: _sim(1024, 1400, True, 16, src, "soft", ("sin", 0.01, 9e8))  # noqa: E731
    a, b, c = mk(), mk(), mk()
    a.step(40)
    b.step_per_function(40)
    c.step(40, steps_per_pass=4)
    _equal(a, b, "per function")
    _equal(a, c, "march")


def test_nonfinite(cuda_lib):
    from simulation_gb300 import _lib
    a = _sim(1500, 1504, True, 8, (700, 700))
    a.naz[900, 1000] = float("nan")
    a.step(16)
    with pytest.raises(_lib.FdtdError):
        a.check()


@pytest.mark.parametrize("lossy,npml", [(False, 0), (False, 12), (True, 12)])
def test_subnormal_fields(cuda_lib, lossy, npml):
    mk = lambda: _sim(1024, 1400, lossy, npml, None)  # noqa: E731
    a, b = mk(), mk()
    for s in (a, b):
        s.dz.mul_(1e-37)
    a.step(24)
    b.step_per_function(24)
    _equal(a, b, "subnormal")
