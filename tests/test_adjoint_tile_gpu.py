"""The adjoint on the chip (checkpoint intervals of 4 and more where the tiles
fit the SMs) against the streaming kernels (interval 3), bitwise: boxes off the
groups of four and over tile borders, with and without loss, both gradients,
partial last segments, hard and soft sources, probes inside the box."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(nx, ny, npml, lossy, box, src, probe, kind, ns, cp):
    from simulation_gb300 import _lib
    from simulation_gb300 import fd2d as G
    s = G.SimTM2D(nx, ny, pml=G.pmlparam(nx, ny, npml), lossy=lossy,
                  source=G.PointSource(*src, ("gauss", 12, 4.0), kind), ns=ns)
    g = torch.Generator().manual_seed(nx)
    i0, j0, ni, nj = box
    s.naz.fill_(1.0)
    s.naz[i0:i0 + ni, j0:j0 + nj] = 1.0 / (1.0 + 3.0 * torch.rand((ni, nj), generator=g)).cuda()
    if lossy:
        s.nbz.zero_()
        s.nbz[i0:i0 + ni, j0:j0 + nj] = 0.02 * torch.rand((ni, nj), generator=g).cuda()
    ap = _lib.AdjointParams2D(ns, cp, probe[0], probe[1], 2.0, _lib.Box2D(*box))
    n = _lib.lib().fdtd2d_tm_adjoint_workspace_size(C.byref(s._p), C.byref(ap))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    trace = torch.zeros(ns, device="cuda")
    J = torch.zeros(1, dtype=torch.float64, device="cuda")
    gn = torch.full((ni, nj), 7.0, device="cuda")
    gb = torch.full((ni, nj), 7.0, device="cuda") if lossy else None
    _lib.call("fdtd2d_tm_adjoint", C.byref(s._p), C.byref(ap), trace.data_ptr(), J.data_ptr(), gn.data_ptr(),
              None if gb is None else gb.data_ptr(), ws.data_ptr(), ws.numel(), _lib.stream_ptr())
    torch.cuda.synchronize()
    return trace, J, gn, gb


@pytest.mark.parametrize("nx,ny,box,src,probe", [
    (40, 40, (10, 9, 18, 21), (12, 20), (30, 20)),          # one tile; the source and the probe in the box
    (100, 128, (30, 40, 40, 50), (25, 64), (65, 64)),
    (130, 260, (1, 1, 128, 258), (40, 130), (80, 131)),     # almost the whole grid
    (300, 516, (60, 113, 170, 301), (50, 258), (90, 259)),
    (700, 512, (300, 250, 99, 3), (290, 256), (330, 255)),
    (1024, 1024, (384, 384, 256, 256), (344, 512), (390, 512)),
])
@pytest.mark.parametrize("lossy", [False, True])
@pytest.mark.parametrize("kind", ["hard", "soft"])
def test_against_streaming(cuda_lib, nx, ny, box, src, probe, lossy, kind):
    a = _run(nx, ny, 8, lossy, box, src, probe, kind, 151, 32)  # segments of 32, 32, 32, 32, 23
    b = _run(nx, ny, 8, lossy, box, src, probe, kind, 151, 3)
    c = _run(nx, ny, 8, lossy, box, src, probe, kind, 151, 50)  # the last of one step
    assert float(b[1]) > 0 and float(b[2].abs().max()) > 0
    for x in (a, c):
        for p, q in zip(x, b):
            assert (p is None and q is None) or torch.equal(p, q)


@pytest.mark.parametrize("box,ns,cp", [((30, 40, 40, 50), 90, 32), ((1, 1, 98, 126), 90, 8), ((1, 1, 98, 126), 400, 8),
                                       ((60, 3, 5, 120), 91, 30)])
def test_recorded_halves(cuda_lib, box, ns, cp):
    """forward_rec/reverse_rec (with and without room for the whole record) equal
    the unrecorded halves, in any order and repeated"""
    from simulation_gb300 import _lib
    from simulation_gb300 import fd2d as G
    s = G.SimTM2D(100, 128, pml=G.pmlparam(100, 128, 8), source=G.PointSource(25, 64, ("gauss", 12, 4.0), "soft"),
                  lossy=False, ns=ns)
    s.naz.fill_(0.7)
    ap = _lib.AdjointParams2D(ns, cp, 50, 64, 2.0, _lib.Box2D(*box))
    n = _lib.lib().fdtd2d_tm_adjoint_workspace_size(C.byref(s._p), C.byref(ap))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    trace = torch.zeros(ns, device="cuda")
    J = torch.zeros(1, dtype=torch.float64, device="cuda")

    def fwd(rec):
        _lib.call("fdtd2d_tm_adjoint_forward" + rec, C.byref(s._p), C.byref(ap), trace.data_ptr(), J.data_ptr(),
                  ws.data_ptr(), ws.numel(), _lib.stream_ptr())
        return trace.clone(), J.clone()

    def rev(rec):
        g = torch.empty(box[2:], device="cuda")
        _lib.call("fdtd2d_tm_adjoint_reverse" + rec, C.byref(s._p), C.byref(ap), g.data_ptr(), None, ws.data_ptr(),
                  ws.numel(), _lib.stream_ptr())
        return g

    want = fwd("") + (rev(""),)
    got = fwd("_rec") + (rev("_rec"), rev(""), rev("_rec"))
    assert float(want[2].abs().max()) > 0
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    for g in got[2:]:
        assert torch.equal(g, want[2])


def test_a_wait_that_ran_out_is_reported(cuda_lib):
    """An expired wait of the forward leaves FDTD_STATUS_TIMEOUT in its word: every
    gradient taken from that forward is then NaN and check() raises; the next forward
    starts clean."""
    from simulation_gb300 import _lib
    from simulation_gb300.adjoint import AdjointProblem
    pr = AdjointProblem(nx=128, ny=128, npml=8, box=(16, 16), src_offset=20, probe_offset=20, ns=240, checkpoint=16)
    pr.set_eps(torch.full((16, 16), 2.0))
    J = pr.forward()
    want = pr.gradient_naz().clone()
    assert bool(torch.isfinite(want).all()) and float(want.abs().max()) > 0
    pr.check()
    pr.status[0] = 2
    assert bool(torch.isnan(pr.gradient_naz()).all())
    with pytest.raises(_lib.FdtdError):
        pr.check()
    assert pr.forward() == J
    assert torch.equal(pr.gradient_naz(), want)
    pr.check()
