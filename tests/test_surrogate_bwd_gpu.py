"""The input packing and the fused backward kernels of the surrogate against plain FP32/FP64 torch:
GELU backward with the bias sum from each of its three sources, and the lift's
backward from FP32 gradients, at row counts and widths off the blocks' shape."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gelu_grad(z):
    u = np.sqrt(2 / np.pi) * (z + 0.044715 * z ** 3)
    t = torch.tanh(u)
    return 0.5 * (1 + t) + 0.5 * z * (1 - t * t) * np.sqrt(2 / np.pi) * (1 + 3 * 0.044715 * z * z)


@pytest.mark.parametrize("C,B,N", [(8, 1, 1), (24, 3, 7), (128, 5, 33), (128, 64, 512), (264, 2, 129), (2048, 2, 5)])
@pytest.mark.parametrize("src", ["dy16", "dy32", "dh"])
def test_gelu_bwd_sum(cuda_lib, C, B, N, src):
    from simulation_gb300 import surrogate as S
    g = torch.Generator().manual_seed(C + N)
    rows = B * N
    pre = torch.randn((rows, C), generator=g).cuda().bfloat16()
    dy = torch.randn((rows, C), generator=g).cuda()
    dh = torch.randn((B, C), generator=g).cuda()
    dz = torch.empty((rows, C), dtype=torch.bfloat16, device="cuda")
    db = torch.ones(C, device="cuda")
    d16 = dy.bfloat16()
    S._call("fno_gelu_bwd_sum", rows, C, N, d16.data_ptr() if src == "dy16" else None,
            dy.data_ptr() if src == "dy32" else None, dh.data_ptr() if src == "dh" else None, pre.data_ptr(),
            dz.data_ptr(), db.data_ptr())
    ref_d = {"dy16": d16.double(), "dy32": dy.double(),
             "dh": (dh / N).bfloat16().double().repeat_interleave(N, 0)}[src]
    ref = ref_d * _gelu_grad(pre.double())
    torch.cuda.synchronize()
    # BF16 rounding (2^-9) of the result, and the hardware tanh (2^-11) in it
    assert float((dz.double() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max())
    # the sum is of the stored values, in FP32: rows rounding errors of the running sum at most
    want = 1 + dz.double().sum(0)
    scale = dz.double().abs().sum(0) + 1
    assert float(((db.double() - want).abs() / scale).max()) <= 1e-6


@pytest.mark.parametrize("cin", [1, 6, 8])
@pytest.mark.parametrize("rows,C", [(1, 8), (77, 24), (4096, 128), (513, 264)])
def test_lift_bwd32(cuda_lib, rows, C, cin):
    from simulation_gb300 import surrogate as S
    g = torch.Generator().manual_seed(rows + cin)
    x = torch.randn((rows, cin), generator=g).cuda()
    dx = torch.randn((rows, C), generator=g).cuda()
    dP, dp = torch.zeros((C, cin), device="cuda"), torch.zeros(C, device="cuda")
    S._call("fno_lift_bwd32", rows, C, cin, x.data_ptr(), dx.data_ptr(), dP.data_ptr(), dp.data_ptr())
    d = dx.bfloat16().double()
    torch.cuda.synchronize()
    lim = 1e-6 * (d.abs().T @ x.double().abs() + 1)
    assert bool(((dP.double() - d.T @ x.double()).abs() <= lim).all())
    assert bool(((dp.double() - d.sum(0)).abs() <= 1e-6 * (d.abs().sum(0) + 1)).all())


@pytest.mark.parametrize("B,M", [(1, 128), (3, 256), (200, 384)])
def test_gemm_gelu_bwd(cuda_lib, B, M):
    """the GELU-gradient epilogue against the plain product and FP64"""
    from simulation_gb300.tc import gemm
    g = torch.Generator().manual_seed(M)
    A = torch.randn((B, M, 128), generator=g).cuda().bfloat16()
    W = (torch.randn((128, 128), generator=g) / 11).cuda().bfloat16()
    z = torch.randn((B, M, 128), generator=g).cuda().bfloat16()
    db = torch.ones(128, device="cuda")
    out = torch.empty((B, M, 128), dtype=torch.bfloat16, device="cuda")
    gemm(A, W, b_mn=True, out=out, gelu_bwd=(z, db))
    y = gemm(A, W, b_mn=True)
    ref = y.double() * _gelu_grad(z.double())
    torch.cuda.synchronize()
    assert float((out.double() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max())
    want = 1 + out.double().sum((0, 1))
    scale = out.double().abs().sum((0, 1)) + 1
    assert float(((db.double() - want).abs() / scale).max()) <= 1e-6


@pytest.mark.parametrize("B,N,cin,ldo,pad", [(1, 1, 1, 16, 1), (3, 33, 6, 64, 0), (8, 32, 15, 64, 1), (41, 100, 6, 24, 1)])
def test_pack_inputs(cuda_lib, B, N, cin, ldo, pad):
    """rows (inputs, 1, zeros) in both layouts, exact; columns past 16 kept unless padded"""
    from simulation_gb300 import surrogate as S
    g = torch.Generator().manual_seed(N)
    x = torch.randn((B, N, cin), generator=g).cuda()
    out = torch.full((B, N, ldo), 5.0, dtype=torch.bfloat16, device="cuda")
    out_t = torch.full((N, B, 16), 5.0, dtype=torch.bfloat16, device="cuda")
    S._call("fno_pack_inputs", B, N, cin, ldo, pad, x.data_ptr(), out.data_ptr(), out_t.data_ptr())
    want = torch.zeros((B, N, ldo), dtype=torch.bfloat16, device="cuda")
    want[..., :cin] = x.bfloat16()
    want[..., cin] = 1.0
    if not pad:
        want[..., 16:] = 5.0
    assert torch.equal(out, want)
    assert torch.equal(out_t, want[..., :16].transpose(0, 1))


@pytest.mark.parametrize("nbins", [1, 100, 2048, 2800, 2801, 3000])
def test_profile_features(cuda_lib, nbins):
    """overlapping, empty, clipped and many layers: the last that holds a cell counts"""
    from simulation_gb300 import surrogate as S
    rng = np.random.default_rng(nbins)
    counts = np.array([0, 1, 5, 300, 2])
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    st = rng.integers(0, 2 * nbins + 20, off[-1]).astype(np.int32)
    en = (st + rng.integers(-3, nbins + 3, off[-1])).astype(np.int32)
    ep, sg = rng.uniform(1, 9, off[-1]), rng.uniform(0, 0.05, off[-1])
    idx = np.array([3, 0, 4, 2, 1, 3], dtype=np.int32)
    want = np.zeros((idx.size, nbins, 6), dtype=np.float32)
    for q, r in enumerate(idx):
        e, s = np.zeros(2 * nbins + 1), np.zeros(2 * nbins + 1)  # cells -1 .. 2 nbins - 1
        for l in range(off[r], off[r + 1]):
            lo, hi = min(st[l], 2 * nbins) + 1, max(min(en[l], 2 * nbins) + 1, 0)  # no negative slice ends
            e[lo:hi] = (ep[l] - 1.0) / S.EPS_SCALE
            s[lo:hi] = sg[l] / S.SIG_SCALE
        for j in range(3):
            want[q, :, j], want[q, :, 3 + j] = e[j:j + 2 * nbins:2], s[j:j + 2 * nbins:2]
    dev = [torch.as_tensor(a).cuda() for a in (idx, off, st, en, ep, sg)]
    out = torch.empty((idx.size, nbins, 6), device="cuda")
    S._call("fno_profile_features", idx.size, *(t.data_ptr() for t in dev), nbins, S.EPS_SCALE, S.SIG_SCALE,
            out.data_ptr())
    assert torch.equal(out.cpu(), torch.from_numpy(want))
