"""The fused spectral layer against the separate products, mean pool included:
the same sums in the same order, so outputs and gradients agree bitwise, at
one tile and several a sample and at batches below and above the SM count."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,layers,B", [(128, 1, 1), (128, 3, 5), (256, 2, 153), (512, 4, 307), (2048, 2, 3)])
@pytest.mark.parametrize("fold", [True, False])
def test_fused_layers_equal_separate(cuda_lib, monkeypatch, N, layers, B, fold):
    from simulation_gb300 import surrogate as S
    m = S.FNO(seed=2, nbins=N, layers=layers)
    m.fold = fold
    g = torch.Generator().manual_seed(N + B)
    m.p["H2"].copy_(((torch.rand(m.p["H2"].shape, generator=g) * 2 - 1) / 16).cuda())
    m._refresh_bf16()
    x = (torch.rand((B, N, 6), generator=g) * 2 - 1).cuda()
    t = torch.randn((B, 128), generator=g).cuda()
    got = []
    fused = S.FNO._fused
    for pick in (lambda self, n: False, fused):
        monkeypatch.setattr(S.FNO, "_fused", pick)
        y = m.forward(x)
        m.loss_and_grad(x, t)
        s = m._saved
        got.append([y, s["h"]] + s["x"] + s["pre"] + s["Fm"])
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("N,layers,B", [(128, 1, 1), (128, 3, 5), (256, 2, 153), (2048, 2, 3)])
def test_gradients_equal_separate(cuda_lib, monkeypatch, N, layers, B):
    """The gradients from either forward.  The weights' come from products: the same bits.
    The lift's and the biases' are added up by atomics in any order: of at most k = 1216
    partial sums p, so two runs differ by 2 k 2^-24 sum|p| = 1.5e-4 sum|p| at most; 1e-3 of
    the largest entry leaves room for sums that cancel to a seventh."""
    from simulation_gb300 import surrogate as S
    m = S.FNO(seed=3, nbins=N, layers=layers)
    g = torch.Generator().manual_seed(N * B)
    m.p["H2"].copy_(((torch.rand(m.p["H2"].shape, generator=g) * 2 - 1) / 16).cuda())
    m._refresh_bf16()
    x = (torch.rand((B, N, 6), generator=g) * 2 - 1).cuda()
    t = torch.randn((B, 128), generator=g).cuda()
    got = []
    fused = S.FNO._fused
    for pick in (lambda self, n: False, fused):
        monkeypatch.setattr(S.FNO, "_fused", pick)
        m.loss_and_grad(x, t)
        got.append({k: v.clone() for k, v in m.g.items()})
    for k, a in got[0].items():
        b = got[1][k]
        assert float(a.abs().max()) > 0, k
        if k.startswith("H") or k.split(".")[-1] in ("W", "Rr", "Ri"):
            assert torch.equal(a, b), k
        else:
            assert float((a - b).abs().max()) <= 1e-3 * float(a.abs().max()), k


def test_layer_refuses(cuda_lib):
    from simulation_gb300 import _lib
    p = torch.zeros(64, device="cuda").data_ptr()
    args = lambda **k: [{**dict(B=1, N=128, C=128, M=32, K1=128), **k}[q] for q in ("B", "N", "C", "M", "K1")]  # noqa: E731
    f = lambda a, xo=p, fm=p, h=None: _lib.lib().fno_layer_fwd(*a, p, p, p, p, p, xo, fm, h, None, None, None)  # noqa: E731
    for bad in (dict(N=100), dict(N=384), dict(N=64), dict(C=64), dict(M=16), dict(K1=96), dict(K1=64), dict(B=0), dict(B=65536)):
        assert f(args(**bad)) == -2
    assert f(args(), p, None) != 0 and f(args(), p, p, p) != 0 and f(args(), p + 4) != 0
