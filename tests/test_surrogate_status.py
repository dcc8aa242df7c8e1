"""The surrogate's kernels wait on their copies for a bounded time.  Every tensor-core
launch of a network carries its status word, so that a wait that runs out is seen:
checked on the CPU with recorded calls in place of the kernels."""
import pytest
import torch

from simulation_gb300 import _lib, build
from simulation_gb300 import surrogate as S


@pytest.mark.parametrize("nbins,modes", [(256, 32), (256, 16)])  # fused layers, and separate products
def test_every_tensor_core_launch_has_the_networks_status_word(monkeypatch, nbins, modes):
    build.build()
    layers, words = [], []

    def call(name, *args):
        if name == "fno_layer_fwd":
            layers.append(args[-1])

    def gemm(A, B, *, out=None, a_mn=False, b_mn=False, status=None, **kw):
        words.append(status)
        if out is None:
            batch = max(A.shape[0] if A.dim() == 3 else 1, B.shape[0] if B.dim() == 3 else 1)
            shape = (A.shape[-1] if a_mn else A.shape[-2], B.shape[-1] if b_mn else B.shape[-2])
            out = torch.zeros((batch,) + shape if max(A.dim(), B.dim()) == 3 else shape)
        return out

    monkeypatch.setattr(S, "_call", call)
    monkeypatch.setattr(S, "gemm", gemm)
    m = S.FNO(device="cpu", nbins=nbins, modes=modes)
    m.fold = False
    m.loss_and_grad(torch.zeros((3, nbins, 6)), torch.zeros((3, 128)))
    assert len(layers) == (m.L if modes == 32 else 0) and len(words) > 10
    assert all(p == m.status.data_ptr() for p in layers)
    assert all(w is m.status for w in words)
    m.check()
    m.status.fill_(2)
    with pytest.raises(_lib.FdtdError) as e:
        m.check()
    assert e.value.code == -7
