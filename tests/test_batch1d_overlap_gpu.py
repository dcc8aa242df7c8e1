"""The batch kernel's overlapping warps against the per-function 1D kernels,
bitwise: run lengths at the edges of its lanes, warps and teams, a run of one
lane, sources and probes inside the overlaps, at the run's last cell and in
every cells-per-thread variant; step counts off the exchange period."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cpt,block", [(8, 1024), (16, 1024), (24, 512), (32, 512), (40, 512)])
def test_overlaps_bitwise(cuda_lib, cpt, block):
    from simulation_gb300 import batch1d as B
    from simulation_gb300 import fd1d as G
    c = cpt + 2  # cells a lane holds
    full = 32 * c
    ke = np.array([c - 1, c + 1, full - 1, full, full + 1, 31 * c * 2 + c, 31 * c * 2 + c + 1, 31 * c * 3 + 5,
                   cpt * block - 1, cpt * block])
    src_k = 3
    rng = np.random.default_rng(cpt)
    pin = np.minimum(ke - 1, np.array([1, 2, 31 * c, 31 * c - 1, 31 * c + c // 2, 31 * c + c // 2 - 1, c - 1, c, 40, 41]))
    pout = np.minimum(ke - 1, np.array([0, ke[1] - 1, ke[2] - 1, 31 * c + 2, 32 * c - 1, 62 * c + 1, 31 * c + c // 2,
                                        93 * c, ke[8] - 1, ke[9] - 2]))
    starts, ends, offs, er, sg = [], [], [0], [], []
    for k in ke:
        for q in range(3):
            a = int(rng.integers(4, max(5, min(k - 1, 3 * full))))
            starts.append(a)
            ends.append(min(int(k), a + int(rng.integers(1, 2 * c))))
            er.append(float(rng.uniform(1, 9)))
            sg.append(float(rng.uniform(0, 0.05)))
        offs.append(len(starts))
    batch = B.SlabBatch(ke, np.array(offs), np.array(starts), np.array(ends), np.array(er), np.array(sg), pin, pout, src_k)
    for ns in (c // 2 * 4, 97):
        r = B.BatchRunner(batch, nsteps=ns, freqs=np.linspace(1e8, 3e9, 33), wave=("gauss", 20, 6.0),
                          tuning={"groups": [{"ke_lo": 0, "ke_hi": 1 << 30, "cpt": cpt, "block": block}]})
        r.run()
        torch.cuda.synchronize()
        assert int(r.status.item()) == 0 and int(r.done.sum()) == ke.size
        for q in range(ke.size):
            ca, cb = batch.coefficients(q)
            sim = G.Sim1D(int(ke[q]), "cacb", ca=ca, cb=cb, src_kind="soft", src_k=src_k, wave=("gauss", 20, 6.0),
                          freq=r.freqs, dt=B.DT, probes=(int(pin[q]), int(pout[q])), ns=ns)
            sim.step_per_function(ns)
            torch.cuda.synchronize()
            want = torch.stack([sim.r_pr[0], sim.i_pr[0], sim.r_pr[1], sim.i_pr[1]])
            assert torch.equal(r.spec[q], want), f"cpt {cpt} ns {ns} run {q} ke {ke[q]} pin {pin[q]} pout {pout[q]}"
