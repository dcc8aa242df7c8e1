"""Learned surrogate: a 1D Fourier neural operator from a layered slab profile
to its transmission spectrum, trained and served on the GPU by the library's
own BF16 tensor-core kernels, with batched FDTD as its judge and fallback.

Network (no reference counterpart):
* input:  cells [0, 2*NBINS) of a slab run as NBINS=2048 bins of 6 channels,
  (eps_r-1)/8 and sigma/0.05 of cells 2b-1, 2b, 2b+1 (the whole profile, with
  the interfaces between neighbouring bins visible inside one bin);
* lift:   x0 = in P^T + p                                   [B, N, C=128]
* 4 spectral layers, 32 retained modes:
    F  = x^T Phi^T        truncated real DFT (cos rows, -sin rows)
    G  = R_k F_k          complex 128x128 weights per mode
    x' = GELU(x W^T + Psi G^T + b)   (pointwise and inverse DFT share one
                                      tensor-core accumulator)
* head:   y = H2 GELU(H1 mean_n(x) + hb1) + hb2              [B, 128]
* frame:  T(f) = y(f) * P(f), P = exp(-i sum_cells k(f, cell)) the single-pass
  propagation factor of the profile through the Yee update, computed by
  ``fno_propagation`` (per-layer wavenumbers in FP32, sums over cells in FP64).  P carries the phase (thousands of radians across a
  thick stack) and the attenuation (down to 1e-20) that BF16 activations
  cannot hold; the network learns the rest: interface transmission, the
  reflection seen at the entry probe and the multiple reflections.

Every contraction runs in ``fdtd_gemm_bf16`` (tcgen05 tensor cores, FP32
accumulation); every other op in the ``fno_*`` kernels.  Backward and Adam
are hand-written too (``FNO.backward``, ``FNO.adam_step``).  Torch allocates
device memory and gathers minibatches; it computes nothing of the network.

Training data come from the batched FDTD kernel with a DC-free
derivative-of-Gaussian soft source (``WAVE``): with the Gaussian pulse of the
reference's programs the static charge left in lossy layers decays over far
more than a run's 8000 steps and the DFT ratio of an opaque stack measures
that tail, not the stack.
"""
from __future__ import annotations

import math
import time

import numpy as np
import torch

from . import _lib
from . import batch1d as B1
from .tc import gemm

NBINS = 2048
CIN = 6
EPS_SCALE, SIG_SCALE = 8.0, 0.05
WIDTH = 128
MODES = 32
LAYERS = 4
HIDDEN = 256
NFREQ = 64
OUT = 2 * NFREQ
BF = torch.bfloat16
FREQS = np.linspace(100e6, 3e9, NFREQ)
WAVE = ("dgauss", 40, 6.0)
NSTEPS = 8000
PROBE_IN, PROBE_GAP = 30, 10  # entry probe cell; exit probe this far behind the stack


def _st():
    return _lib.stream_ptr()


def _call(name, *args):
    _lib.call(name, *(list(args) + [_st()]))


def dft_matrices(n: int = NBINS, m: int = MODES):
    """Phi [2M][N] (cos rows, -sin rows) and Psi [N][2M] (inverse with a_0=1/N, a_k=2/N), float64."""
    k = np.arange(m)[:, None]
    x = np.arange(n)[None, :]
    th = 2 * np.pi * k * x / n
    phi = np.concatenate([np.cos(th), -np.sin(th)], axis=0)
    a = np.full(m, 2.0 / n)
    a[0] = 1.0 / n
    psi = np.concatenate([(a[:, None] * np.cos(th)).T, (-a[:, None] * np.sin(th)).T], axis=1)
    return phi, psi


def profile_features(batch: "B1.SlabBatch", idx=None, nbins: int = NBINS) -> np.ndarray:
    """[n][nbins][6] float32 inputs: (eps_r-1)/8 of cells 2b-1, 2b, 2b+1, then
    sigma/0.05 of the same cells (vacuum = 0, also beyond a run's end)."""
    idx = np.arange(batch.nruns) if idx is None else np.asarray(idx)
    out = np.zeros((idx.size, nbins, CIN), dtype=np.float32)
    ncell = 2 * nbins
    e = np.zeros(ncell + 2)  # e[c + 1] = cell c, padded with vacuum on both sides
    s = np.zeros(ncell + 2)
    for q, r in enumerate(idx):
        e[:] = 0.0
        s[:] = 0.0
        a, b = batch.layer_off[r], batch.layer_off[r + 1]
        for l in range(a, b):
            lo, hi = int(batch.layer_start[l]), min(int(batch.layer_end[l]), ncell)
            if lo < hi:
                e[lo + 1:hi + 1] = (batch.epsr[l] - 1.0) / EPS_SCALE
                s[lo + 1:hi + 1] = batch.sigma[l] / SIG_SCALE
        for j in range(3):  # cell 2b-1+j sits at e[2b+j]
            out[q, :, j] = e[j:j + ncell:2]
            out[q, :, 3 + j] = s[j:j + ncell:2]
    return out


def device_features(batch: "B1.SlabBatch", idx=None, nbins: int = NBINS, device="cuda") -> torch.Tensor:
    """``profile_features`` built on the device from the batch's layer tables
    (``fno_profile_features``): [n][nbins][6] float32, bitwise the same values.
    The tables are copied to the device once per batch object."""
    dev = torch.device(device)
    tabs = getattr(batch, "_feature_tables", None)
    if tabs is None or tabs[0].device != dev:
        i32 = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.int32)).to(dev)  # noqa: E731
        f64 = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).to(dev)  # noqa: E731
        pad = lambda a: a if a.size else np.zeros(1)  # noqa: E731
        tabs = (i32(batch.layer_off), i32(pad(batch.layer_start)), i32(pad(batch.layer_end)), f64(pad(batch.epsr)),
                f64(pad(batch.sigma)))
        batch._feature_tables = tabs
    idx_t = None
    n = batch.nruns
    if idx is not None:
        idx_t = torch.as_tensor(np.ascontiguousarray(idx, dtype=np.int32)).to(dev)
        n = idx_t.numel()
    out = torch.empty((n, nbins, CIN), dtype=torch.float32, device=dev)
    if n:
        _call("fno_profile_features", n, None if idx_t is None else idx_t.data_ptr(), *(t.data_ptr() for t in tabs),
              nbins, EPS_SCALE, SIG_SCALE, out.data_ptr())
    return out


_WDT = {}


def _wdt_table(device, freqs=FREQS, dt: float | None = None) -> torch.Tensor:
    """w*dt per frequency on ``device`` (float64), copied there once: a copy per
    call would also break CUDA-graph capture and race across streams."""
    dt = B1.DT if dt is None else dt
    key = (str(device), float(dt), tuple(np.asarray(freqs, dtype=np.float64).tolist()))
    wdt = _WDT.get(key)
    if wdt is None:
        wdt = torch.as_tensor(2 * np.pi * np.asarray(freqs, dtype=np.float64) * dt, device=device)
        _WDT[key] = wdt
    return wdt


def propagation(inp: torch.Tensor, freqs=FREQS, dt: float | None = None) -> torch.Tensor:
    """[B][2*nf] float32 frame P of each profile (``fno_propagation``)."""
    dt = B1.DT if dt is None else dt
    wdt = _wdt_table(inp.device, freqs, dt)
    nf = wdt.numel()
    P = torch.empty((inp.shape[0], 2 * nf), dtype=torch.float32, device=inp.device)
    _call("fno_propagation", inp.shape[0], inp.shape[1], inp.data_ptr(), nf, wdt.data_ptr(), EPS_SCALE, SIG_SCALE,
          dt / (2 * B1.EPS0), PROBE_IN, PROBE_GAP, P.data_ptr())
    return P


def cmul(P: torch.Tensor, y: torch.Tensor, conj: bool = False) -> torch.Tensor:
    """P (.) y (or conj(P) (.) y) for spectra stored [Re | Im]."""
    out = torch.empty_like(y)
    _call("fno_cmul", y.shape[0], y.shape[1] // 2, P.data_ptr(), y.data_ptr(), int(conj), out.data_ptr())
    return out


def spectrum_targets(T: np.ndarray) -> np.ndarray:
    """[n][128] float32: (Re T, Im T) of the 64-frequency transmission."""
    return np.concatenate([T.real, T.imag], axis=1).astype(np.float32)


# Spectra of opaque stacks: the FDTD's own FP32 noise is ~1e-7 of the incident
# pulse and thick lossy stacks transmit far less (|T| down to 1e-17), so the
# relative error is taken against max(||T||, FLOOR * sqrt(NFREQ)), i.e. a
# -60 dB floor per frequency.
SPECTRUM_FLOOR = 1e-3


def rel_l2_spectrum(pred: np.ndarray, ref: np.ndarray, floor: float = SPECTRUM_FLOOR) -> np.ndarray:
    """Per-sample relative L2 error of the complex spectrum (from [n][128] arrays),
    relative to max(||T||, floor*sqrt(nfreq))."""
    nf = ref.shape[1] // 2
    den = np.maximum(np.linalg.norm(ref, axis=1), floor * np.sqrt(nf))
    return np.linalg.norm(pred - ref, axis=1) / den


class FNO:
    """Parameters (FP32 master + BF16 copies) and the forward/backward kernels."""

    def __init__(self, seed: int = 0, device="cuda", nbins: int = NBINS, width: int = WIDTH, modes: int = MODES,
                 layers: int = LAYERS, hidden: int = HIDDEN, out: int = OUT, cin: int = CIN):
        self.dev = torch.device(device)
        self.N, self.C, self.M, self.L, self.H, self.D = nbins, width, modes, layers, hidden, out
        self.cin = cin
        self.fold = True  # inference folds the lift into the first layer (see _refresh_folded)
        g = torch.Generator().manual_seed(seed)
        C, M, H, D = width, modes, hidden, out

        def u(*shape, scale):
            return ((torch.rand(shape, generator=g, dtype=torch.float64) * 2 - 1) * scale).float().to(self.dev)

        self.p = {
            "P": u(C, cin, scale=1.0), "pb": u(C, scale=0.5),
            "H1": u(H, C, scale=1 / math.sqrt(C)), "hb1": u(H, scale=0.1),
            # zero output layer: an untrained network predicts y = 0
            "H2": torch.zeros((D, H), device=self.dev), "hb2": torch.zeros(D, device=self.dev),
        }
        for l in range(layers):
            self.p[f"L{l}.W"] = u(C, C, scale=1 / math.sqrt(C))
            self.p[f"L{l}.b"] = u(C, scale=0.1)
            self.p[f"L{l}.Rr"] = u(M, C, C, scale=1 / C)
            self.p[f"L{l}.Ri"] = u(M, C, C, scale=1 / C)
        phi, psi = dft_matrices(nbins, modes)
        self.phi16 = torch.as_tensor(phi, dtype=torch.float32).to(self.dev).to(BF).contiguous()
        self.psi16 = torch.as_tensor(psi, dtype=torch.float32).to(self.dev).to(BF).contiguous()
        self.g = {k: torch.zeros_like(v) for k, v in self.p.items()}
        self.m = {k: torch.zeros_like(v) for k, v in self.p.items()}
        self.v = {k: torch.zeros_like(v) for k, v in self.p.items()}
        self.step = 0
        self.status = torch.zeros(1, dtype=torch.int32, device=self.dev)  # of every product and fused layer
        self._refresh_bf16()

    # ------------------------------------------------------------ helpers
    def _gemm(self, *args, **kw):
        return gemm(*args, status=self.status, **kw)

    def check(self) -> None:
        """Raise FdtdError if a bounded wait ran out in a tensor-core kernel of this
        network since ``status`` was last zero, whose results are then wrong (host sync)."""
        v = int(self.status.item())
        if v:
            raise _lib.FdtdError(_lib.lib().fdtd_status_to_error(v), f"FNO status word {v:#x}")

    def _refresh_bf16(self):
        self.w16 = {}
        for k in ["H1", "H2"] + [f"L{l}.W" for l in range(self.L)]:
            t = torch.empty(self.p[k].shape, dtype=BF, device=self.dev)
            _call("fno_to_bf16", self.p[k].numel(), self.p[k].data_ptr(), t.data_ptr())
            self.w16[k] = t
        self.rbig = []
        for l in range(self.L):
            t = torch.empty((self.M, 2 * self.C, 2 * self.C), dtype=BF, device=self.dev)
            _call("fno_build_rbig", self.M, self.C, self.p[f"L{l}.Rr"].data_ptr(), self.p[f"L{l}.Ri"].data_ptr(),
                  t.data_ptr())
            self.rbig.append(t)
        self._folded_stale = True  # rebuilt by the next inference forward

    # ------------------------------------------------------------ folded first layer (inference)
    KIN = 16  # packed input width of the DFT operand: cin features, a constant 1, zeros
    KPW = 64  # the pointwise operand is packed 64 wide (128-byte rows load fast through TMA)

    def _refresh_folded(self):
        """The lift x0 = in P^T + p is linear, so inference can skip it: with
        P' = [P | p | 0] ([C][KIN]) and inputs (features, 1, 0...), the first
        layer's pointwise weight becomes W0 P' and its complex mode weights
        R_k P' (FP32 products on the device, then BF16).  The first layer then
        reads 16 input channels instead of a 128-channel activation."""
        C, M, KIN = self.C, self.M, self.KIN
        self._folded_stale = False
        KPW = self.KPW
        Pw = torch.zeros((C, KPW), dtype=torch.float32, device=self.dev)  # assembled by copies
        Pw[:, :self.cin].copy_(self.p["P"])
        Pw[:, self.cin].copy_(self.p["pb"])
        Pp = Pw[:, :KIN].contiguous()
        w0 = torch.empty((C, KPW), dtype=torch.float32, device=self.dev)
        _call("fno_small_matmul", 1, C, KPW, C, self.p["L0.W"].data_ptr(), Pw.data_ptr(), w0.data_ptr())
        self.w0f16 = torch.empty((C, KPW), dtype=BF, device=self.dev)
        _call("fno_to_bf16", w0.numel(), w0.data_ptr(), self.w0f16.data_ptr())
        self.w0k16 = self.w0f16[:, :KIN].contiguous()  # the fused layer's, without the padding
        rr = torch.empty((M, C, KIN), dtype=torch.float32, device=self.dev)
        ri = torch.empty((M, C, KIN), dtype=torch.float32, device=self.dev)
        _call("fno_small_matmul", M, C, KIN, C, self.p["L0.Rr"].data_ptr(), Pp.data_ptr(), rr.data_ptr())
        _call("fno_small_matmul", M, C, KIN, C, self.p["L0.Ri"].data_ptr(), Pp.data_ptr(), ri.data_ptr())
        self.rbig0f = torch.empty((M, 2 * C, 2 * KIN), dtype=BF, device=self.dev)
        _call("fno_build_rbig_rect", M, C, KIN, rr.data_ptr(), ri.data_ptr(), self.rbig0f.data_ptr())

    def _first_modes_folded(self, inp: torch.Tensor, padded: bool):
        """The packed inputs [B][N][KIN] ([B][N][KPW] with ``padded``) and their mode
        coefficients [M][B][2 KIN]."""
        Bn, N, C, M, KIN = inp.shape[0], self.N, self.C, self.M, self.KIN
        dev = self.dev
        # the 64-wide operand lives per (stream, batch size): its zero padding is
        # written once, and each call rewrites only the 16 live columns
        key = (torch.cuda.current_stream(dev).cuda_stream, Bn)
        if not hasattr(self, "_packed"):
            self._packed = {}
        inp16 = self._packed.get(key) if padded else torch.empty((Bn, N, KIN), dtype=BF, device=dev)
        if inp16 is None:
            inp16 = torch.zeros((Bn, N, self.KPW), dtype=BF, device=dev)
            self._packed[key] = inp16
        inpT = torch.empty((N, Bn * KIN), dtype=BF, device=dev)  # position-major copy
        _call("fno_pack_inputs", Bn, N, self.cin, inp16.shape[2], 0, inp.data_ptr(), inp16.data_ptr(), inpT.data_ptr())
        # the DFT of every sample's 16 channels in one product: F[(b, c)][j] = sum_n inpT[n][(b, c)] Phi[j][n]
        F = torch.empty((Bn, KIN, 2 * M), dtype=torch.float32, device=dev)
        self._gemm(inpT, self.phi16, a_mn=True, out=F.view(Bn * KIN, 2 * M))
        Fm = torch.empty((M, Bn, 2 * KIN), dtype=BF, device=dev)
        _call("fno_dft_to_modes", Bn, KIN, M, F.data_ptr(), Fm.data_ptr())
        return inp16, Fm

    def _first_layer_folded(self, inp: torch.Tensor) -> torch.Tensor:
        """x1 of the first spectral layer straight from the packed inputs."""
        Bn, N, C, M, dev = inp.shape[0], self.N, self.C, self.M, self.dev
        inp16, Fm = self._first_modes_folded(inp, True)
        Gm = torch.empty((M, Bn, 2 * C), dtype=torch.float32, device=dev)
        self._gemm(Fm, self.rbig0f, out=Gm)
        G = torch.empty((Bn, C, 2 * M), dtype=BF, device=dev)
        _call("fno_modes_to_dft", Bn, C, M, Gm.data_ptr(), G.data_ptr())
        x = torch.empty((Bn, N, C), dtype=BF, device=dev)
        self._gemm(inp16, self.w0f16, out=x, bias=self.p["L0.b"], gelu=True, second=(self.psi16, G, False, False))
        return x

    # ------------------------------------------------------------ fused layers
    def _fused(self, Bn: int) -> bool:
        """Whether ``fno_layer_fwd`` takes this network and batch."""
        return self.C == 128 and self.M == 32 and self.N >= 128 and self.N & (self.N - 1) == 0 and Bn <= 65535

    def _layers_fused(self, inp: torch.Tensor, saved: dict | None) -> torch.Tensor:
        """h [B][C], the mean of the last layer's output: two launches a layer,
        the mode product and ``fno_layer_fwd``."""
        Bn, N, C, M, dev = inp.shape[0], self.N, self.C, self.M, self.dev
        folded = saved is None and self.fold and self.cin + 1 <= self.KIN
        if folded:
            x, Fm = self._first_modes_folded(inp, False)
        else:
            x = torch.empty((Bn, N, C), dtype=BF, device=dev)
            _call("fno_lift_fwd", Bn * N, C, self.cin, inp.data_ptr(), self.p["P"].data_ptr(),
                  self.p["pb"].data_ptr(), x.data_ptr())
            F = self._gemm(x, self.phi16.unsqueeze(0).expand(Bn, -1, -1), a_mn=True)
            Fm = torch.empty((M, Bn, 2 * C), dtype=BF, device=dev)
            _call("fno_dft_to_modes", Bn, C, M, F.data_ptr(), Fm.data_ptr())
        Gm = torch.empty((M, Bn, 2 * C), dtype=BF, device=dev)
        h = torch.empty((Bn, C), dtype=BF, device=dev)
        for l in range(self.L):
            first, last = folded and l == 0, l == self.L - 1
            self._gemm(Fm, self.rbig0f if first else self.rbig[l], out=Gm)
            w = self.w0k16 if first else self.w16[f"L{l}.W"]
            pre = None
            if saved is not None:
                pre = torch.empty((Bn, N, C), dtype=BF, device=dev)
                for k, v in (("x", x), ("pre", pre), ("Fm", Fm)):
                    saved[k].append(v)
            xn = fn = None
            if not last:
                xn = torch.empty((Bn, N, C), dtype=BF, device=dev)
                fn = torch.empty((M, Bn, 2 * C), dtype=BF, device=dev)
            _call("fno_layer_fwd", Bn, N, C, M, w.shape[1], x.data_ptr(), w.data_ptr(), self.p[f"L{l}.b"].data_ptr(),
                  self.psi16.data_ptr(), Gm.data_ptr(), None if last else xn.data_ptr(),
                  None if last else fn.data_ptr(), h.data_ptr() if last else None,
                  None if pre is None else pre.data_ptr(), self.status.data_ptr())
            x, Fm = xn, fn
        return h

    def state_dict(self):
        return {k: v.detach().cpu().clone() for k, v in self.p.items()}

    def load_state_dict(self, d):
        for k in self.p:
            self.p[k].copy_(d[k].to(self.dev))
        self._refresh_bf16()

    # ------------------------------------------------------------ forward
    def forward(self, inp: torch.Tensor, keep: bool = False) -> torch.Tensor:
        """inp [B][N][cin] float32 (device) -> network output y [B][D] float32."""
        Bn, N, C, M = inp.shape[0], self.N, self.C, self.M
        dev = self.dev
        folded = not keep and self.fold and self.cin + 1 <= self.KIN
        if folded and self._folded_stale:
            self._refresh_folded()
        saved = {"inp": inp, "x": [], "pre": [], "Fm": []}
        if self._fused(Bn) and self.L > 0:
            return self._head(self._layers_fused(inp, saved if keep else None), saved if keep else None)
        phi_b = self.phi16.unsqueeze(0).expand(Bn, -1, -1)  # stride 0 over the batch
        if folded:
            x = self._first_layer_folded(inp)
        else:
            x = torch.empty((Bn, N, C), dtype=BF, device=dev)
            _call("fno_lift_fwd", Bn * N, C, self.cin, inp.data_ptr(), self.p["P"].data_ptr(),
                  self.p["pb"].data_ptr(), x.data_ptr())
        F = torch.empty((Bn, C, 2 * M), dtype=torch.float32, device=dev)
        Fm = torch.empty((M, Bn, 2 * C), dtype=BF, device=dev)
        Gm = torch.empty((M, Bn, 2 * C), dtype=torch.float32, device=dev)
        G = torch.empty((Bn, C, 2 * M), dtype=BF, device=dev)
        for l in range(1 if folded else 0, self.L):
            # truncated DFT: F_b[C][2M] = x_b^T Phi^T   (A = x_b stored [N][C]: MN-major)
            self._gemm(x, phi_b, a_mn=True, out=F)
            _call("fno_dft_to_modes", Bn, C, M, F.data_ptr(), Fm.data_ptr())
            # mode mixing: Gm_k[B][2C] = Fm_k Rbig_k^T
            self._gemm(Fm, self.rbig[l], out=Gm)
            _call("fno_modes_to_dft", Bn, C, M, Gm.data_ptr(), G.data_ptr())
            # pointwise + inverse DFT in one accumulator, then bias and GELU:
            # x'_b = GELU(x_b W^T + Psi G_b^T + b); pre-activation kept for backward
            xn = torch.empty((Bn, N, C), dtype=BF, device=dev)
            pre = torch.empty((Bn, N, C), dtype=BF, device=dev) if keep else None
            self._gemm(x, self.w16[f"L{l}.W"], out=xn, bias=self.p[f"L{l}.b"], gelu=True, pre=pre,
                       second=(self.psi16, G, False, False))
            if keep:
                saved["x"].append(x)
                saved["pre"].append(pre)
                saved["Fm"].append(Fm.clone())
            x = xn
        h = torch.empty((Bn, C), dtype=BF, device=dev)
        _call("fno_meanpool", Bn, N, C, x.data_ptr(), h.data_ptr())
        return self._head(h, saved if keep else None)

    def _head(self, h: torch.Tensor, saved: dict | None) -> torch.Tensor:
        """y [B][D] from the pooled activations h [B][C]."""
        Bn, dev = h.shape[0], self.dev
        a1 = torch.empty((Bn, self.H), dtype=BF, device=dev)
        z1 = torch.empty((Bn, self.H), dtype=BF, device=dev)
        self._gemm(h, self.w16["H1"], out=a1, bias=self.p["hb1"], gelu=True, pre=z1)
        o = torch.empty((Bn, self.D), dtype=torch.float32, device=dev)
        self._gemm(a1, self.w16["H2"], out=o, bias=self.p["hb2"])
        if saved is not None:
            saved.update(h=h, a1=a1, z1=z1)
            self._saved = saved
        return o

    # ------------------------------------------------------------ backward
    def backward(self, dO: torch.Tensor) -> None:
        """Accumulate parameter gradients into self.g from dL/do [B][D] (float32)."""
        s = self._saved
        Bn, N, C, M, H, D = dO.shape[0], self.N, self.C, self.M, self.H, self.D
        dev = self.dev
        for k in self.g:
            self.g[k].zero_()
        dO16 = torch.empty((Bn, D), dtype=BF, device=dev)
        _call("fno_to_bf16", dO.numel(), dO.data_ptr(), dO16.data_ptr())
        # head
        self._gemm(dO16, s["a1"], a_mn=True, b_mn=True, out=self.g["H2"])       # dH2 = dO^T a1
        _call("fno_colsum", Bn, D, None, dO.data_ptr(), self.g["hb2"].data_ptr())
        da1 = self._gemm(dO16, self.w16["H2"], b_mn=True)                       # da1 = dO H2  [B][H]
        dz1 = torch.empty((Bn, H), dtype=BF, device=dev)
        _call("fno_gelu_bwd", Bn * H, None, da1.data_ptr(), s["z1"].data_ptr(), dz1.data_ptr())
        self._gemm(dz1, s["h"], a_mn=True, b_mn=True, out=self.g["H1"])         # dH1 = dz1^T h
        _call("fno_colsum", Bn, H, dz1.data_ptr(), None, self.g["hb1"].data_ptr())
        dh = self._gemm(dz1, self.w16["H1"], b_mn=True)                         # dh = dz1 H1  [B][C]
        wide = C % 8 == 0 and C <= 2048  # the fused kernels' channel groups
        dx16 = dx32 = None
        if not wide:
            dx16 = torch.empty((Bn, N, C), dtype=BF, device=dev)
            _call("fno_meanpool_bwd", Bn, N, C, dh.data_ptr(), dx16.data_ptr())
        parts = torch.empty((Bn, C, C), dtype=torch.float32, device=dev)
        dG = torch.empty((Bn, C, 2 * M), dtype=torch.float32, device=dev)
        dGm = torch.empty((M, Bn, 2 * C), dtype=BF, device=dev)
        dFm = torch.empty((M, Bn, 2 * C), dtype=torch.float32, device=dev)
        dF = torch.empty((Bn, C, 2 * M), dtype=BF, device=dev)
        dRbig = torch.empty((M, 2 * C, 2 * C), dtype=torch.float32, device=dev)
        # the input gradient of a layer leaves its product as the next layer's dz, GELU backward
        # and bias sum included, where the GEMM has that epilogue
        chained = C == 128 and N % 128 == 0
        dz = torch.empty((Bn, N, C), dtype=BF, device=dev)
        dz2 = torch.empty_like(dz) if chained else None
        psi_b = self.psi16.unsqueeze(0).expand(Bn, -1, -1)
        for l in reversed(range(self.L)):
            x, pre, Fm = s["x"][l], s["pre"][l], s["Fm"][l]
            p16, p32 = None if dx16 is None else dx16.data_ptr(), None if dx32 is None else dx32.data_ptr()
            if chained and l < self.L - 1:
                pass  # dz and its sum came with layer l + 1
            elif wide:
                _call("fno_gelu_bwd_sum", Bn * N, C, N, None, p32, dh.data_ptr() if p32 is None else None,
                      pre.data_ptr(), dz.data_ptr(), self.g[f"L{l}.b"].data_ptr())
            else:
                _call("fno_gelu_bwd", dz.numel(), p16 if p32 is None else None, p32, pre.data_ptr(), dz.data_ptr())
                _call("fno_colsum", Bn * N, C, dz.data_ptr(), None, self.g[f"L{l}.b"].data_ptr())
            # dW = sum_b dz_b^T x_b  (per-sample products, then summed)
            self._gemm(dz, x, a_mn=True, b_mn=True, out=parts)
            _call("fno_sum_parts", Bn, C * C, parts.data_ptr(), self.g[f"L{l}.W"].data_ptr())
            # spectral branch: dG_b = dz_b^T Psi ; dFm_k = dGm_k Rbig_k ; dRbig_k = dGm_k^T Fm_k
            self._gemm(dz, psi_b, a_mn=True, b_mn=True, out=dG)
            _call("fno_dft_to_modes", Bn, C, M, dG.data_ptr(), dGm.data_ptr())
            self._gemm(dGm, self.rbig[l], b_mn=True, out=dFm)
            self._gemm(dGm, Fm, a_mn=True, b_mn=True, out=dRbig)
            _call("fno_fold_drbig", M, C, dRbig.data_ptr(), self.g[f"L{l}.Rr"].data_ptr(), self.g[f"L{l}.Ri"].data_ptr())
            _call("fno_modes_to_dft", Bn, C, M, dFm.data_ptr(), dF.data_ptr())
            # dx = dz W + Phi^T dF^T in one accumulator (Phi stored [2M][N]: MN-major, shared)
            if chained and l > 0:
                self._gemm(dz, self.w16[f"L{l}.W"], b_mn=True, out=dz2, second=(self.phi16, dF, True, False),
                           gelu_bwd=(s["pre"][l - 1], self.g[f"L{l - 1}.b"]))
                dz, dz2 = dz2, dz
                continue
            nd = torch.empty((Bn, N, C), dtype=torch.float32, device=dev)
            self._gemm(dz, self.w16[f"L{l}.W"], b_mn=True, out=nd, second=(self.phi16, dF, True, False))
            dx32 = nd
        if wide:
            _call("fno_lift_bwd32", Bn * N, C, self.cin, s["inp"].data_ptr(), dx32.data_ptr(), self.g["P"].data_ptr(),
                  self.g["pb"].data_ptr())
            return
        dx0 = torch.empty((Bn, N, C), dtype=BF, device=dev)
        _call("fno_to_bf16", dx32.numel(), dx32.data_ptr(), dx0.data_ptr())
        _call("fno_lift_bwd", Bn * N, C, self.cin, s["inp"].data_ptr(), dx0.data_ptr(), self.g["P"].data_ptr(),
              self.g["pb"].data_ptr())

    def adam_step(self, lr: float = 1e-3, b1: float = 0.9, b2: float = 0.999, eps: float = 1e-8) -> None:
        self.step += 1
        for k in self.p:
            _call("fno_adam", self.p[k].numel(), self.p[k].data_ptr(), self.g[k].data_ptr(), self.m[k].data_ptr(),
                  self.v[k].data_ptr(), lr, b1, b2, eps, self.step, None)
        self._refresh_bf16()

    def loss_and_grad(self, inp: torch.Tensor, target: torch.Tensor, relative: bool = False,
                      frame: torch.Tensor | None = None) -> torch.Tensor:
        """Forward, loss and backward.  With ``frame`` P the loss is taken on
        T = P (.) y (and dL/dy = conj(P) (.) dL/dT); ``relative`` uses the
        per-sample relative squared error with the spectrum floor (the metric
        the judge applies), otherwise the plain mean squared error."""
        y = self.forward(inp, keep=True)
        o = y if frame is None else cmul(frame, y)
        dO = torch.empty_like(o)
        loss = torch.zeros(1, dtype=torch.float32, device=self.dev)
        if relative:
            floor2 = float(SPECTRUM_FLOOR ** 2 * (o.shape[1] // 2))
            _call("fno_rel_mse", o.shape[0], o.shape[1], floor2, o.data_ptr(), target.data_ptr(), dO.data_ptr(),
                  loss.data_ptr())
        else:
            _call("fno_mse", o.shape[0], o.shape[1], o.data_ptr(), target.data_ptr(), dO.data_ptr(),
                  loss.data_ptr())
        self.backward(dO if frame is None else cmul(frame, dO, conj=True))
        return loss

    def predict(self, inp: torch.Tensor, chunk: int = 4096) -> torch.Tensor:
        """Network output y for [B][N][cin] inputs, ``chunk`` profiles per pass."""
        outs = [self.forward(inp[i:i + chunk]) for i in range(0, inp.shape[0], chunk)]
        return torch.cat(outs) if len(outs) > 1 else outs[0]

    def spectrum(self, inp: torch.Tensor, chunk: int = 4096, streams: int = 3) -> torch.Tensor:
        """Predicted transmission [B][2*NFREQ] = [Re T | Im T] = P (.) y.

        Chunks alternate between ``streams`` CUDA streams, so that one chunk's
        lighter kernels (permutes, frame, head) overlap another's GEMMs."""
        main = torch.cuda.current_stream(self.dev)
        # shared tables are made on the caller's stream, before any side stream reads them
        _wdt_table(inp.device)
        if self.fold and self._folded_stale and self.cin + 1 <= self.KIN:
            self._refresh_folded()
        nchunk = -(-inp.shape[0] // chunk)
        if nchunk == 1 or streams <= 1:
            outs = [cmul(propagation(inp[i:i + chunk]), self.forward(inp[i:i + chunk]))
                    for i in range(0, inp.shape[0], chunk)]
            return torch.cat(outs) if len(outs) > 1 else outs[0]
        if not hasattr(self, "_streams") or len(self._streams) < streams:
            self._streams = [torch.cuda.Stream(device=self.dev) for _ in range(streams)]
        outs = []
        for k, i in enumerate(range(0, inp.shape[0], chunk)):
            st = self._streams[k % streams]
            st.wait_stream(main)  # the input (and anything before this call) is ready
            with torch.cuda.stream(st):
                part = inp[i:i + chunk]
                o = cmul(propagation(part), self.forward(part))
            o.record_stream(main)  # read by the concatenation on the caller's stream
            outs.append(o)
        for st in self._streams[:streams]:
            main.wait_stream(st)
        return torch.cat(outs)


# ------------------------------------------------------------------ data and serving
def solve_fdtd(batch: "B1.SlabBatch", nsteps: int = NSTEPS, chunk: int = 4096, device="cuda") -> np.ndarray:
    """[n][128] transmission spectra of ``batch`` from the batched FDTD kernel."""
    out = np.zeros((batch.nruns, OUT), dtype=np.float32)
    for s in range(0, batch.nruns, chunk):
        idx = np.arange(s, min(batch.nruns, s + chunk))
        r = B1.BatchRunner(batch.subset(idx), nsteps=nsteps, freqs=FREQS, wave=WAVE, device=device)
        r.run()
        out[idx] = spectrum_targets(r.transmission())
    return out


def solve_fdtd_device(batch: "B1.SlabBatch", nsteps: int = NSTEPS, device="cuda") -> torch.Tensor:
    """``solve_fdtd`` left on the device, enqueued on the current stream: [n][128]."""
    r = B1.BatchRunner(batch, nsteps=nsteps, freqs=FREQS, wave=WAVE, device=device)
    r.run()
    return r.spectrum()


def rel_l2_spectrum_device(pred: torch.Tensor, ref: torch.Tensor, floor: float = SPECTRUM_FLOOR) -> torch.Tensor:
    """``rel_l2_spectrum`` on device tensors (float64 norms)."""
    nf = ref.shape[1] // 2
    den = torch.clamp(torch.linalg.vector_norm(ref.double(), dim=1), min=floor * math.sqrt(nf))
    return torch.linalg.vector_norm((pred - ref).double(), dim=1) / den


def generate_dataset(n: int, seed: int, nsteps: int = NSTEPS, chunk: int = 4096, device="cuda",
                     on_device: bool = False):
    """Slab runs of the batched-FDTD distribution solved by the batched kernel:
    returns (inputs [n][NBINS][6], targets [n][128], batch), as host arrays,
    or (on_device) as device tensors built and kept on the GPU."""
    batch = B1.slab_batch(n, seed=seed)
    if np.any(batch.probe_in != PROBE_IN) or np.any(batch.probe_out != batch.layer_end[batch.layer_off[1:] - 1]
                                                    + PROBE_GAP):
        raise ValueError("probe placement differs from the surrogate's frame")
    if not on_device:
        return profile_features(batch), solve_fdtd(batch, nsteps, chunk, device), batch
    Y = torch.empty((n, OUT), dtype=torch.float32, device=device)
    for s in range(0, n, chunk):
        idx = np.arange(s, min(n, s + chunk))
        Y[s:s + idx.size] = solve_fdtd_device(batch.subset(idx), nsteps, device=device)
    return device_features(batch, device=device), Y, batch


def train(model: FNO, inp: np.ndarray, tgt: np.ndarray, samples: int = 200_000, batch: int = 256,
          lr: float = 1e-3, lr_final: float = 1e-3, seed: int = 0, log_every: int = 100) -> list:
    """Adam on random minibatches until ``samples`` samples have been seen; the
    loss is the relative spectrum error of T = P (.) y.  The learning rate
    follows a cosine from ``lr`` to ``lr_final``."""
    rng = np.random.default_rng(seed)
    dev = model.dev
    X = torch.as_tensor(inp).to(dev)
    Y = torch.as_tensor(tgt).to(dev)
    frames = torch.cat([propagation(X[i:i + 65536]) for i in range(0, X.shape[0], 65536)])
    hist = []
    steps = max(1, samples // batch)
    for it in range(steps):
        idx = torch.as_tensor(rng.integers(0, X.shape[0], size=batch)).to(dev)
        loss = model.loss_and_grad(X.index_select(0, idx).contiguous(), Y.index_select(0, idx).contiguous(),
                                   relative=True, frame=frames.index_select(0, idx).contiguous())
        a = 0.5 * (1 + math.cos(math.pi * it / max(1, steps - 1)))
        model.adam_step(lr_final + (lr - lr_final) * a)
        if it % log_every == 0 or it == steps - 1:
            hist.append((it, float(loss.item())))
            model.check()
    return hist


def damping_gate(batch: "B1.SlabBatch", layer_max: float = 1.0, total_max: float = 6.0) -> np.ndarray:
    """[n] bool: profiles whose spectrum carries internal echoes.  A layer with
    sigma*d/sqrt(eps_r) < ``layer_max`` (S/m x cells; one pass attenuates by
    exp(-1.885 x that)) keeps its multiple reflections, and they show in T when
    the whole stack is transparent enough (sum < ``total_max``).  The network
    resolves the single-pass interface physics but not those echo trains
    (phases 2 k d of up to ~10^3 rad), so a gated server sends such profiles to
    the FDTD.  Decided from the profile alone, before anything is solved."""
    out = np.zeros(batch.nruns, dtype=bool)
    for r in range(batch.nruns):
        a, b = batch.layer_off[r], batch.layer_off[r + 1]
        d = (batch.layer_end[a:b] - batch.layer_start[a:b]).astype(np.float64)
        damp = batch.sigma[a:b] * d / np.sqrt(batch.epsr[a:b])
        out[r] = damp.min() < layer_max and damp.sum() < total_max
    return out


class JudgedSurrogate:
    """Surrogate predictions with batched FDTD as judge and fallback: a
    fraction of each request is re-solved by FDTD; a spot-checked profile whose
    error exceeds ``tol`` is replaced by its FDTD spectrum.  With ``gate`` =
    (layer_max, total_max), profiles selected by ``damping_gate`` skip the
    network and are solved by FDTD directly.

    Everything stays on the device: the inputs are built there from the layer
    tables (``device_features``).  The network is enqueued first; the FDTD
    runs of the spot check (and of the gated profiles) are then prepared on
    the host while it runs and enqueued on a second stream, so the two
    overlap; the replacement waits for both."""

    def __init__(self, model: FNO, check_frac: float = 0.01, tol: float = 0.01, nsteps: int = NSTEPS, seed: int = 0,
                 gate: tuple | None = None):
        self.model, self.check_frac, self.tol, self.nsteps = model, check_frac, tol, nsteps
        self.gate = gate
        self.rng = np.random.default_rng(seed)
        self._side = None

    def __call__(self, batch: "B1.SlabBatch", inp: torch.Tensor | None = None):
        """(pred [n][128] device tensor, info).  ``inp``: the batch's inputs
        already on the device (built here otherwise)."""
        dev = self.model.dev
        n = batch.nruns
        routed = damping_gate(batch, *self.gate) if self.gate else np.zeros(n, dtype=bool)
        served = np.nonzero(~routed)[0]
        routed_idx = np.nonzero(routed)[0]
        k = max(1, int(round(self.check_frac * served.size))) if served.size else 0
        idx = np.sort(self.rng.choice(served, size=min(k, served.size), replace=False)) if k else served[:0]
        main = torch.cuda.current_stream(dev)
        if self._side is None:
            self._side = torch.cuda.Stream(device=dev)
        side = self._side
        side.wait_stream(main)
        pred = torch.zeros((n, OUT), dtype=torch.float32, device=dev)
        if served.size:  # the network, enqueued first: the GPU runs it while the host prepares the judge
            sv = torch.as_tensor(served, device=dev)
            if inp is None:
                x = device_features(batch, served, nbins=self.model.N, device=dev)
            else:
                x = inp.index_select(0, sv).contiguous()
            pred.index_copy_(0, sv, self.model.spectrum(x))
        ref = fall = None
        with torch.cuda.stream(side):  # the judge's FDTD, overlapping the network
            if idx.size:
                ref = solve_fdtd_device(batch.subset(idx), self.nsteps, device=dev)
            if routed_idx.size:
                fall = solve_fdtd_device(batch.subset(routed_idx), self.nsteps, device=dev)
        main.wait_stream(side)
        for t in (ref, fall):
            if t is not None:
                t.record_stream(main)
        info = {"routed": int(routed.sum()), "checked": int(idx.size), "fell_back": 0, "checked_idx": idx}
        if routed_idx.size:
            pred.index_copy_(0, torch.as_tensor(routed_idx, device=dev), fall)
        if idx.size:
            ci = torch.as_tensor(idx, device=dev)
            err = rel_l2_spectrum_device(pred.index_select(0, ci), ref)
            bad = err > self.tol
            pred.index_copy_(0, ci, torch.where(bad[:, None], ref, pred.index_select(0, ci)))
            e = err.cpu().numpy()
            self.model.check()
            info.update(check_err_median=float(np.median(e)), check_err_p90=float(np.quantile(e, 0.9)),
                        fell_back=int((e > self.tol).sum()))
        return pred, info


def time_served(model: FNO, batch: "B1.SlabBatch", check_frac: float = 0.01, tol: float = 0.01, reps: int = 1,
                seed: int = 0) -> dict:
    """Spectra per second of the judged server on ``batch`` (one request of
    batch.nruns profiles): inputs built on the device, network, frame and
    product, the 1% FDTD spot check overlapping them, replacements; timed
    with CUDA events around whole requests (host work included)."""
    judge = JudgedSurrogate(model, check_frac=check_frac, tol=tol, seed=seed)
    judge(batch)  # warm-up: plans, buffers, module loads
    st = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record(st)
    for _ in range(reps):
        pred, info = judge(batch)
    e1.record(st)
    torch.cuda.synchronize()
    return {"spectra_per_s": reps * batch.nruns / (e0.elapsed_time(e1) / 1e3), "checked": info["checked"],
            "fell_back": info["fell_back"], "pred": pred}


def time_inference(model: FNO, n: int = 65536, chunk: int = 4096, reps: int = 2, seed: int = 0) -> float:
    """Spectra per second of the served path (network, frame and product) at
    batch ``n``, timed with CUDA events on the current stream.  Inputs are
    ``chunk`` seeded slab profiles reused for every chunk: the network's cost
    does not depend on the values; the frame's grows with the number of
    material changes along a profile (a few per layered stack)."""
    one = torch.as_tensor(profile_features(B1.slab_batch(chunk, seed=seed), nbins=model.N)).to(model.dev)
    inp = one.repeat((max(1, n // chunk), 1, 1))  # n profiles in HBM, served in chunks
    model.spectrum(inp, chunk=chunk)
    st = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record(st)
    for _ in range(reps):
        model.spectrum(inp, chunk=chunk)
    e1.record(st)
    torch.cuda.synchronize()
    return reps * inp.shape[0] / (e0.elapsed_time(e1) / 1e3)


def flops_per_sample(model: FNO) -> float:
    """Tensor-core FLOPs of one forward pass (the GEMMs)."""
    N, C, M, H, D = model.N, model.C, model.M, model.H, model.D
    per_layer = 2 * N * C * 2 * M + 2 * M * (2 * C) * (2 * C) + 2 * N * C * (C + 2 * M)
    return model.L * per_layer + 2 * C * H + 2 * H * D


def main(argv=None) -> None:
    """Train on batched-FDTD data, evaluate on held-out profiles and serve them
    through the judge, with and without the damping gate; prints one JSON line.

    python -m simulation_gb300.surrogate [--train 200000] [--samples 2000000] [--test 4096]
    """
    import argparse
    import json
    ap = argparse.ArgumentParser()
    ap.add_argument("--train", type=int, default=200_000, help="training profiles (batched-FDTD runs)")
    ap.add_argument("--samples", type=int, default=2_000_000, help="minibatch samples seen in training")
    ap.add_argument("--test", type=int, default=4096, help="held-out profiles")
    ap.add_argument("--seed", type=int, default=100)
    ap.add_argument("--save", default=None, help="write the trained parameters here (torch.save)")
    args = ap.parse_args(argv)
    ev = lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731
    e0, e1 = ev(), ev()
    e0.record()
    X, Y, batch = generate_dataset(args.train + args.test, seed=args.seed)
    e1.record()
    torch.cuda.synchronize()
    out = {"train_profiles": args.train, "test_profiles": args.test, "samples_seen": args.samples,
           "dataset_s": e0.elapsed_time(e1) / 1e3}
    m = FNO(seed=0)
    e0.record()
    hist = train(m, X[:args.train], Y[:args.train], samples=args.samples, lr=1e-3, lr_final=1e-5, log_every=1000)
    e1.record()
    torch.cuda.synchronize()
    out["train_s"] = e0.elapsed_time(e1) / 1e3
    out["loss_first_last"] = [hist[0][1], hist[-1][1]]
    if args.save:
        torch.save(m.state_dict(), args.save)
    Yte = Y[args.train:]
    test = batch.subset(np.arange(args.train, args.train + args.test))
    Xd = torch.as_tensor(X[args.train:]).to(m.dev)
    big = np.linalg.norm(Yte, axis=1) > SPECTRUM_FLOOR * np.sqrt(NFREQ)

    def summary(err):
        return {"median": float(np.median(err)), "p90": float(np.quantile(err, 0.9)),
                "frac_le_1pct": float(np.mean(err <= 0.01)), "frac_le_5pct": float(np.mean(err <= 0.05)),
                "transmissive_median": float(np.median(err[big])),
                "transmissive_frac_le_1pct": float(np.mean(err[big] <= 0.01))}

    P = propagation(Xd)
    ones = torch.zeros_like(P)
    ones[:, :NFREQ] = 1.0
    out["transmissive_fraction"] = float(big.mean())
    out["baseline_zero"] = summary(rel_l2_spectrum(np.zeros_like(Yte), Yte))
    out["baseline_frame_only"] = summary(rel_l2_spectrum(cmul(P, ones).cpu().numpy(), Yte))
    out["network"] = summary(rel_l2_spectrum(m.spectrum(Xd).cpu().numpy(), Yte))
    m.check()
    for name, gate in (("judged", None), ("judged_gated", (1.0, 6.0))):
        judge = JudgedSurrogate(m, check_frac=0.01, tol=0.01, gate=gate, seed=1)
        judge(test, Xd)  # warm-up (plans, buffers)
        torch.cuda.synchronize()
        e0.record()
        pred, info = judge(test, Xd)
        e1.record()
        torch.cuda.synchronize()
        err = rel_l2_spectrum(pred.cpu().numpy(), Yte)
        out[name] = {**summary(err), "routed": info["routed"], "checked": info["checked"],
                     "fell_back": info["fell_back"], "spectra_per_s": args.test / (e0.elapsed_time(e1) / 1e3)}
    e0.record()
    solve_fdtd(test)
    e1.record()
    torch.cuda.synchronize()
    out["fdtd_spectra_per_s"] = args.test / (e0.elapsed_time(e1) / 1e3)
    out["network_spectra_per_s"] = time_inference(m, n=65536, chunk=4096, reps=1)
    print(json.dumps(out), flush=True)


if __name__ == "__main__":
    main()
