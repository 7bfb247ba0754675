"""Learned surrogate for the fitness mode (parameter estimation).

The reference computes the fitness of every candidate parameter set by full
simulation (kernel.cu:365-423, calculateFitness 2phase_n-tau-leaping.cu:
3324-3408).  Here a small MLP, trained on trajectories the simulator itself
produces, screens candidates first; every retained candidate is re-simulated
with the plain method, which also measures the surrogate's error.

Network: x = (8 scaled log rate constants, scaled t) -> 256 -> 256 -> 256 ->
256 -> 2*S (per-species mean and log-variance of the standardised counts),
SiLU, BF16 weights and activations, FP32 accumulation and master weights,
Gaussian negative log-likelihood, Adam.  A training step runs in the project's
own fused tcgen05 kernels (ctl_mlp_forward, ctl_mlp_backward) and Adam in one
launch (ctl_mlp_adam_step); single products are ctl_mlp_gemm.  Screening runs
the whole network and the fitness in one fused tcgen05 kernel
(ctl_mlp_screen, `screen`).  PyTorch only provides device memory.
"""
from __future__ import annotations

import ctypes as C
import math
from dataclasses import dataclass

import numpy as np

from . import CtlError, OK, lib

EPI_ATOMIC_F32, EPI_BIAS_SILU, EPI_BIAS, EPI_SILU_GRAD, EPI_F32 = range(5)
IN_PAD = 64      # 9 inputs padded to one K tile
HIDDEN = 256
LAYERS = 4       # hidden layers of width 256


class GemmDesc(C.Structure):
    _fields_ = [("A", C.c_void_p), ("B", C.c_void_p), ("lda", C.c_int32), ("ldb", C.c_int32),
                ("M", C.c_int32), ("N", C.c_int32), ("K", C.c_int32), ("epilogue", C.c_int32),
                ("splits", C.c_int32), ("bias", C.c_void_p), ("z_in", C.c_void_p), ("ldz", C.c_int32),
                ("out_f32", C.c_void_p), ("ldo", C.c_int32), ("out_bf", C.c_void_p), ("ldob", C.c_int32),
                ("out_bfT", C.c_void_p), ("ldobT", C.c_int32), ("err", C.c_void_p)]


class ScreenDesc(C.Structure):
    _fields_ = [("theta", C.c_void_p), ("n_par", C.c_int32), ("n_cand", C.c_uint32), ("tvec", C.c_void_p),
                ("ns", C.c_uint32), ("t_end", C.c_float), ("log_lo", C.c_void_p), ("log_hi", C.c_void_p),
                ("y_mean", C.c_void_p), ("y_std", C.c_void_p), ("S", C.c_int32), ("out_w", C.c_int32),
                ("target", C.c_void_p), ("wpack", C.c_void_p), ("bias", C.c_void_p), ("fitness", C.c_void_p),
                ("err", C.c_void_p)]


class StepDesc(C.Structure):
    _fields_ = [("X", C.c_void_p), ("W", C.c_void_p * 5), ("WT", C.c_void_p * 5), ("bias", C.c_void_p * 5),
                ("z", C.c_void_p * 4), ("y", C.c_void_p), ("hp", C.c_void_p * 5), ("dp", C.c_void_p * 5),
                ("wpack", C.c_void_p), ("target", C.c_void_p), ("loss", C.c_void_p), ("dW", C.c_void_p * 5),
                ("db", C.c_void_p * 5), ("B", C.c_int32), ("S", C.c_int32), ("out_w", C.c_int32), ("err", C.c_void_p)]


class AdamDesc(C.Structure):
    _fields_ = [(k, C.c_void_p * 5) for k in ("w", "b", "g", "gb", "m", "v", "mb", "vb", "wb", "wbT")] + \
        [("out_w", C.c_int32), ("step", C.c_int32)] + \
        [(k, C.c_float) for k in ("lr", "beta1", "beta2", "eps", "weight_decay")]


def _bind():
    L = lib()
    if not getattr(L, "_mlp_bound", False):
        P = C.c_void_p
        L.ctl_mlp_pack_bytes.argtypes = [C.c_int32]
        L.ctl_mlp_pack_bytes.restype = C.c_size_t
        L.ctl_mlp_pack.argtypes = [C.POINTER(C.c_void_p), C.POINTER(C.c_int32), C.c_int32, P, P]
        L.ctl_mlp_screen.argtypes = [C.POINTER(ScreenDesc), P]
        L.ctl_mlp_gemm.argtypes = [C.POINTER(GemmDesc), P]
        L.ctl_mlp_nll_grad.argtypes = [P, C.c_int32, P, C.c_int32, C.c_int32, P, C.c_int32, P, C.c_int32, P, P]
        L.ctl_mlp_colsum.argtypes = [P, C.c_int32, C.c_int32, C.c_int32, P, P]
        L.ctl_mlp_adam.argtypes = [P, P, P, P, C.c_int32, C.c_int32, C.c_float, C.c_float, C.c_float,
                                   C.c_float, C.c_int32, C.c_float, P, P, P]
        L.ctl_mlp_forward.argtypes = [C.POINTER(StepDesc), P]
        L.ctl_mlp_backward.argtypes = [C.POINTER(StepDesc), P]
        L.ctl_mlp_adam_step.argtypes = [C.POINTER(AdamDesc), P]
        L._mlp_bound = True
    return L


def _ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _stream():
    import torch
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def gemm(A, B, *, epilogue, out_f32=None, out_bf=None, out_bfT=None, bias=None, z_in=None,
         splits=1, err=None):
    """C = A . B^T (A [M][K], B [N][K], BF16 torch tensors) on the tcgen05 kernel."""
    L = _bind()
    M, K = A.shape
    N, K2 = B.shape
    assert K == K2
    d = GemmDesc(_ptr(A), _ptr(B), A.stride(0), B.stride(0), M, N, K, epilogue, splits,
                 _ptr(bias), _ptr(z_in), 0 if z_in is None else z_in.stride(0),
                 _ptr(out_f32), 0 if out_f32 is None else out_f32.stride(0),
                 _ptr(out_bf), 0 if out_bf is None else out_bf.stride(0),
                 _ptr(out_bfT), 0 if out_bfT is None else out_bfT.stride(0), _ptr(err))
    st = L.ctl_mlp_gemm(C.byref(d), _stream())
    if st != OK:
        raise CtlError(st, "ctl_mlp_gemm")


@dataclass
class Scaling:
    """Input and output scaling of the surrogate."""
    log_lo: np.ndarray      # [8] log of the prior box low end
    log_hi: np.ndarray      # [8]
    t_end: float
    y_mean: np.ndarray      # [S] per-species mean count
    y_std: np.ndarray       # [S]


def make_inputs(theta_log, t, sc: Scaling, torch_mod):
    """X [n][64] BF16: scaled log rate constants in [-1, 1], scaled time, zeros."""
    torch = torch_mod
    n = theta_log.shape[0]
    X = torch.zeros((n, IN_PAD), dtype=torch.float32, device="cuda")
    lo = torch.as_tensor(sc.log_lo, dtype=torch.float32, device="cuda")
    hi = torch.as_tensor(sc.log_hi, dtype=torch.float32, device="cuda")
    X[:, :8] = 2.0 * (theta_log - lo) / (hi - lo) - 1.0
    X[:, 8] = 2.0 * t / sc.t_end - 1.0
    return X.to(torch.bfloat16)


class MLP:
    """9 -> 256 x 4 -> 2S surrogate with its own tcgen05 forward/backward."""

    def __init__(self, S: int, seed: int = 0):
        import torch
        self.torch = torch
        self.S = S
        if 2 * S > 128:
            raise ValueError("the surrogate predicts at most 64 species")
        self.out_w = max(64, (2 * S + 63) // 64 * 64)  # output layer padded to a K tile
        self.dims = [IN_PAD] + [HIDDEN] * LAYERS + [self.out_w]
        g = torch.Generator(device="cpu").manual_seed(seed)
        self.W, self.b, self.Wb, self.WbT, self.m, self.v, self.mb, self.vb = ([] for _ in range(8))
        for l in range(len(self.dims) - 1):
            fan_in, fan_out = (9 if l == 0 else self.dims[l]), self.dims[l + 1]
            w = torch.zeros(fan_out, self.dims[l])
            live = 2 * S if l == len(self.dims) - 2 else fan_out  # padded outputs stay zero
            w[:live, :fan_in] = torch.randn(live, fan_in, generator=g) * math.sqrt(1.0 / fan_in)
            if l == len(self.dims) - 2:
                w *= 0.1
            w = w.cuda()
            self.W.append(w)
            self.b.append(torch.zeros(fan_out, device="cuda"))
            self.Wb.append(w.to(torch.bfloat16).contiguous())
            self.WbT.append(w.t().contiguous().to(torch.bfloat16))
            self.m.append(torch.zeros_like(w))
            self.v.append(torch.zeros_like(w))
            self.mb.append(torch.zeros(fan_out, device="cuda"))
            self.vb.append(torch.zeros(fan_out, device="cuda"))
        self.step_count = 0   # Adam's bias-correction step
        self.version = 0      # changes with every weight update (keys the packed copy)
        self.err = torch.zeros(1, dtype=torch.int32, device="cuda")
        self._bufs = {}

    # -- buffers ---------------------------------------------------------------
    def _buf(self, name, shape, dtype):
        t = self._bufs.get(name)
        if t is None or t.shape != shape or t.dtype != dtype:
            t = self.torch.empty(shape, dtype=dtype, device="cuda")
            self._bufs[name] = t
        return t

    def forward(self, X, keep=True):
        """X [B][64] BF16 (B % 128 == 0) -> y [B][out_w] FP32, in one kernel
        (ctl_mlp_forward).  With `keep`, what backward needs is kept too: the
        pre-activations and the packed layer inputs."""
        torch = self.torch
        L = _bind()
        assert X.shape[1] == IN_PAD
        X = X.contiguous()
        Bn = X.shape[0]
        self.z = self._buf("z", (LAYERS, Bn, HIDDEN), torch.float32)
        self.hp = self._buf("hp", (Bn * (IN_PAD + LAYERS * HIDDEN),), torch.bfloat16) if keep else None
        y = self._buf("y", (Bn, self.out_w), torch.float32)
        d = StepDesc()
        d.X, d.y, d.wpack, d.err = X.data_ptr(), y.data_ptr(), self._wstage().data_ptr(), self.err.data_ptr()
        d.W[:], d.bias[:] = [w.data_ptr() for w in self.Wb], [v.data_ptr() for v in self.b]
        d.z[:] = self._z_ptrs(Bn)
        if keep:
            d.hp[:] = self._hp_ptrs(Bn)
        d.B, d.out_w = Bn, self.out_w
        st = L.ctl_mlp_forward(C.byref(d), _stream())
        if st != OK:
            raise CtlError(st, "ctl_mlp_forward")
        return y

    # where each layer's part lies in the buffers: FP32 pre-activations, packed layer inputs
    def _z_ptrs(self, Bn):
        z = self.z.data_ptr()
        return [z + l * Bn * HIDDEN * 4 for l in range(LAYERS)]

    def _hp_ptrs(self, Bn):
        h = self.hp.data_ptr()
        return [h] + [h + Bn * (IN_PAD + l * HIDDEN) * 2 for l in range(LAYERS)]

    def _wstage(self):
        L = _bind()
        return self._buf("wstage", (L.ctl_mlp_pack_bytes(self.out_w) // 2,), self.torch.bfloat16)

    def backward(self, y, target):
        """Gaussian NLL of y = [mu | log var | ...] (FP32 [B][2S or more], any
        row stride) against target [B][S] (FP32); returns (loss sum, gradients
        dW[l], db[l])."""
        torch = self.torch
        L = _bind()
        Bn, S = target.shape
        if Bn != self.z.shape[1]:
            raise ValueError("backward: another batch size than the last forward's")
        if y.dim() != 2 or y.shape[0] != Bn or y.shape[1] < 2 * S:
            raise ValueError("backward: y must be [B][2S] or wider, as forward returns it")
        if any(t.dtype != torch.float32 or t.device != self.err.device for t in (y, target)):
            raise ValueError("backward: y and target must be FP32 tensors on the network's device")
        # the kernel steps y by rows of out_w floats from a 32-byte boundary
        if y.shape[1] != self.out_w or not y.is_contiguous() or y.data_ptr() % 32:
            w = min(2 * S, self.out_w)
            rows = self._buf("y_rows", (Bn, self.out_w), torch.float32)
            rows[:, :w].copy_(y[:, :w])
            y = rows
        target = target.contiguous()
        # loss and gradients in one zeroed allocation (they are accumulated)
        sizes = [w.numel() for w in self.W] + [b.numel() for b in self.b] + [1]
        parts = torch.zeros(sum(sizes), device="cuda").split(sizes)
        dW = [g.view(w.shape) for g, w in zip(parts, self.W)]
        db, loss = list(parts[len(dW):-1]), parts[-1]
        d = StepDesc()
        d.y, d.target, d.loss, d.wpack = y.data_ptr(), target.data_ptr(), loss.data_ptr(), self._wstage().data_ptr()
        d.WT[:], d.hp[:], d.z[:] = [w.data_ptr() for w in self.WbT], self._hp_ptrs(Bn), self._z_ptrs(Bn)
        dp = self._buf("dp", (Bn * (LAYERS * HIDDEN + 128),), torch.bfloat16).data_ptr()
        d.dp[:] = [dp + l * Bn * HIDDEN * 2 for l in range(LAYERS + 1)]
        d.dW[:], d.db[:] = [g.data_ptr() for g in dW], [g.data_ptr() for g in db]
        d.B, d.S, d.out_w, d.err = Bn, S, self.out_w, self.err.data_ptr()
        st = L.ctl_mlp_backward(C.byref(d), _stream())
        if st != OK:
            raise CtlError(st, "ctl_mlp_backward")
        return loss, dW, db

    def adam(self, dW, db, lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, wd=0.0):
        L = _bind()
        self.step_count += 1
        self.version += 1
        d = AdamDesc()
        for k, ts in (("w", self.W), ("b", self.b), ("g", dW), ("gb", db), ("m", self.m), ("v", self.v),
                      ("mb", self.mb), ("vb", self.vb), ("wb", self.Wb), ("wbT", self.WbT)):
            getattr(d, k)[:] = [t.data_ptr() for t in ts]
        d.out_w, d.step = self.out_w, self.step_count
        d.lr, d.beta1, d.beta2, d.eps, d.weight_decay = lr, beta1, beta2, eps, wd
        st = L.ctl_mlp_adam_step(C.byref(d), _stream())
        if st != OK:
            raise CtlError(st, "ctl_mlp_adam_step")

    def packed(self):
        """Weights in the screening kernel's streaming layout and the
        concatenated biases; rebuilt after every Adam step."""
        torch = self.torch
        if getattr(self, "_packed_at", None) != self.version:
            L = _bind()
            wp = torch.empty(L.ctl_mlp_pack_bytes(self.out_w) // 2, dtype=torch.bfloat16, device="cuda")
            ptrs = (C.c_void_p * 5)(*[w.data_ptr() for w in self.Wb])
            lds = (C.c_int32 * 5)(*[w.stride(0) for w in self.Wb])
            st = L.ctl_mlp_pack(ptrs, lds, self.out_w, _ptr(wp), _stream())
            if st != OK:
                raise CtlError(st, "ctl_mlp_pack")
            self._wpack = wp
            self._bias = torch.cat(self.b).contiguous()
            self._packed_at = self.version
        return self._wpack, self._bias

    # -- optimiser state ---------------------------------------------------------
    _STATE = ("W", "b", "Wb", "WbT", "m", "v", "mb", "vb")

    def state(self):
        """A copy of the weights and the optimiser state."""
        st = {k: [t.clone() for t in getattr(self, k)] for k in self._STATE}
        st["step_count"] = self.step_count
        return st

    def load_state(self, st):
        for k in self._STATE:
            for dst, src in zip(getattr(self, k), st[k]):
                dst.copy_(src)
        self.step_count = st["step_count"]
        self.version += 1

    def reset_optimizer(self):
        """Fresh Adam moments (and bias correction) for a new training phase."""
        for k in ("m", "v", "mb", "vb"):
            for t in getattr(self, k):
                t.zero_()
        self.step_count = 0

    def check_error_flag(self):
        if int(self.err.item()) != 0:
            raise RuntimeError("tcgen05 GEMM reported a bounded-wait timeout")

    def state_numpy(self):
        return ([w.cpu().numpy() for w in self.W], [b.cpu().numpy() for b in self.b])


def screen(net: MLP, theta_log, tvec, target, sc: Scaling):
    """Fitness of each candidate from the surrogate's ensemble mean, in one
    fused kernel (ctl_mlp_screen): theta_log [n][n_par] FP32 device tensor,
    tvec [ns], target [ns][S]; returns a FP64 device tensor [n]."""
    torch = net.torch
    L = _bind()
    theta = theta_log.to(torch.float32).contiguous()
    n, n_par = theta.shape
    # the small host arrays in one copy
    parts = [np.asarray(a, dtype=np.float32).reshape(-1)
             for a in (tvec, target, sc.log_lo, sc.log_hi, sc.y_mean, sc.y_std)]
    buf = torch.from_numpy(np.concatenate(parts)).cuda()
    tv, tg, lo, hi, ym, ys = (C.c_void_p(buf.data_ptr() + 4 * o)
                              for o in np.cumsum([0] + [p.size for p in parts[:-1]]).tolist())
    wp, bias = net.packed()
    fit = torch.empty(n, dtype=torch.float64, device="cuda")
    d = ScreenDesc(_ptr(theta), n_par, n, tv, parts[0].size, float(sc.t_end), lo, hi, ym, ys, net.S, net.out_w, tg,
                   _ptr(wp), _ptr(bias), _ptr(fit), _ptr(net.err))
    st = L.ctl_mlp_screen(C.byref(d), _stream())
    if st != OK:
        raise CtlError(st, "ctl_mlp_screen")
    return fit
