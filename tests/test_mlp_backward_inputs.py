"""What MLP.backward takes as y and target: the kernel reads y in rows of out_w
floats, so any other layout has to reach it as such rows.  On the CPU with a
stand-in for the C entry point that records the memory it is given; on the GPU
against the call with forward's own y."""
import ctypes as C

import numpy as np
import pytest
import torch

from cutauleaping_b200 import surrogate as sg

B = 128


class _CpuTorch:
    """torch with "cuda" tensors placed in host memory."""

    def __getattr__(self, name):
        return getattr(torch, name)

    def zeros(self, *a, device=None, **k):
        return torch.zeros(*a, **k)

    def empty(self, *a, device=None, **k):
        return torch.empty(*a, **k)


class _Lib:
    def ctl_mlp_pack_bytes(self, out_w):
        return (64 + 3 * 256 + out_w) * 256 * 2

    def ctl_mlp_backward(self, d, stream):
        d = d._obj
        self.y = np.ctypeslib.as_array(C.cast(d.y, C.POINTER(C.c_float)), (d.B, d.out_w)).copy()
        self.target = np.ctypeslib.as_array(C.cast(d.target, C.POINTER(C.c_float)), (d.B, d.S)).copy()
        assert d.y % 32 == 0
        return 0


def _cpu_net(S, monkeypatch):
    monkeypatch.setattr(torch.Tensor, "cuda", lambda self: self)
    monkeypatch.setattr(torch, "zeros", lambda *a, _z=torch.zeros, device=None, **k: _z(*a, **k))
    net = sg.MLP(S)
    monkeypatch.undo()
    net.torch = _CpuTorch()
    lib = _Lib()
    monkeypatch.setattr(sg, "_bind", lambda: lib)
    monkeypatch.setattr(sg, "_stream", lambda: None)
    net.z = net._buf("z", (sg.LAYERS, B, sg.HIDDEN), torch.float32)
    net.hp = net._buf("hp", (B * (sg.IN_PAD + sg.LAYERS * sg.HIDDEN),), torch.bfloat16)
    return net, lib


def _views(full, S):
    """The same values in every layout that a caller may have them in."""
    wide = torch.zeros(full.shape[0], 3 * full.shape[1], dtype=full.dtype, device=full.device)
    wide[:, 5:5 + 2 * S] = full[:, :2 * S]
    odd = torch.zeros(full.numel() + 1, dtype=full.dtype, device=full.device)[1:].view(full.shape)
    odd.copy_(full)
    return {"forward's": full, "2S columns": full[:, :2 * S], "2S contiguous": full[:, :2 * S].contiguous(),
            "part of wider rows": wide[:, 5:5 + 2 * S], "off a 32-byte boundary": odd,
            "column-major": full.t().contiguous().t()}


@pytest.mark.parametrize("S", [3, 32, 33, 64])
def test_rows_reach_the_kernel(S, monkeypatch):
    net, lib = _cpu_net(S, monkeypatch)
    g = torch.Generator().manual_seed(S)
    full, tgt = torch.randn(B, net.out_w, generator=g), torch.randn(B, S, generator=g)
    for what, y in _views(full, S).items():
        net.backward(y, tgt)
        assert np.array_equal(lib.y[:, :2 * S], full[:, :2 * S].numpy()), what
        assert np.array_equal(lib.target, tgt.numpy())
    net.backward(full, torch.cat([tgt, tgt], 1)[:, :S])
    assert np.array_equal(lib.target, tgt.numpy())


def test_refused_inputs(monkeypatch):
    S = 3
    net, lib = _cpu_net(S, monkeypatch)
    y, tgt = torch.zeros(B, net.out_w), torch.zeros(B, S)
    for bad_y, bad_t in ((y[:, :2 * S - 1], tgt), (y[:-1], tgt), (y.double(), tgt), (y, tgt.double()), (y.half(), tgt),
                         (y, torch.zeros(2 * B, S))):
        with pytest.raises(ValueError):
            net.backward(bad_y, bad_t)


@pytest.mark.gpu
@pytest.mark.parametrize("S", [3, 33])
def test_every_layout_gives_the_same_gradients(S):
    """One 128-row tile: a single CTA per layer, so the gradients' sums have one
    order and are equal bit for bit; the loss adds eight warps' sums in any order."""
    net = sg.MLP(S, seed=1)
    g = torch.Generator().manual_seed(S)
    X = torch.zeros(B, sg.IN_PAD)
    X[:, :9] = 2 * torch.rand(B, 9, generator=g) - 1
    tgt = torch.randn(B, S, generator=g).cuda()
    full = net.forward(X.cuda().to(torch.bfloat16)).clone()
    ref = net.backward(full, tgt)
    mu, lv = full[:, :S].double(), full[:, S:2 * S].double()
    terms = 0.5 * (lv.abs() + (tgt - mu) ** 2 * (-lv).exp())
    for what, y in _views(full, S).items():
        loss, dW, db = net.backward(y, tgt)
        assert abs(loss.item() - ref[0].item()) <= 2.0 ** -20 * terms.sum().item(), what
        for a, b in zip(dW + db, ref[1] + ref[2]):
            assert torch.equal(a, b), what
    net.check_error_flag()
