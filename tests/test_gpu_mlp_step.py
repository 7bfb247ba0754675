"""The fused training step (forward, loss and data gradients, weight
gradients, Adam) at the edges of its shapes: one tile of 128 rows, fewer tiles
than the weight-gradient kernel has CTAs per layer and more, output widths of
64 and 128 with and without padding.  Forward and gradients against the CPU
FP32 oracle, which rounds to BF16 at the same points (relative Frobenius error
2e-2, as the single-step test; the loss 1e-3); Adam against the same FP32
formula in PyTorch (1e-6 relative: one rounding per operation)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,B", [(3, 128), (33, 384), (64, 2560), (32, 6016)])
def test_step_matches_oracle(S, B):
    import torch
    from cutauleaping_b200 import surrogate as sg
    from oracle import mlp_oracle as mo
    net = sg.MLP(S, seed=S)
    rng = np.random.default_rng(B)
    for b in net.b:
        b.copy_(torch.from_numpy(rng.normal(0, 0.1, b.shape).astype(np.float32)))
    net.b[-1][2 * S:] = 0.0
    X = np.zeros((B, sg.IN_PAD), np.float32)
    X[:, :9] = rng.uniform(-1, 1, (B, 9))
    tgt = rng.normal(0, 1, (B, S)).astype(np.float32)
    W = [w.cpu().numpy() for w in net.W]
    b = [x.cpu().numpy() for x in net.b]
    y = net.forward(torch.from_numpy(X).cuda().to(torch.bfloat16))
    y0 = net.forward(torch.from_numpy(X).cuda().to(torch.bfloat16), keep=False).clone()
    y = net.forward(torch.from_numpy(X).cuda().to(torch.bfloat16))
    assert torch.equal(y, y0)
    loss, dW, db = net.backward(y, torch.from_numpy(tgt).cuda())
    torch.cuda.synchronize()
    net.check_error_flag()
    l_o, dW_o, db_o, y_o = mo.backward(X, W, b, tgt)
    assert np.allclose(y.cpu().numpy(), y_o, rtol=2e-2, atol=2e-3)
    assert abs(loss.item() - l_o) <= 1e-3 * abs(l_o)
    for l in range(len(W)):
        for g, o, what in ((dW[l], dW_o[l], "dW"), (db[l], db_o[l], "db")):
            g = g.cpu().numpy()
            assert g.shape == o.shape
            assert np.linalg.norm(g - o) <= 2e-2 * np.linalg.norm(o) + 1e-7, f"{what}[{l}]"
    for step in (1, 2):
        ref = []
        for p, g, m, v in [(net.W[l], dW[l], net.m[l], net.v[l]) for l in range(5)] + \
                [(net.b[l], db[l], net.mb[l], net.vb[l]) for l in range(5)]:
            m1, v1 = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            ref.append(p - 1e-3 * (m1 / (1 - 0.9 ** step)) / ((v1 / (1 - 0.999 ** step)).sqrt() + 1e-8))
        net.adam(dW, db, lr=1e-3)
        for p, r in zip(net.W + net.b, ref):
            # the update's own rounding, and 1 - 0.999^step in FP32 (relative error about 1e-4)
            assert (p - r).abs().max().item() <= 1e-6 * r.abs().max().item() + 1e-3 * 2e-4
        for w, wb, wbT in zip(net.W, net.Wb, net.WbT):
            assert torch.equal(wb, w.to(torch.bfloat16)) and torch.equal(wbT, wb.t())
