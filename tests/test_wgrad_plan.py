"""The length of the weight-gradient kernel's accumulation chains, whose MMAs
round towards zero: over every batch up to 65,536 rows and several SM counts no
chain is longer than 512 rows or 1/64 of the batch (CPU), and one step at a
batch whose tiles do not divide evenly (GPU)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import cutauleaping_b200 as ctl

CSRC = os.path.join(os.path.dirname(ctl.__file__), "csrc")

MAIN = r'''
#include <cstdint>
#include <cstdio>
#include "ctl_train_plan.h"
using namespace ctl::mlp;
int main() {
    for (int sms : {64, 132, 148, 160})
        for (int tiles = 1; tiles <= 512; tiles++)
            for (int l = 0; l < TR_L; l++) {
                const int parts = wg_ctas(l, tiles, sms);
                int longest = 0;
                for (int part = 0; part < parts; part++) {  // the kernel's split
                    const int t = (int)((int64_t)tiles * (part + 1) / parts) - (int)((int64_t)tiles * part / parts);
                    const int chains = wg_chains(l) < t ? wg_chains(l) : t;
                    int len[4] = {0, 0, 0, 0};
                    for (int i = 0; i < t; i++) len[i * chains / t]++;
                    for (int n : len) longest = n > longest ? n : longest;
                }
                printf("%d %d %d %d %d\n", sms, tiles, l, parts, longest);
            }
}
'''


def test_no_chain_is_longer_than_the_bound(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ is not installed")
    (tmp_path / "plan.cpp").write_text(MAIN)
    exe = str(tmp_path / "plan")
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CSRC}", "-o", exe, str(tmp_path / "plan.cpp")], check=True)
    rows = np.array([[int(v) for v in line.split()] for line in
                     subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()])
    sms, tiles, layer, parts, longest = rows.T
    assert (parts >= 1).all() and (parts <= tiles).all()
    assert (longest * 128 <= np.maximum(512, tiles * 128 // 64)).all()


@pytest.mark.gpu
def test_step_with_uneven_shares_matches_the_oracle():
    """153 tiles over 39 CTAs a layer; tolerances as the single-step test's."""
    import torch
    from cutauleaping_b200 import surrogate as sg
    from oracle import mlp_oracle as mo
    S, B = 3, 19584
    net = sg.MLP(S, seed=4)
    rng = np.random.default_rng(1)
    X = np.zeros((B, sg.IN_PAD), np.float32)
    X[:, :9] = rng.uniform(-1, 1, (B, 9))
    tgt = rng.normal(0, 1, (B, S)).astype(np.float32)
    y = net.forward(torch.from_numpy(X).cuda().to(torch.bfloat16))
    loss, dW, db = net.backward(y, torch.from_numpy(tgt).cuda())
    torch.cuda.synchronize()
    net.check_error_flag()
    l_o, dW_o, db_o, _ = mo.backward(X, [w.cpu().numpy() for w in net.W], [b.cpu().numpy() for b in net.b], tgt)
    assert abs(loss.item() - l_o) <= 1e-3 * abs(l_o)
    for l in range(len(net.W)):
        for g, o in ((dW[l], dW_o[l]), (db[l], db_o[l])):
            assert np.linalg.norm(g.cpu().numpy() - o) <= 2e-2 * np.linalg.norm(o) + 1e-7, l
