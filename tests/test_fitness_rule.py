"""The rule that picks a fitness kernel: many small sets go to a thread per set
whatever their samples, few or large ones to a CTA or cluster per set (CPU: the
header's host code, built by nvcc); and both sides of the line give the bits of
the numpy restatement (GPU)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import cutauleaping_b200 as ctl
from tests.test_gpu_fitness_kernels import _reference

CSRC = os.path.join(os.path.dirname(ctl.__file__), "csrc")

MAIN = r'''
#include <cstdio>
#include "ctl_fitness.cuh"
int main() {
    static uint32_t dummy;
    unsigned sets, p_rep, ns, so, rep, threads, sums;
    while (scanf("%u %u %u %u %u %u %u", &sets, &p_rep, &ns, &so, &rep, &threads, &sums) == 7) {
        ctl::fit::Args a{sums ? nullptr : &dummy, nullptr, nullptr, nullptr, nullptr, threads, sets, p_rep, ns, so, 1, rep};
        const ctl::fit::Shape s = ctl::fit::shape_for(a, 148);
        printf("%d %d\n", s.cl, s.loaders);
    }
}
'''

# sets, p_rep, ns, s_out, repetitions, threads, sums -> CTAs per set (0: a thread per set), loaders
RULE = [
    ((65536, 64, 2, 3, 1, 1, 0), (0, 0)),      # 103 us with a thread per set, 400 with a CTA
    ((262144, 32, 1, 3, 16, 32, 0), (0, 0)),   # 44, 2,633
    ((16384, 64, 2, 3, 1, 32, 0), (0, 0)),     # 17, 97
    ((8192, 1, 50, 32, 3, 1, 0), (0, 0)),      # 1,299, 1,384
    ((8192, 10, 20, 3, 1, 1, 1), (0, 0)),
    ((32768, 32, 20, 3, 1, 1, 0), (1, 128)),   # 915, 363
    ((256, 1, 20, 3, 1, 1, 0), (1, 128)),      # 29, 7
    ((64, 512, 50, 32, 1, 1, 0), (1, 512)),
    ((256, 512, 50, 32, 1, 1, 0), (2, 128)),
    ((1, 1, 1, 1, 129, 1, 0), (0, 0)),         # more repetitions than a step's buffer holds
]


def test_rule(tmp_path):
    nvcc = shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("nvcc is not installed")
    (tmp_path / "rule.cu").write_text(MAIN)
    exe = str(tmp_path / "rule")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", f"-I{CSRC}", "-o", exe,
                    str(tmp_path / "rule.cu")], check=True)
    text = "\n".join(" ".join(map(str, shape)) for shape, _ in RULE)
    p = subprocess.run([exe], input=text, capture_output=True, text=True, check=True)
    assert [tuple(map(int, line.split())) for line in p.stdout.splitlines()] == [want for _, want in RULE]


@pytest.mark.gpu
@pytest.mark.parametrize("sets,p_rep,ns,so,threads", [(4096, 64, 2, 3, 32), (4096, 64, 2, 3, 1), (4097, 33, 3, 1, 1),
                                                      (2048, 20, 7, 5, 1), (2048, 20, 7, 5, 32)])
def test_both_sides_of_the_line(sets, p_rep, ns, so, threads):
    import torch
    rng = np.random.default_rng(sets)
    samples = rng.integers(0, 2000, size=(sets * p_rep, ns, so)).astype(np.uint32)
    target = rng.integers(0, 1500, size=(ns, 1, 1, so)).astype(np.uint32)
    swarm = np.zeros(sets, np.uint8)
    dev = lambda a: torch.as_tensor(a, device="cuda")
    ds, dt, dw = dev(samples.view(np.int32).reshape(-1)), dev(target.view(np.int32).reshape(-1)), dev(swarm)
    out = torch.full((sets,), float("nan"), dtype=torch.float64, device="cuda")
    P = C.c_void_p
    assert ctl.lib().ctl_fitness_device(P(ds.data_ptr()), ns, so, P(dt.data_ptr()), P(dw.data_ptr()), 1, 1, threads,
                                        sets * p_rep // threads, p_rep, P(out.data_ptr()),
                                        P(torch.cuda.current_stream().cuda_stream)) == ctl.OK
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), _reference(samples, target, swarm, threads, p_rep))
