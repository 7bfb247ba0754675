"""calculateFitness's kernels (ctl_fitness_device, ctl_fitness_sums_device)
against a numpy restatement, bit for bit, over the shapes their dispatch
separates: a CTA or a cluster per parameter set, a thread per set, aligned and
ragged rows, several target repetitions, more than one set per block row, and
sums beyond 2^53, where the FP64 running sum itself rounds."""
import ctypes as C

import numpy as np
import pytest

import cutauleaping_b200 as ctl

pytestmark = pytest.mark.gpu


def _reference(samples, target, swarm, threads, p_rep):
    """samples [n][ns][so] uint32, target [ns][E][REP][so] -> fitness [sets]."""
    n, ns, so = samples.shape
    sets = n // p_rep
    REP = target.shape[2]
    fit = np.empty(sets)
    for k in range(sets):
        rows = (k // threads * p_rep + np.arange(p_rep)) * threads + k % threads
        mean = np.add.accumulate(samples[rows].astype(np.float64), axis=0)[-1] / float(p_rep)
        tg = target[:, swarm[k]].astype(np.int32).astype(np.float64)  # [ns][REP][so]
        d = np.abs(tg - mean[:, None, :])
        d = np.where(tg != 0, d / np.where(tg != 0, tg, 1.0), d)
        sub = np.float32(0.0)
        for v in d.transpose(0, 2, 1).ravel():  # instants, species, repetitions
            sub = np.float32(np.float64(sub) + v)
        fit[k] = ((1.0 / ns) * (1.0 / so)) * np.float64(sub)
    return fit


@pytest.mark.parametrize("sets,p_rep,threads,ns,so,E,REP,big", [
    (1, 1, 1, 1, 1, 1, 1, False),
    (2, 700, 1, 13, 32, 1, 1, False),    # few large sets, aligned rows
    (80, 3300, 1, 16, 5, 1, 1, False),   # two CTAs per set
    (76, 1030, 1, 15, 17, 2, 1, False),  # two CTAs per set, ragged rows
    (12, 5, 4, 7, 9, 2, 3, False),       # block rows of four sets, three repetitions
    (3, 2, 1, 3, 5, 1, 128, False),      # as many repetitions as a step holds
    (3, 2, 1, 3, 5, 1, 129, False),      # more: a thread per set
    (9000, 1, 1, 5, 2, 1, 1, False),     # many small sets: a thread per set
    (1, (1 << 21) + 5, 1, 1, 1, 1, 1, True),
])
def test_fitness_kernels_match_restatement(sets, p_rep, threads, ns, so, E, REP, big):
    import torch
    L = ctl.lib()
    rng = np.random.default_rng(sets + p_rep)
    n = sets * p_rep
    if big:  # samples whose sum passes 2^53
        samples = (0xFFFFFFFF - rng.integers(0, 3, size=(n, ns, so))).astype(np.uint32)
    else:
        samples = rng.integers(0, 2000, size=(n, ns, so)).astype(np.uint32)
    target = rng.integers(0, 1500, size=(ns, E, REP, so)).astype(np.uint32)
    target[rng.random(target.shape) < 0.1] = 0
    target[0, 0, 0, 0] = 0xFFFFFFF0  # read as a negative int, as the reference does
    swarm = (np.arange(sets) % E).astype(np.uint8)
    ref = _reference(samples, target, swarm, threads, p_rep)
    dev = lambda a: torch.as_tensor(a, device="cuda")
    P = C.c_void_p
    ds, dt, dw = dev(samples.view(np.int32).reshape(-1)), dev(target.view(np.int32).reshape(-1)), dev(swarm)
    out = torch.full((sets,), float("nan"), dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    args = (ns, so, P(dt.data_ptr()), P(dw.data_ptr()), E, REP, threads, n // threads, p_rep)
    assert L.ctl_fitness_device(P(ds.data_ptr()), *args, P(out.data_ptr()), P(stream)) == ctl.OK
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), ref)
    if big:
        return  # the sums path converts the integer sum once
    rows = (np.arange(sets) // threads * p_rep)[:, None] * threads + np.arange(p_rep)[None, :] * threads \
        + (np.arange(sets) % threads)[:, None]
    sums = samples.astype(np.uint64)[rows].sum(axis=1)
    dsum = dev(sums.view(np.int64).reshape(-1))
    L.ctl_fitness_sums_device.argtypes = [P, C.c_uint32, C.c_uint32, P, P] + [C.c_uint32] * 5 + [P, P]
    out.fill_(float("nan"))
    assert L.ctl_fitness_sums_device(P(dsum.data_ptr()), *args, P(out.data_ptr()), P(stream)) == ctl.OK
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), ref)
