"""The register-resident sweep at the edges of its shapes, against the CPU
oracle bit for bit: one reaction to sixteen, helper lanes without a simulation,
warps whose simulations leap and step at the same time, Poisson means from
below 1 to beyond the straight-line quotients, propensity sums too small or too
large for them -- in both schedules, the library's kernels and the compiled ones."""
import numpy as np
import pytest

import cutauleaping_b200 as ctl
from cutauleaping_b200 import inputs
from tests.netutil import oracle_run, same_info

pytestmark = pytest.mark.gpu


def _net(left, right, X0, c, t_end=1.0, ns=7):
    left, right = np.array(left, np.int32), np.array(right, np.int32)
    return inputs.Network(left, right, np.zeros(left.shape[1], np.int32), np.array(X0, np.int32), np.array(c, float),
                          np.linspace(t_end / ns, t_end, ns))


def _mixed(n):
    """A + B <-> C, 3A -> 2A and an inflow of B; populations from a few to 10^7."""
    X0 = np.array([[3 * 10 ** (i % 8), 10 ** (1 + i % 7), i % 5] for i in range(n)])
    c = np.array([[10.0 ** -(i % 8), 0.5 + i % 3, 10.0 ** -(1 + 2 * (i % 8)), 5.0] for i in range(n)])
    return _net([[1, 1, 0], [0, 0, 1], [3, 0, 0], [0, 0, 0]], [[0, 0, 1], [1, 1, 0], [2, 0, 0], [0, 1, 0]], X0, c, 0.5)


NETS = {
    "1x1": lambda: _net([[1]], [[0]], [[10 ** (i % 9)] for i in range(70)], [[1.5]] * 70),
    "catalytic": lambda: _net([[1, 0], [0, 1]], [[1, 0], [0, 1]], [[100, 3]] * 33, [[1.0, 2.0]] * 33),
    "faint": lambda: _net([[1, 0], [0, 1]], [[0, 1], [1, 0]], [[50, 7]] * 40, [[1e-30 * (i + 1), 1e-33] for i in range(40)]),
    "fierce": lambda: _net([[1, 0], [0, 1]], [[0, 1], [1, 0]], [[50, 7]] * 40, [[1e19 * (i + 1), 3e19] for i in range(40)]),
    "mixed": lambda: _mixed(75),
    "8x16": lambda: inputs.synthetic(8, 16, 45, seed=4, t_end=0.4, samples=9, x0_range=(5, 40000), perturb_sigma=0.7,
                                     perturb_seed=2),
}


@pytest.mark.parametrize("name", NETS)
def test_register_resident_edges_match_the_oracle(name):
    net = NETS[name]()
    m = ctl.Model.create(net.left, net.right, net.feed, net.tvec, net.cs)
    assert m.launch_info(net.n).warp_sims > 0
    for flags in (0, ctl.FORCE_SSA):
        kw = dict(seed=29, flags=flags, max_steps=3000)
        out_o, info_o = oracle_run(net, **kw)
        for sched, ws, spec in ((0, 0, 0), (1, 3, 0), (2, 32, 0), (1, 16, -1), (2, 5, -1)):
            out, info = m.run(net.X0, net.c, sched=sched, warp_sims=ws, spec=spec, check=False, **kw)
            what = f"{name} flags={flags} sched={sched} warp_sims={ws} spec={spec}"
            assert np.array_equal(out, out_o), what
            assert same_info(info, info_o) is None, what


def test_schedule_follows_the_batch():
    """One simulation per warp, block rounds, full warps in lockstep; a shape
    given by the caller keeps rounds."""
    net = inputs.schlogl(4, samples=5, t_end=0.1)
    m = ctl.Model.create(net.left, net.right, net.feed, net.tvec, net.cs)
    sms = m.launch_info(1).sm_count
    for n, sched, ws in ((1, 2, 1), (8 * sms, 2, 1), (8 * sms + 1, 1, 5), (64 * sms, 1, 16), (64 * sms + 1, 2, 32)):
        li = m.launch_info(n)
        assert (li.sched, li.warp_sims) == (sched, ws), n
    assert m.launch_info(1, warp_sims=2).sched == 1 and m.launch_info(1, threads=64).sched == 1
