"""The lanes per simulation that the library takes for networks of 1,024 leaves
and more, on both sides of each line of the rule, and the sweep at the lines:
the same bits as with a group size given by the caller, and as the oracle."""
import numpy as np
import pytest

import cutauleaping_b200 as ctl
from cutauleaping_b200 import inputs
from tests.netutil import oracle_run, same_info

pytestmark = pytest.mark.gpu


def _net(S, R, n):
    return inputs.synthetic(S, R, n, seed=0, t_end=4e-4, samples=4, c_range=(1e-5, 1e-1), x0_range=(1, 100000))


def _model(net):
    return ctl.Model.create(net.left, net.right, net.feed, net.tvec, net.cs)


@pytest.mark.parametrize("S,R,G", [(512, 1024, 64), (1024, 2048, 128)])
def test_lanes_follow_the_batch(S, R, G):
    m = _model(_net(S, R, 2))
    sms = m.launch_info(1, uniform_rates=1).sm_count
    two, wave = 512 * sms // (2 * G), 768 * sms // G
    for n, lanes in ((1, 2 * G), (two, 2 * G), (two + 1, G), (wave, G), (wave + 1, 2 * G), (wave + wave // 4, 2 * G),
                     (wave + wave // 4 + 1, G), (2 * wave, G), (4 * wave, G)):
        assert m.launch_info(n, uniform_rates=1).group == lanes, n
        assert m.launch_info(n, uniform_rates=1, flags=ctl.FORCE_SSA).group == G, n
        assert m.launch_info(n, uniform_rates=1, group=32).group == 32


def test_sweep_at_the_lines():
    sms = _model(_net(512, 1024, 2)).launch_info(1).sm_count
    for n in (1, 4 * sms, 4 * sms + 1, 12 * sms + 1):
        net = _net(512, 1024, n)
        m = _model(net)
        out, info = m.run(net.X0, net.c, seed=3)
        ref, ref_info = m.run(net.X0, net.c, seed=3, group=32)
        assert np.array_equal(out, ref) and same_info(info, ref_info) is None, n
        net.X0, net.c = net.X0[:4], net.c[:4]
        out_o, info_o = oracle_run(net, seed=3)
        assert np.array_equal(out[:4], out_o) and same_info(info[:4], info_o) is None, n
