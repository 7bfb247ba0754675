"""The shared-memory sweep where a propensity overflows FP32: a catalytic
reaction that changes no species has an infinite one, the others leap and fire
critically.  Against the CPU oracle bit for bit, but for the infinite reaction's
own firings: a Poisson draw of infinite mean is 2^31 - 1 or no number, which a
CPU converts to 0 and the GPU to 2^31, so firings are compared modulo 2^31."""
import numpy as np
import pytest

import cutauleaping_b200 as ctl
from cutauleaping_b200 import inputs
from tests.netutil import oracle_run, same_info

pytestmark = pytest.mark.gpu


def _net(place, R=8):
    """Reaction `place` is 2 A -> 2 A at an infinite rate; another one consumes
    a species of few molecules (critical), the rest many."""
    S, n = R + 2, 40
    left, right = np.zeros((R, S), np.int32), np.zeros((R, S), np.int32)
    X0, c = np.zeros((n, S), np.int32), np.zeros((n, R))
    for r in range(R):
        left[r, 1 + r] = right[r, 1 + (r + 1) % R] = 1
        X0[:, 1 + r] = 3000 + 100 * r
        c[:, r] = 0.5 + 0.1 * r
    left[place], right[place] = 0, 0
    left[place, 0] = right[place, 0] = 2
    X0[:, 0] = 1000 + np.arange(n)
    c[:, place] = 1e37
    rare = (place + 3) % R
    left[rare], right[rare] = 0, 0
    left[rare, S - 1], right[rare, 1] = 1, 1
    X0[:, S - 1] = 1 + np.arange(n) % 9
    c[:, rare] = 20.0
    return inputs.Network(left, right, np.zeros(S, np.int32), X0, c, np.linspace(0.02, 0.3, 9))


@pytest.mark.parametrize("G", [1, 4, 8, 32, 64])
@pytest.mark.parametrize("place", [0, 2])
def test_infinite_propensity_matches_the_oracle(place, G):
    net = _net(place, R=8 if G < 64 else 70)
    m = ctl.Model.create(net.left, net.right, net.feed, net.tvec, net.cs)
    for flags in (0, ctl.Q2_OFF):
        kw = dict(seed=5, flags=flags, max_steps=2000)
        out_o, want = oracle_run(net, **kw)
        want["firings"] %= 1 << 31
        assert (out_o[:, -1, -1] < out_o[:, 0, -1]).any() or flags == 0  # the critical reaction fires
        for spec in (-1, 1) if G == 8 else (-1,):
            out, info = m.run(net.X0, net.c, group=G, spec=spec, check=False, **kw)
            assert np.array_equal(out, out_o), (flags, spec)
            info["firings"] %= 1 << 31
            assert same_info(info, want) is None, (flags, spec, same_info(info, want))
