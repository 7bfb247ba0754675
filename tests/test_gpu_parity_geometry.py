"""The shared-memory sweep on networks at the edges of its geometry, against
the CPU oracle bit for bit: one to three reactions (a sum tree smaller than one
four-leaf chunk), fewer leaves than the lanes' chunks, more species than
leaves, a species on which every reaction depends, and lanes that own more
chunks than their registers hold -- in the library's kernels and the ones
compiled for the network."""
import numpy as np
import pytest

import cutauleaping_b200 as ctl
from cutauleaping_b200 import inputs
from tests.netutil import oracle_run, same_info

pytestmark = pytest.mark.gpu


def _hub(R):
    """R reactions that all consume species 0 and a species of their own."""
    S = R + 1
    left, right = np.zeros((R, S), np.int32), np.zeros((R, S), np.int32)
    left[:, 0] = 1
    for r in range(R):
        left[r, 1 + r] = 1 + r % 2
        right[r, 1 + (r + 1) % R] = 1
        right[r, 0] = r % 2
    X0 = np.tile(np.concatenate([[4000], np.full(R, 60)]).astype(np.int32), (24, 1))
    c = np.tile(10.0 ** -(3 + np.arange(R) % 3), (24, 1))
    return inputs.Network(left, right, np.zeros(S, np.int32), X0, c, np.linspace(0.05, 1.0, 12))


def _net(S, R, seed):
    # nine species or more: not the register-resident sweep's
    return inputs.synthetic(S, R, 24, seed=seed, t_end=0.5, samples=9, x0_range=(5, 3000), perturb_sigma=0.4,
                            perturb_seed=seed)


CASES = [("9x1", lambda: _net(9, 1, 1)), ("9x2", lambda: _net(9, 2, 2)), ("12x3", lambda: _net(12, 3, 3)),
         ("70x5", lambda: _net(70, 5, 4)), ("20x17", lambda: _net(20, 17, 5)), ("hub40", lambda: _hub(40)),
         ("24x130", lambda: _net(24, 130, 6))]


@pytest.mark.parametrize("name,make", CASES, ids=[n for n, _ in CASES])
def test_edge_geometries_match_the_oracle(name, make):
    net = make()
    m = ctl.Model.create(net.left, net.right, net.feed, net.tvec, net.cs)
    for flags in (0, ctl.FORCE_SSA):
        out_o, info_o = oracle_run(net, seed=19, flags=flags)
        shapes = [(1, 1, -1), (2, 1, -1), (8, 2, -1), (32, 1, -1), (64, 1, -1)]
        if name in ("9x2", "hub40", "24x130"):  # seconds of compilation each
            shapes += [(1, 2, 1), (4, 1, 1)]
        for G, sched, spec in shapes:
            out, info = m.run(net.X0, net.c, seed=19, flags=flags, group=G, sched=sched, spec=spec)
            what = f"{name} flags={flags} G={G} sched={sched} spec={spec}"
            assert np.array_equal(out, out_o), what
            assert same_info(info, info_o) is None, what
