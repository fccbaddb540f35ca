"""Inputs at the ends of the double range: an infinite or overflowing pipe
gradient leaves its scenario unconverged, without a pivot failing and without
a trace in the other scenarios of the batch."""
import numpy as np
import pytest
import torch

from wdsgpu_b200 import GGASolver, implicit_solve, synth

pytestmark = pytest.mark.gpu


def _case(cuda, links=120, layout="auto"):
    net = synth.looped_network(3, 100, 1, links, n_emitters=5)
    d, _ = synth.config2_scenarios(net, 2, seed=4)
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    s = GGASolver(net, device=cuda, dense_status_machine=True)
    s.sm100_layout = layout
    # a pipe of a loop: both its junctions have three links or more
    deg = np.bincount(np.r_[net.link_n1, net.link_n2], minlength=net.N)
    k = int(np.flatnonzero((deg[net.link_n1] >= 3) & (deg[net.link_n2] >= 3))[0])
    return s, torch.tensor(d, device=cuda), torch.tensor(rh, device=cuda), k


@pytest.mark.parametrize("layout", ["auto", "global"])
@pytest.mark.parametrize("what,value", [("r", np.inf), ("r", 1e308), ("q0", np.inf),
                                        ("q0", -np.inf), ("q0", np.nan), ("q0", 1e308)])
def test_overflowing_pipe_gradient_leaves_its_scenario_unconverged(cuda, layout, what, value):
    s, d, rh, k = _case(cuda, layout=layout)
    r = s.r_hw.repeat(2, 1)
    q0 = torch.ones(2, s.L, dtype=torch.float64, device=cuda)
    e0 = torch.zeros(2, s.N, dtype=torch.float64, device=cuda)
    (r if what == "r" else q0)[0, k] = value
    o = s.solve(d, rh, r_hw=r, q0=q0, e0=e0, status_machine=True, accuracy=1e-7)
    assert o["converged"].tolist() == [False, True]
    one = s.solve(d[1:], rh[1:], r_hw=r[1:], q0=q0[1:], e0=e0[1:], status_machine=True,
                  accuracy=1e-7)
    for f in ("head_ft", "flow_cfs", "emitter_cfs", "iters"):
        assert torch.equal(o[f][1], one[f][0]), f


def test_infinite_resistance_is_reported_as_unconverged(cuda):
    s, d, rh, k = _case(cuda)
    r = s.r_hw.repeat(2, 1)
    r[0, k] = np.inf
    with pytest.raises(RuntimeError, match="did not converge"):
        implicit_solve(s, d, rh, r_hw=r, accuracy=1e-7)
