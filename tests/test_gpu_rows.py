"""Many right-hand sides per kept factor in one launch (wds_sensitivity): more
rows than the plan holds scenarios, with ACTIVE valves (scratch by resident
group), on the shared-memory and on the large-network layout; and batches on
both sides of the scenario groups per CTA."""
import numpy as np
import pytest
import torch

from wdsgpu_b200 import GGASolver, implicit_solve, synth
from wdsgpu_b200.sensitivity import sensitivity_matrix

pytestmark = pytest.mark.gpu


def _net(which):
    return {"valves": synth.config2_network,
            "small": lambda: synth.looped_network(3, 100, 1, 120, n_emitters=5),
            "large": lambda: synth.looped_network(5, 3000, 2, 3600)}[which]()


@pytest.mark.parametrize("which,T,m", [("valves", 1, 40), ("valves", 3, 7), ("valves", 20, 30),
                                       ("small", 1, 33), ("small", 9, 1), ("large", 2, 5)])
def test_rows_equal_head_gradients(which, T, m):
    # row (t, i) is d head_i / d r of frame t: the gradient of one head, from
    # the same refined solve on the same factor (1e-9 relative)
    net = _net(which)
    d, _ = synth.config2_scenarios(net, T, seed=4)
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    sens = synth.sensor_nodes(net, m, seed=1)
    s = GGASolver(net, device="cuda:0", dense_status_machine=True)
    S = sensitivity_matrix(s, d, rh, None, sens, wrt="r", accuracy=1e-8)
    assert S.shape == (T * m, net.L)
    D, RH = torch.tensor(d, device="cuda:0"), torch.tensor(rh, device="cuda:0")
    for t, i in {(0, 0), (T - 1, m - 1), (T // 2, m // 2)}:
        r = s.r_hw.expand(T, -1).clone().requires_grad_(True)
        h = implicit_solve(s, D, RH, r_hw=r, accuracy=1e-8)[0]
        h[t, int(sens[i])].backward()
        g = r.grad[t].cpu().numpy()
        assert np.abs(S[t * m + i] - g).max() <= 1e-9 * np.abs(g).max()


@pytest.mark.parametrize("B", [1, 2, 147, 148, 149, 296, 297, 445, 593])
def test_batch_sizes_around_the_groups_per_cta(B):
    # a launch takes as few scenario groups per CTA as hold the batch; a
    # scenario's results do not depend on it
    net = _net("small")
    d, _ = synth.config2_scenarios(net, 593, seed=9)
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    s = GGASolver(net, device="cuda:0", dense_status_machine=True)

    def step(lo, hi):
        D = torch.tensor(d[lo:hi], device="cuda:0", requires_grad=True)
        h = implicit_solve(s, D, torch.tensor(rh[lo:hi], device="cuda:0"), accuracy=1e-6)[0]
        (h ** 2).sum().backward()
        return h.detach(), D.grad

    h, g = step(0, B)
    for b in {0, B // 2, B - 1}:
        h1, g1 = step(b, b + 1)
        assert torch.equal(h1[0], h[b]) and torch.equal(g1[0], g[b])
