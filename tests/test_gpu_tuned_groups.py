"""A caller's groups per CTA at sizes that only the order of the fewest entries
fits."""
import numpy as np
import pytest
import torch

from wdsgpu_b200 import GGASolver, implicit_solve, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nj,links,groups", [(975, 1023, 3), (1100, 1320, 2), (475, 760, 4)])
def test_tuned_groups_at_the_border(nj, links, groups):
    # the same fixed point as the planner's own choice (1e-9 m)
    net = synth.looped_network(3, nj, 2, links)
    d, _ = synth.config2_scenarios(net, 5, seed=11)
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    heads = []
    for g in (0, groups):
        s = GGASolver(net, device="cuda:0", dense_status_machine=True)
        if g:
            s.sm100_tuning = dict(groups_per_cta=g)
        h = implicit_solve(s, torch.tensor(d, device="cuda:0"), torch.tensor(rh, device="cuda:0"),
                           accuracy=1e-7)[0]
        if g:
            assert s.plan(5).stats()["groups_per_cta"] == g
        heads.append(h.cpu().numpy())
    assert np.abs(heads[0] - heads[1]).max() < 1e-9 / 0.3048
