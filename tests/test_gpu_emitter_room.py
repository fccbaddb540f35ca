"""Networks with an emitter at many junctions: what a scenario holds per
emitter slot must not cost the layout or the scenario groups per CTA.  The
sizes are those whose state and tables just fit."""
import numpy as np
import pytest
import torch

from oracle.gga import Model
from wdsgpu_b200 import GGASolver, implicit_solve, synth
from wdsgpu_b200.autodiff import solve_unrolled
from wdsgpu_b200.multi import implicit_solve_multi

pytestmark = pytest.mark.gpu


def _case(nj, links, emitters, B=2):
    net = synth.looped_network(3, nj, 2, links, n_emitters=emitters)
    d, _ = synth.config2_scenarios(net, B, seed=11)
    return net, d, np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()


# (500, 800), (525, 1050) and (425, 850): more links than 1.5 a junction, so
# the link pass's vector is the longest of the state; the others: 50 % emitters
@pytest.mark.parametrize("nj,links,emitters,groups",
                         [(540, 648, 270, 4), (660, 792, 330, 3), (900, 1080, 450, 2),
                          (500, 800, 0, 4), (425, 850, 0, 3), (525, 1050, 0, 2)])
def test_groups_per_cta_of_networks_that_just_fit(cuda, nj, links, emitters, groups):
    net, d, rh = _case(nj, links, emitters)
    ref = Model(net).implicit(d, rh, accuracy=1e-7, polish_steps=3)[0]["head_ft"]
    for g in (groups, 1):
        s = GGASolver(net, device=cuda, dense_status_machine=True)
        s.sm100_tuning = dict(groups_per_cta=g)
        assert s.plan(2).stats()["groups_per_cta"] == g
        h = implicit_solve(s, torch.tensor(d, device=cuda), torch.tensor(rh, device=cuda),
                           accuracy=1e-7)[0]
        # polished heads are the Newton fixed point
        assert np.abs(h.cpu().numpy() - ref).max() < 1e-9 / 0.3048


@pytest.mark.parametrize("nj,links,emitters", [(1600, 1680, 800), (1380, 1656, 690),
                                               (900, 1440, 450)])
def test_small_layout_of_networks_that_just_fit(cuda, nj, links, emitters):
    net, d, rh = _case(nj, links, emitters)
    s = GGASolver(net, device=cuda, dense_status_machine=True)
    s.sm100_layout = "shared"
    h = implicit_solve(s, torch.tensor(d, device=cuda), torch.tensor(rh, device=cuda),
                       accuracy=1e-7)[0]
    assert s.plan(2).stats()["smem_bytes"] > 0
    ref = Model(net).implicit(d, rh, accuracy=1e-7, polish_steps=3)[0]["head_ft"]
    assert np.abs(h.cpu().numpy() - ref).max() < 1e-9 / 0.3048


def test_callers_order_keeps_its_groups(cuda):
    # the order of the fewest entries, given by the caller: four groups fit
    net, d, rh = _case(660, 792, 0)
    t = GGASolver(net, device=cuda, dense_status_machine=True)
    t.sm100_tuning = dict(groups_per_cta=4)
    s = GGASolver(net, device=cuda, dense_status_machine=True, perm=t.symbolic()["perm"])
    assert s.plan(2).stats()["groups_per_cta"] == 4
    h = implicit_solve(s, torch.tensor(d, device=cuda), torch.tensor(rh, device=cuda),
                       accuracy=1e-7)[0]
    ref = Model(net).implicit(d, rh, accuracy=1e-7, polish_steps=3)[0]["head_ft"]
    assert np.abs(h.cpu().numpy() - ref).max() < 1e-9 / 0.3048


@pytest.mark.parametrize("nj,links,emitters,groups", [(540, 648, 270, 4), (425, 850, 0, 3),
                                                      (525, 1050, 30, 2), (60, 70, 60, 4)])
def test_results_do_not_depend_on_where_the_state_lies(cuda, nj, links, emitters, groups):
    # one elimination order; many groups per CTA share the vectors' room and
    # keep the emitters' constants in global memory, one group does not: the
    # same values, bit for bit, from the solve, both adjoints and the unrolled
    # iterations
    net, d, rh = _case(nj, links, emitters, B=3)
    t = GGASolver(net, device=cuda, dense_status_machine=True)
    t.sm100_tuning = dict(groups_per_cta=groups)
    perm = t.symbolic()["perm"]
    res = []
    for g in (groups, 1):
        s = GGASolver(net, device=cuda, dense_status_machine=True, perm=perm)
        s.sm100_tuning = dict(groups_per_cta=g)
        out = []
        for f in (lambda D, K: implicit_solve(s, D, torch.tensor(rh, device=cuda), ke=K,
                                              accuracy=1e-7),
                  lambda D, K: tuple(solve_unrolled(s, D, torch.tensor(rh, device=cuda), ke=K,
                                                    K=6).values())):
            D = torch.tensor(d, device=cuda, requires_grad=True)
            K = s.node_ke_default.clone().requires_grad_(True)
            o = f(D, K)
            (o[0] ** 2).sum().backward()
            out += [x.detach() for x in o[:3]] + [D.grad, K.grad]
        res.append(out)
    assert all(torch.equal(x, y) for x, y in zip(*res))


def test_networks_that_just_fit_in_one_launch(cuda):
    # the multi-network launch takes the plans' own placement: as each alone
    ss, D, RH, alone = [], [], [], []
    for case in ((540, 648, 270), (425, 850, 0)):
        net, d, rh = _case(*case, B=3)
        s = GGASolver(net, device=cuda, dense_status_machine=True)
        ss.append(s)
        D.append(torch.tensor(d, device=cuda, requires_grad=True))
        RH.append(torch.tensor(rh, device=cuda))
        h = implicit_solve(s, D[-1], RH[-1], accuracy=1e-7)[0]
        alone.append((h.detach(), torch.autograd.grad((h ** 2).sum(), D[-1])[0]))
    out = implicit_solve_multi(ss, D, RH, accuracy=1e-7)
    grads = torch.autograd.grad(sum((o[0] ** 2).sum() for o in out), D)
    for (h, g), o, gm in zip(alone, out, grads):
        assert torch.equal(h, o[0]) and torch.equal(g, gm)
