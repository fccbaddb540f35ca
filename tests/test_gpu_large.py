"""Networks beyond shared memory: the per-warp rounds of the factorisation and
the substitutions, with lists of one entry (a tree) to hundreds (no top block),
levels of one item to thousands, against the oracle."""
import numpy as np
import pytest
import torch

from oracle.gga import Model
from wdsgpu_b200 import GGASolver, implicit_solve, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nj,links,top", [(2500, 2501, 0), (2200, 2640, 0), (2200, 2640, -1),
                                          (2200, 2640, 3), (2203, 4400, 0), (2203, 4400, -1)])
def test_rounds_of_large_networks(nj, links, top):
    # polished heads are the Newton fixed point (1e-9 m), gradients follow
    # from one refined adjoint solve on the terminal factor (1e-8 relative)
    net = synth.looped_network(3, nj, 1, links, n_emitters=5)
    d, _ = synth.config2_scenarios(net, 2, seed=11)
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    s = GGASolver(net, device="cuda:0", dense_status_machine=True)
    s.sm100_tuning = dict(top_max=top)
    D = torch.tensor(d, device="cuda:0", requires_grad=True)
    h, q, e = implicit_solve(s, D, torch.tensor(rh, device="cuda:0"), accuracy=1e-7)
    assert s.plan(2).stats()["smem_bytes"] == 0    # no shared-memory layout
    (h ** 2).sum().backward()
    m = Model(net)
    out, st = m.implicit(d, rh, accuracy=1e-7, polish_steps=3)
    gd = m.backward(st, 2.0 * out["head_ft"], np.zeros_like(out["flow_cfs"]),
                    np.zeros_like(out["emitter_cfs"]))[0]
    assert np.abs(h.detach().cpu().numpy() - out["head_ft"]).max() < 1e-9 / 0.3048
    assert np.abs(D.grad.cpu().numpy() - gd).max() < 1e-8 * np.abs(gd).max()


@pytest.mark.parametrize("nj,links", [(964, 1542), (1593, 1911), (1957, 2054)])
def test_border_of_the_small_layout(nj, links):
    # networks that fill shared memory: the small layout takes them, and both
    # layouts have the same fixed point (1e-9 m)
    net = synth.looped_network(3, nj, 2, links)
    d, _ = synth.config2_scenarios(net, 2, seed=11)
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    heads = []
    for layout in ("shared", "global"):
        s = GGASolver(net, device="cuda:0", dense_status_machine=True)
        s.sm100_layout = layout
        h = implicit_solve(s, torch.tensor(d, device="cuda:0"), torch.tensor(rh, device="cuda:0"),
                           accuracy=1e-7)[0]
        assert (s.plan(2).stats()["smem_bytes"] > 0) == (layout == "shared")
        heads.append(h.cpu().numpy())
    assert np.abs(heads[0] - heads[1]).max() < 1e-9 / 0.3048
