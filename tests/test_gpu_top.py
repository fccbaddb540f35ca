"""Dense top block of the elimination tree: every number of 4-column blocks
and 8-row tiles, full and partial, against the oracle."""
import numpy as np
import pytest
import torch

from oracle.gga import Model
from wdsgpu_b200 import GGASolver, implicit_solve, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["shared", "global"])
@pytest.mark.parametrize("top", [-1, 3, 4, 5, 7, 8, 9, 12, 15, 16, 17, 24, 31, 33, 40, 41, 48])
def test_top_block_sizes(top, layout):
    # polished heads are the Newton fixed point (1e-9 m), gradients follow
    # from one refined adjoint solve on the terminal factor (1e-8 relative)
    net = synth.looped_network(3, 100, 1, 120, n_emitters=5)
    d, _ = synth.config2_scenarios(net, 3, seed=11)
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    s = GGASolver(net, device="cuda:0", dense_status_machine=True)
    s.sm100_tuning = dict(top_max=top)
    s.sm100_layout = layout
    D = torch.tensor(d, device="cuda:0", requires_grad=True)
    h, q, e = implicit_solve(s, D, torch.tensor(rh, device="cuda:0"), accuracy=1e-7)
    (h ** 2).sum().backward()
    m = Model(net)
    out, st = m.implicit(d, rh, accuracy=1e-7, polish_steps=3)
    gd = m.backward(st, 2.0 * out["head_ft"], np.zeros_like(out["flow_cfs"]),
                    np.zeros_like(out["emitter_cfs"]))[0]
    assert np.abs(h.detach().cpu().numpy() - out["head_ft"]).max() < 1e-9 / 0.3048
    assert np.abs(D.grad.cpu().numpy() - gd).max() < 1e-8 * np.abs(gd).max()
