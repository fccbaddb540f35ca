"""The power function of the link and emitter coefficients: the head-loss and
emitter exponents a network can have, link flows over eight decades."""
import numpy as np
import pytest
import torch

from oracle.gga import Model
from wdsgpu_b200 import GGASolver, implicit_solve, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-5, 1e-2, 1.0, 1.5])
@pytest.mark.parametrize("form,qexp", [("H-W", 2.0), ("H-W", 1.5), ("C-M", 2.0), ("C-M", 1.0 / 0.6)])
def test_exponents_and_flow_decades(form, qexp, scale):
    # polished heads are the Newton fixed point (1e-9 m), gradients follow
    # from one refined adjoint solve on the terminal factor (1e-8 relative)
    net = synth.looped_network(3, 100, 1, 120, n_emitters=5)
    net.meta.update(headloss=form, qexp=qexp)
    d, _ = synth.config2_scenarios(net, 3, seed=11)
    d = d * scale
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    s = GGASolver(net, device="cuda:0", dense_status_machine=True)
    D = torch.tensor(d, device="cuda:0", requires_grad=True)
    h, q, e = implicit_solve(s, D, torch.tensor(rh, device="cuda:0"), accuracy=1e-7)
    (h ** 2).sum().backward()
    m = Model(net)
    out, st = m.implicit(d, rh, accuracy=1e-7, polish_steps=3)
    gd = m.backward(st, 2.0 * out["head_ft"], np.zeros_like(out["flow_cfs"]),
                    np.zeros_like(out["emitter_cfs"]))[0]
    assert np.abs(h.detach().cpu().numpy() - out["head_ft"]).max() < 1e-9 / 0.3048
    assert np.abs(D.grad.cpu().numpy() - gd).max() < 1e-8 * np.abs(gd).max()
