"""Large-network layout (tables in global memory, one CTA per scenario): bitwise
equal to the shared-memory layout where both apply, and correct against the
oracle on networks too large for shared memory, with control valves too; the
per-warp rounds of the factorisation and the substitutions, with lists of one
entry (a tree) to hundreds (no top block), levels of one item to thousands,
against the oracle."""
import numpy as np
import pytest
import torch

from oracle.gga import Model
from wdsgpu_b200 import GGASolver, implicit_solve, synth

pytestmark = pytest.mark.gpu

POLISHED_HEAD_ATOL_FT = 1e-9 / 0.3048


def _run(net, cuda, layout, d, rh, B):
    s = GGASolver(net, device=cuda, dense_status_machine=True)
    s.sm100_layout = layout
    ke = s.node_ke_default.unsqueeze(0).contiguous()
    r = s.r_hw.unsqueeze(0).contiguous()
    o = s.run(torch.tensor(d, device=cuda), torch.tensor(rh, device=cuda), ke, r, B, 200,
              1e-6, True, 3)
    torch.cuda.synchronize()
    return s, o


@pytest.mark.parametrize("which", ["config2", "feature"])
def test_global_layout_equals_shared_layout_bitwise(cuda, which):
    net = synth.config2_network() if which == "config2" else synth.feature_network()
    B = 6
    d, rh = synth.config2_scenarios(net, B, seed=21, sigma=0.3)
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    s1, a = _run(net, cuda, "shared", d, rh, B)
    s2, b = _run(net, cuda, "global", d, rh, B)
    assert s1.plan_stats(B)["smem_bytes"] > 0 and s2.plan_stats(B)["smem_bytes"] == 0
    for k in ("head", "flow", "emit", "status", "iters", "info"):
        assert torch.equal(a[k], b[k]), k
    # adjoint on the kept terminal state
    for s in (s1, s2):
        D = torch.tensor(d, device=cuda, requires_grad=True)
        h = implicit_solve(s, D, torch.tensor(rh, device=cuda), accuracy=1e-6)[0]
        (h ** 2).sum().backward()
        s._g = D.grad.clone()
    assert torch.equal(s1._g, s2._g)


def test_network_beyond_shared_memory_matches_oracle(cuda):
    """3000 junctions / 3600 pipes: the plan falls back to the global layout;
    iterations exact, polished heads within 1e-9 m, gradients within 1e-6."""
    net = synth.config3_networks()[3]
    B = 2
    d, rh = synth.config2_scenarios(net, B, seed=5, sigma=0.3)
    s = GGASolver(net, device=cuda, dense_status_machine=True)
    assert s.plan_stats(B)["smem_bytes"] == 0                 # global layout chosen
    D = torch.tensor(d, device=cuda, requires_grad=True)
    sens = synth.sensor_nodes(net, 30)
    h, q, e = implicit_solve(s, D, torch.tensor(rh, device=cuda), accuracy=1e-9)
    (h[:, sens] ** 2).sum().backward()
    m = Model(net)
    o, st = m.implicit(d, rh, accuracy=1e-9)
    assert np.abs(h.detach().cpu().numpy() - o["head_ft"]).max() <= POLISHED_HEAD_ATOL_FT
    assert np.abs(q.detach().cpu().numpy() - o["flow_cfs"]).max() <= 1e-9
    gH = np.zeros((B, net.N))
    gH[:, sens] = 2.0 * o["head_ft"][:, sens]
    gd = m.backward(st, gH, np.zeros((B, net.L)), np.zeros((B, net.N)))[0]
    g = D.grad.cpu().numpy()
    assert np.abs(g - gd).max() <= 1e-6 * np.abs(gd).max()
    f = s.solve(d, rh, status_machine=True, accuracy=1e-6)
    ref = m.solve(d, rh, accuracy=1e-6, status_machine=True)
    assert np.array_equal(f["iters"].cpu().numpy(), ref["iters"])


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


@pytest.mark.parametrize("links,prv,zone,B", [(2640, 3, (25, 70), 2), (2310, 36, (4, 30), 1)])
def test_control_valves_of_large_networks(cuda, links, prv, zone, B):
    """Valve, link-status and Woodbury passes of the 1024-thread layout (a lane
    of the last warp per valve: 36 take two turns): iterations and statuses
    exact, polished heads within 1e-9 m, flows within 1e-9 cfs, gradients within
    1e-6 of the largest."""
    net = synth.looped_network(2, 2200, 2, links, n_prv=prv, n_emitters=20, zone_size=zone)
    d, rh = synth.config2_scenarios(net, B, seed=5, sigma=0.3)
    rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
    s = GGASolver(net, device=cuda, dense_status_machine=True)
    st0 = s.plan_stats(B)
    assert st0["smem_bytes"] == 0 and st0["n_prv"] == prv
    m = Model(net)
    f = s.solve(d, rh, status_machine=True, accuracy=1e-6)
    ref = m.solve(d, rh, accuracy=1e-6, status_machine=True)
    assert np.array_equal(f["iters"].cpu().numpy(), ref["iters"])
    assert np.array_equal(f["status"].cpu().numpy(), ref["status"])
    D = torch.tensor(d, device=cuda, requires_grad=True)
    h, q, e = implicit_solve(s, D, torch.tensor(rh, device=cuda), accuracy=1e-7)
    assert (f["status"][:, torch.as_tensor(s.pcv_links, device=cuda)] == 4).any()   # ACTIVE
    (h ** 2).sum().backward()
    o, st = m.implicit(d, rh, accuracy=1e-7, polish_steps=3)
    assert np.abs(h.detach().cpu().numpy() - o["head_ft"]).max() <= POLISHED_HEAD_ATOL_FT
    assert np.abs(q.detach().cpu().numpy() - o["flow_cfs"]).max() <= 1e-9
    gd = m.backward(st, 2.0 * o["head_ft"], np.zeros((B, net.L)), np.zeros((B, net.N)))[0]
    assert np.abs(D.grad.cpu().numpy() - gd).max() <= 1e-6 * np.abs(gd).max()
