"""Error of one linear solve on stiff node matrices (links without flow beside
ordinary ones, conductances over seven decades and more), where the dense top
block holds most of the columns."""
import numpy as np
import pytest
import torch

from wdsgpu_b200 import GGASolver, synth

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _system(net, s, q, d, rh, dtype):
    """Node matrix and right-hand side of the first iteration from flows q."""
    n1, n2 = np.asarray(net.link_n1), np.asarray(net.link_n2)
    junc = np.flatnonzero(np.asarray(net.node_type) == 0)
    row = np.full(net.N, -1)
    row[junc] = np.arange(junc.size)
    q, r, ex = q.astype(dtype), s.r_hw.cpu().numpy().astype(dtype), dtype(s.hexp)
    hg = ex * r * np.power(np.maximum(np.abs(q), dtype(1e-30)), ex - 1)
    lin = hg < dtype(s.rqtol)
    P = 1 / np.where(lin, dtype(s.rqtol), hg)
    z = np.where(lin, q, q / ex) - q
    A, F = np.zeros((junc.size, junc.size), dtype), -d[junc].astype(dtype)
    for k in range(net.L):
        a, b = row[n1[k]], row[n2[k]]
        if a >= 0:
            A[a, a] += P[k]
            F[a] += z[k] + (P[k] * dtype(rh[n2[k]]) if b < 0 else 0)
        if b >= 0:
            A[b, b] += P[k]
            F[b] -= z[k] - (P[k] * dtype(rh[n1[k]]) if a < 0 else 0)
        if a >= 0 and b >= 0:
            A[a, b] -= P[k]
            A[b, a] -= P[k]
    return junc, A, F


def _solve(A, F):
    A, x = A.copy(), F.copy()
    n = x.size
    for i in range(n):
        f = A[i + 1:, i] / A[i, i]
        A[i + 1:] -= np.outer(f, A[i])
        x[i + 1:] -= f * x[i]
    for i in range(n - 1, -1, -1):
        x[i] = (x[i] - A[i, i + 1:] @ x[i + 1:]) / A[i, i]
    return x


def _sweeps(A):
    """Inverse by symmetric sweeps of one column at a time, in double."""
    D = 2.0 ** -np.round(np.floor(np.log2(np.diag(A))) / 2)
    S = A * D[:, None] * D
    for k in range(len(S)):
        p, c = S[k, k], S[:, k].copy()
        c[k] = p - 1.0
        S = S - np.outer(c / p, c)
        S[k, k] = -1.0 / p
    return -S * D[:, None] * D


def test_unrefined_solve_is_as_accurate_as_single_column_sweeps(cuda):
    # 960 systems of 7 to 45 junctions: the geometric mean of the error against
    # 80-bit elimination, in units of the one by single-column sweeps in double.
    # Its spread is about a factor of e per system, so 3 % over all of them; 1.1
    # is three times that above equality.
    ratio = []
    for nj, links in ((7, 7), (12, 14), (20, 24), (33, 40), (45, 60)):
        for seed in range(1, 33):
            net = synth.looped_network(seed, nj, 1, links)
            s = GGASolver(net, device=cuda, dense_status_machine=True)
            d, _ = synth.config2_scenarios(net, 6, seed=seed)
            rh = np.broadcast_to(np.nan_to_num(net.fixed_head_ft_at(0)), d.shape).copy()
            rng = np.random.default_rng(seed)
            q0 = rng.normal(size=(6, net.L)) * 0.5
            for b in (1, 4):
                q0[b, rng.random(net.L) < 0.3] = 0.0
            for b in (2, 5):
                q0[b] *= 10.0 ** rng.uniform(-7, 1, net.L)
            o = s.solve(d, rh, status_machine=True, accuracy=1e-6, max_iter=1,
                        q0=torch.tensor(q0, device=cuda),
                        e0=torch.zeros(6, net.N, dtype=torch.float64, device=cuda))
            h = o["head_ft"].cpu().numpy()
            for b in range(6):
                junc, A, F = _system(net, s, q0[b], d[b], rh[b], LD)
                x = _solve(A, F)
                _, A, F = _system(net, s, q0[b], d[b], rh[b], np.float64)
                err = [float(np.abs(v - x).max() / np.abs(x).max())
                       for v in (h[b, junc], _sweeps(A) @ F)]
                ratio.append(np.log((err[0] + 1e-18) / (err[1] + 1e-18)))
    assert np.exp(np.mean(ratio)) <= 1.1
