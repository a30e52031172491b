"""Smoothing over stored neighbour rows: trees larger than one slice of rows."""
import numpy as np
import pytest

from nbodylib_gb300 import KDTree

pytestmark = pytest.mark.gpu


def test_more_particles_than_a_slice(gpu):
    """CalcSmoothVel on 2^23 + 3 particles (two slices) against the same sums formed in torch
    from FindNearest's rows: relative to the largest component, 1e-12 as the path's."""
    import torch
    n, k = (1 << 23) + 3, 4
    g = torch.Generator(device="cuda").manual_seed(3)
    pos, vel = (torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64) for _ in range(2))
    mass = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) + 0.5
    rho = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) + 0.5
    t = KDTree(pos, vel, mass, 16, kerntype=0, device=True)
    got = t.CalcSmoothVel(k, rho)
    nn, d2 = t.FindNearest(k)
    perm = t.GetPerm().long()
    table = torch.from_numpy(np.asarray(t.GetKernel()[0])).cuda()
    h = 0.5 * torch.sqrt(d2[:, -1:])
    u = torch.sqrt(d2) / h * (0.5 * (table.numel() - 1))
    i = u.long().clamp_max(table.numel() - 2)
    w = table[i] + (table[i + 1] - table[i]) * (u - i.double())
    w[:, -1] = table[-1]
    w = 0.5 * w / h ** 3
    me, them = perm[:, None].expand(-1, k), perm[nn.long()]
    want = torch.zeros_like(got)
    for d in range(3):
        want[:, d].index_add_(0, me.reshape(-1),
                              (w * mass[them] / rho[them] * vel[them, d]).reshape(-1))
        want[:, d].index_add_(0, them.reshape(-1),
                              (w * mass[me] / rho[me] * vel[me, d]).reshape(-1))
    worst = ((got - want).abs() / want.abs().max()).max().item()
    assert worst <= 1e-12, worst
