"""The persistent network kernels at the edges of their tiling: one tile, a tile
that straddles the x and y faces of a case or two cases (nx ny an odd multiple
of 64), as many tiles as blocks and more, rectangular grids.  A face's correction
does not depend on its place in a tile, so a batch's corrections are those of
its cases alone bit for bit; the gradient is compared with the CPU FP64
restatement with the bounds of tests/test_nn.py (BF16 operands rounded at the
same points, FP32 accumulation: 2e-3 per parameter block)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import nn_oracle

pytestmark = pytest.mark.gpu


def states(batch, nx, ny, seed):
    rng = np.random.default_rng(seed)
    y, x = np.meshgrid(np.arange(ny) / ny, np.arange(nx) / nx, indexing="ij")
    out = np.zeros((batch, 4, ny, nx))
    for b in range(batch):
        ph = rng.uniform(0, 2 * np.pi, 4)
        rho = 1.0 + 0.2 * np.sin(2 * np.pi * x + ph[0]) * np.cos(2 * np.pi * y + ph[1])
        u = 0.5 * np.sin(2 * np.pi * y + ph[2])
        v = 0.5 * np.cos(2 * np.pi * x + ph[3])
        p = 1.0 + 0.1 * np.cos(2 * np.pi * (x + y) + ph[0])
        out[b] = np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])
    return out


@pytest.mark.parametrize("batch,nx,ny", [(1, 8, 8), (3, 24, 8), (1, 8, 40), (7, 16, 16), (30, 40, 32), (51, 40, 40)])
def test_forward_and_gradient_match_cpu(batch, nx, ny):
    from dev_field_efvm_b200.device import FluxNet

    net = FluxNet(out_scale=1e-2, seed=11)
    rng = np.random.default_rng(batch)
    p = net.params().astype(np.float64)
    p[nn_oracle.P_W3:nn_oracle.P_B1] = rng.normal(0, 0.3, nn_oracle.NOUT * nn_oracle.H)
    p[nn_oracle.P_B1:] = rng.normal(0, 0.1, nn_oracle.P_COUNT - nn_oracle.P_B1)
    p = p.astype(np.float32)
    net.set_params(p)
    s = states(batch, nx, ny, 3)
    resid = rng.normal(0, 1e-2, s.shape)
    dx, dy, w = 10.0 / nx, 10.0 / ny, [1.0, 2.0, 2.0, 0.5]
    st = torch.tensor(s, device="cuda")
    corr = torch.zeros((batch, 2, 4, ny, nx), dtype=torch.float32, device="cuda")
    net.forward(st, corr)
    grad = torch.zeros(net.P, dtype=torch.float32, device="cuda")
    loss = net.loss_grad(st, torch.tensor(resid, device="cuda"), dx, dy, w, grad)
    for b in range(batch):
        alone = torch.zeros((1, 2, 4, ny, nx), dtype=torch.float32, device="cuda")
        net.forward(st[b:b + 1].contiguous(), alone)
        assert torch.equal(alone[0], corr[b])
    ref_loss, ref, _ = nn_oracle.loss_grad(p.astype(np.float64), s, resid, dx, dy, w, 1e-2)
    assert abs(loss - ref_loss) <= 1e-5 * ref_loss
    g, full = grad.cpu().numpy().astype(np.float64), np.linalg.norm(ref)
    cuts = [nn_oracle.P_W1, nn_oracle.P_W2, nn_oracle.P_W3, nn_oracle.P_B1, nn_oracle.P_B2, nn_oracle.P_B3,
            nn_oracle.P_COUNT]
    for k, (a, b) in enumerate(zip(cuts[:-1], cuts[1:])):
        diff = np.linalg.norm(g[a:b] - ref[a:b])
        # the output bias's gradient telescopes to round-off: judged against the whole
        assert diff < (1e-4 * full if k == 5 else 2e-3 * np.linalg.norm(ref[a:b])), (k, diff)
    pad = g[:nn_oracle.P_W2].reshape(nn_oracle.H, nn_oracle.K1)[:, nn_oracle.IN:]
    assert not pad.any()
