"""Cylinder lengths at which a cone forward kernel's shared memory comes just
under the 48 KB that a launch has without opting in: its static arrays count
against them too."""

import numpy as np
import pytest
import torch

import mbirtorch_b200 as mb
from mbirtorch_b200 import kernels

pytestmark = pytest.mark.gpu


def _step(V, R, C, N, S, weighted):
    m = mb.ConeBeamModel((V, R, C), np.linspace(0, 2 * np.pi, V, endpoint=False), 12.0 * S, 6.0 * S)
    m.set_params(no_warning=True, verbose=0, delta_det_channel=2.0, delta_det_row=2.0)
    m.auto_set_recon_geometry(no_warning=True)
    m.set_params(no_warning=True, recon_shape=(N, N, S), sigma_y=0.5, sigma_x=0.2)
    w = torch.rand((V, R, C), device='cuda') + 0.5 if weighted else None
    upd = m.create_vcd_subset_updater(m.compute_hessian_diagonal(weights=w),
                                      weights=1 if w is None else w)
    err = torch.rand((V, R, C), device='cuda')
    cost = (lambda e: float((e * e).sum())) if w is None else (lambda e: float((w * e * e).sum()))
    before = cost(err)
    idx = torch.arange(5, N * N, 9, device='cuda')
    flat, err, _, alpha, _ = upd(torch.zeros((N * N, S), device='cuda'), err, idx)
    assert float(alpha) > 1e-3 and cost(err) < before


@pytest.mark.parametrize('S', [685, 688, 692, 693, 696, 697, 700])
@pytest.mark.parametrize('R', [200, 320])
def test_subset_step(S, R):
    """The streamed line search; its step lowers the data fit."""
    _step(8, R, 40, 24, S, False)


@pytest.mark.parametrize('weighted', [False, True])
@pytest.mark.parametrize('R,S', [(1000, 1570), (1000, 1650), (1000, 1648), (1024, 1770)])
def test_subset_step_that_one_kernel_alone_can_hold(R, S, weighted):
    """Long cylinders on detectors of 1000 rows: where a forward kernel's staging
    no longer fits shared memory, the other takes the step."""
    _step(4, R, 30, 12, S, weighted)


@pytest.mark.parametrize('band', range(270, 292, 2))
def test_slice_band_forward(band):
    V, R, C, N, S = 5, 200, 30, 24, 600
    g = kernels.make_geometry('cone', V, R, C, N, N, S, 1, 1, False, 2.0, 2.0, 0.0, 0.0, 1.0, 1.0,
                              1.0, 0.0, 2.0, 12.0 * S)
    vp = np.stack([np.linspace(0, 3, V), np.zeros(V)], axis=1).astype(np.float32)
    proj = kernels.DeviceProjector(g, vp, torch.device('cuda', 0))
    idx = torch.arange(0, N * N, 7, device='cuda')
    x = torch.rand((idx.numel(), band), device='cuda')
    cut = band // 2
    whole = proj.forward(x, idx, slice_start=150)
    halves = proj.forward(x[:, :cut].contiguous(), idx, slice_start=150) + \
        proj.forward(x[:, cut:].contiguous(), idx, slice_start=150 + cut)
    assert float((whole - halves).norm() / halves.norm()) <= 2e-6
