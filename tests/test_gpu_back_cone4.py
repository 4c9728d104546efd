"""The cone back projector with vector columns and slice pairs, at the edges
of its row groups (128), slice chunks (64 to 256) and forms: slices inside the
column buffer's padding, beyond it (helical shifts), and taller than two rows.

Bar: a slice's row m_p = m0 + w_r k is formed in FP32, so its error is two
roundings of a number up to the detector's rows R, R 2^-23 in all, and so much
of a cell's value may land on its neighbour: with random cells of either sign
that is the relative error of a (view, voxel) term.  Short detectors keep the
1e-5 of the other projector tests."""

import numpy as np
import pytest
import torch

import oracle
from conftest import rel_l2
from mbirtorch_b200 import _lib, kernels
from oracle import OracleGeometry

pytestmark = pytest.mark.gpu


def _setup(R, S, dvs, shift, N=14, V=37, C=30):
    og = OracleGeometry(num_det_rows=R, num_det_channels=C, num_recon_rows=N, num_recon_cols=N,
                        num_slices=S, delta_det_channel=2.0, delta_det_row=2.0,
                        det_channel_offset=-0.4, det_row_offset=0.8, delta_voxel=1.0,
                        delta_voxel_row=1.0, delta_voxel_slice=dvs, recon_slice_offset=-0.3,
                        magnification=2.0, source_detector_dist=40.0 * N, psf_radius=1)
    g = kernels.make_geometry('cone', V, R, C, N, N, S, 1, 1, False, 2.0, 2.0, -0.4, 0.8, 1.0,
                              1.0, dvs, -0.3, 2.0, 40.0 * N)
    ang = np.linspace(0, 2 * np.pi, V, endpoint=False)
    vp = np.stack([ang, np.linspace(-shift, shift, V)], axis=1).astype(np.float32)
    return og, kernels.DeviceProjector(g, vp, torch.device('cuda', 0)), vp


@pytest.mark.parametrize('power', [1, 2])
@pytest.mark.parametrize('R,S,dvs,shift', [
    (4, 33, 1.0, 0.0), (36, 64, 1.0, 0.0), (64, 65, 1.0, 30.0), (128, 128, 1.0, 0.0),
    (132, 129, 0.7, 3.0), (256, 200, 1.0, 0.0), (260, 256, 1.0, 60.0), (320, 257, 1.0, 0.0),
    (388, 300, 1.1, 5.0), (520, 256, 1.9, 0.0),
    (64, 70, 2.03, 0.0),   # slices around two rows tall: both tap forms
])
def test_back_matches_oracle(R, S, dvs, shift, power):
    og, proj, vp = _setup(R, S, dvs, shift)
    V, C = proj.geom.num_views, proj.geom.num_det_channels
    rng = np.random.default_rng(R + S)
    idx = np.sort(rng.choice(14 * 14, size=61, replace=False)).astype(np.int64)
    y = rng.standard_normal((V, R, C)).astype(np.float32)
    sino, pix = torch.as_tensor(y).cuda(), torch.as_tensor(idx).cuda()
    got = proj.back(sino, pix, coeff_power=power)
    want = oracle.cone_back(og, vp.astype(np.float64), y, idx, power)
    assert rel_l2(got.cpu().numpy(), want) <= max(1e-5, R * 2.0 ** -23)
    vcr = sino.transpose(1, 2).contiguous()
    assert torch.equal(got, proj.back(vcr, pix, coeff_power=power, layout=_lib.MBIR_LAYOUT_VCR))
    # a slice band of more than 32 slices takes the same kernel
    if S > 80:
        s0 = S - 70
        band = proj.back(sino, pix, coeff_power=power, slice_start=s0, band_slices=70)
        assert rel_l2(band.cpu().numpy(), want[:, s0:]) <= max(1e-5, R * 2.0 ** -23)
    # a sinogram that is not 16-byte aligned takes the scalar columns
    off = torch.empty(vcr.numel() + 1, device='cuda')[1:].view(vcr.shape)
    off.copy_(vcr)
    scalar = proj.back(off, pix, coeff_power=power, layout=_lib.MBIR_LAYOUT_VCR)
    assert rel_l2(got.cpu().numpy(), scalar.cpu().numpy()) <= max(2e-6, R * 2.0 ** -23)


def test_nonfinite_cells_reach_the_same_voxels():
    _, proj, _ = _setup(64, 70, 1.0, 0.0)
    idx = torch.arange(14 * 14, device='cuda')
    for bad in (float('inf'), float('nan')):
        y = torch.ones((proj.geom.num_views, proj.geom.num_det_channels, 64), device='cuda')
        y[3, 15, 30] = bad
        off = torch.empty(y.numel() + 1, device='cuda')[1:].view(y.shape)
        off.copy_(y)
        a = proj.back(y, idx, layout=_lib.MBIR_LAYOUT_VCR)
        b = proj.back(off, idx, layout=_lib.MBIR_LAYOUT_VCR)
        assert torch.equal(torch.isfinite(a), torch.isfinite(b))
