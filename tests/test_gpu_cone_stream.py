"""The streamed cone forward at the sizes where it can go wrong: rows around
its 64-row warps, cylinders that are not a multiple of four slices, channels
that are not a multiple of its blocks, flat slices (its general footprint
form), and the subset step's forward on the row counts that take it.

Bars: a row's centre slice k_m = (m - m0) / w_r is formed in FP32 from m0, so
its error is two roundings of a number up to the slice count S, S 2^-23 in
all, and so much of a voxel's value may land on its neighbour: with random
voxels of either sign that is the relative error of a row.  Short cylinders
keep the 1e-5 of the other projector tests (FP32 sums and geometry), the step
size its 1e-4.  Where slices under half a row tall outnumber the taps, the
taps' choice jumps with the rounding of k_m, in FP32 as in FP64, so there the
bar is against the FP32 kernel of slice bands (1e-6: the same taps, other
roundings)."""

import numpy as np
import pytest
import torch

import mbirtorch_b200 as mb
import oracle
from conftest import rel_l2
from mbirtorch_b200 import kernels
from oracle import OracleGeometry
from oracle import vcd as ovcd

pytestmark = pytest.mark.gpu


def _geometry(V, R, C, N, S, dvs=1.0, bp=1, curved=False):
    og = OracleGeometry(num_det_rows=R, num_det_channels=C, num_recon_rows=N, num_recon_cols=N,
                        num_slices=S, delta_det_channel=2.0, delta_det_row=2.0,
                        det_channel_offset=0.6, det_row_offset=-0.9, delta_voxel=1.0,
                        delta_voxel_row=1.0, delta_voxel_slice=dvs, recon_slice_offset=0.4,
                        magnification=2.0, source_detector_dist=8.0 * N, psf_radius=1,
                        bp_psf_radius=bp, use_curved_detector=curved)
    g = kernels.make_geometry('cone', V, R, C, N, N, S, 1, bp, curved, 2.0, 2.0, 0.6, -0.9, 1.0,
                              1.0, dvs, 0.4, 2.0, 8.0 * N)
    ang = np.linspace(0, 2 * np.pi, V, endpoint=False)
    vp = np.stack([ang, np.linspace(-2, 2, V)], axis=1).astype(np.float32)
    return og, g, vp


@pytest.mark.parametrize('R,S,C,dvs', [
    (1, 1, 7, 1.0), (31, 17, 33, 1.0), (32, 32, 48, 1.0), (33, 40, 50, 1.0), (64, 64, 40, 1.0),
    (65, 52, 47, 1.0), (128, 130, 40, 1.0), (129, 96, 61, 1.0), (200, 201, 40, 1.0),
    (320, 256, 37, 1.0),
    (70, 60, 45, 0.35),    # slices under half a row tall: the general form
    (70, 60, 45, 0.52),    # both forms, by the pixel's magnification
])
def test_whole_cylinders_match_oracle(R, S, C, dvs):
    N, V = 26, 9
    og, g, vp = _geometry(V, R, C, N, S, dvs=dvs, curved=R % 2 == 0)
    rng = np.random.default_rng(R + S)
    idx = np.sort(rng.choice(N * N, size=300, replace=False)).astype(np.int64)
    x = rng.standard_normal((idx.size, S)).astype(np.float32)
    dev = torch.device('cuda', 0)
    proj = kernels.DeviceProjector(g, vp, dev)
    values, pix = torch.as_tensor(x, device=dev), torch.as_tensor(idx, device=dev)
    if dvs < 0.5:
        bar, half = 1e-6, S // 2
        want = sum(proj.forward(values[:, a:b].contiguous(), pix, slice_start=a)
                   for a, b in ((0, half), (half, S))).cpu().numpy()
    else:
        bar = max(1e-5, S * 2.0 ** -23)
        want = oracle.cone_forward(og, vp.astype(np.float64), x, idx)
    assert rel_l2(proj.forward(values, pix).cpu().numpy(), want) <= bar
    # a cylinder array that is not 16-byte aligned takes the 4-byte copies
    shifted = torch.empty(x.size + 1, device=dev)[1:].view(x.shape)
    shifted.copy_(values)
    got = proj.forward(shifted, pix)
    assert rel_l2(got.cpu().numpy(), want) <= bar
    assert torch.equal(got, proj.forward(shifted, pix))


def test_nonfinite_voxels_reach_the_rows_of_the_three_tap_form():
    """An infinite or NaN voxel reaches the rows whose centre slice is within
    one of it, and no others (the taps of zero weight included)."""
    N, V, R, S, C = 24, 5, 100, 64, 40
    og, g, vp = _geometry(V, R, C, N, S)
    dev = torch.device('cuda', 0)
    proj = kernels.DeviceProjector(g, vp, dev)
    idx = torch.arange(N * N, device=dev)
    for bad in (float('inf'), float('nan')):
        x = torch.ones((N * N, S), device=dev)
        x[N * (N // 2) + 5, 30] = bad
        got = proj.forward(x, idx)
        # the slice band form keeps one row per thread and the clamped weights
        band = torch.zeros_like(got)
        for s0, s1 in ((0, 40), (40, S)):
            band += proj.forward(x[:, s0:s1].contiguous(), idx, slice_start=s0)
        assert torch.equal(torch.isfinite(got), torch.isfinite(band))


@pytest.mark.parametrize('R,S,weighted,storage', [
    (100, 96, False, 'float32'), (128, 128, True, 'float32'), (129, 70, False, 'float32'),
    (200, 161, True, 'float32'), (256, 256, False, 'float32'), (320, 200, True, 'float16'),
])
def test_subset_step_matches_oracle(R, S, weighted, storage):
    N, V, C = 40, 16, 53
    ang = np.linspace(0, 2 * np.pi, V, endpoint=False)
    m = mb.ConeBeamModel((V, R, C), ang, source_detector_dist=8.0 * N, source_iso_dist=4.0 * N)
    m.set_params(no_warning=True, verbose=0, delta_det_channel=2.0, delta_det_row=2.0)
    m.auto_set_recon_geometry(no_warning=True)
    m.set_params(no_warning=True, recon_shape=(N, N, S), sigma_y=0.5, sigma_x=0.2)
    m.set_storage_precision(storage)
    g = m._geometry()
    og = OracleGeometry(num_det_rows=R, num_det_channels=C, num_recon_rows=N, num_recon_cols=N,
                        num_slices=S, delta_det_channel=2.0, delta_det_row=2.0,
                        delta_voxel=g.delta_voxel, delta_voxel_row=g.delta_voxel_row,
                        delta_voxel_slice=g.delta_voxel_slice, magnification=g.magnification,
                        recon_slice_offset=g.recon_slice_offset,
                        source_detector_dist=g.source_detector_dist, psf_radius=g.psf_radius,
                        bp_psf_radius=g.bp_psf_radius)
    rng = np.random.default_rng(R)
    y = rng.standard_normal((V, R, C)).astype(np.float32)
    w = rng.uniform(0.5, 1.5, (V, R, C)).astype(np.float32) if weighted else None
    x0 = (0.1 * rng.random((N, N, S))).astype(np.float32)
    H = m.compute_hessian_diagonal(weights=w)
    dev = torch.device('cuda', 0)
    upd = m.create_vcd_subset_updater(H, weights=1 if w is None else torch.as_tensor(w, device=dev))
    sub = np.sort(rng.choice(mb.gen_full_indices((N, N, S)), size=90, replace=False)).astype(np.int64)
    flat = torch.as_tensor(x0.reshape(-1, S), device=dev).clone()
    err = torch.as_tensor(y, device=dev).clone()
    flat, err, _, alpha, _ = upd(flat, err, torch.as_tensor(sub, device=dev))
    prob = ovcd.Problem('cone', og, m._view_params_array().astype(np.float64), (N, N, S),
                        source_iso_dist=4.0 * N)
    ou = ovcd.SubsetUpdater(prob, H.reshape(-1, S), w, 0.5, 0.2,
                            dc_profile=ovcd.dc_damping_profile(prob))
    oflat, oerr = x0.reshape(-1, S).astype(np.float64), y.astype(np.float64)
    _, oalpha, _ = ou(oflat, oerr, sub)
    # 16-bit storage rounds the stored residual: 2^-11 of its size
    bar = 1e-5 if storage == 'float32' else 1e-3
    assert abs(float(alpha) - oalpha) <= 10 * bar * abs(oalpha)
    assert rel_l2(flat.cpu().numpy(), oflat) <= bar
    assert rel_l2(err.cpu().numpy(), oerr) <= bar
