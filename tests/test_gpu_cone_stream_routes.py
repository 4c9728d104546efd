"""Which cone forward kernel a projection takes (rows, pixels a tile, CTAs, the
cylinders' length and alignment) changes its time and the order of its sums,
nothing else: both sides of each line against the FP64 oracle, at detectors
that reach the streamed kernel, and few-CTA calls that stay with the kernel of
one row per thread.

Bars as in the streamed kernel's own tests: 1e-5, or S 2^-23 for long
cylinders, whose centre slices are formed in FP32."""

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


def _setup(V, R, C, N, S):
    og = OracleGeometry(num_det_rows=R, num_det_channels=C, num_recon_rows=N, num_recon_cols=N,
                        num_slices=S, delta_det_channel=2.0, delta_det_row=2.0,
                        det_channel_offset=0.6, det_row_offset=-0.9, delta_voxel=1.0,
                        delta_voxel_row=1.0, delta_voxel_slice=1.0, recon_slice_offset=0.4,
                        magnification=2.0, source_detector_dist=12.0 * max(N, S), psf_radius=1)
    g = kernels.make_geometry('cone', V, R, C, N, N, S, 1, 1, False, 2.0, 2.0, 0.6, -0.9, 1.0,
                              1.0, 1.0, 0.4, 2.0, 12.0 * max(N, S))
    ang = np.linspace(0, 2 * np.pi, V, endpoint=False)
    vp = np.stack([ang, np.linspace(-2, 2, V)], axis=1).astype(np.float32)
    return og, kernels.DeviceProjector(g, vp, torch.device('cuda', 0)), vp


def _views(ctas_per_sm, C):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return -(-ctas_per_sm * sms // ((C + 15) // 16)) + 1


def _check(V, R, C, N, S, P, few_views=9):
    """The forward of P pixels over V views; a few of the views against the
    oracle, all of them against the kernel of slice bands (another order of
    sums)."""
    og, proj, vp = _setup(V, R, C, N, S)
    rng = np.random.default_rng(R + S)
    idx = np.sort(rng.choice(N * N, size=P, replace=False)).astype(np.int64)
    x = rng.standard_normal((P, S)).astype(np.float32)
    values, pix = torch.as_tensor(x).cuda(), torch.as_tensor(idx).cuda()
    got = proj.forward(values, pix)
    bar = max(1e-5, S * 2.0 ** -23)
    seen = np.linspace(0, V - 1, few_views).astype(int)
    want = oracle.cone_forward(og, vp[seen].astype(np.float64), x, idx)
    assert rel_l2(got[torch.as_tensor(seen, device='cuda')].cpu().numpy(), want) <= bar
    half = max(1, S // 2)
    bands = proj.forward(values[:, :half].contiguous(), pix, slice_start=0)
    if half < S:
        bands += proj.forward(values[:, half:].contiguous(), pix, slice_start=half)
    assert float((got - bands).norm() / bands.norm()) <= bar
    # views in two calls: the same kernel, the same bits
    cut = V // 3
    parts = [proj.forward(values, pix, view_start=0, view_count=cut),
             proj.forward(values, pix, view_start=cut, view_count=V - cut)]
    assert torch.equal(got, torch.cat(parts))
    return got, proj, values, pix


@pytest.mark.parametrize('R,S,per_sm,P', [
    (17, 20, 3, 60), (17, 20, 3, 120), (32, 32, 3, 120), (32, 32, 18, 120),   # n = 21 and 43
    (19, 17, 3, 180), (19, 17, 3, 240), (19, 17, 13, 240),                     # slice by slice
    (9, 9, 3, 40), (9, 9, 3, 60), (16, 482, 3, 60), (16, 479, 3, 60),
    (50, 48, 23, 60), (50, 48, 25, 60), (64, 64, 25, 60), (64, 64, 25, 24), (64, 484, 3, 60),
    (97, 96, 5, 60), (128, 128, 7, 60), (128, 127, 7, 60), (100, 480, 3, 60),
    (130, 129, 13, 60), (130, 129, 15, 60), (150, 149, 6, 60), (150, 149, 8, 60), (150, 148, 8, 60),
    (161, 160, 6, 60), (192, 191, 8, 60), (192, 192, 8, 60), (161, 484, 2, 60),
])
def test_both_sides_of_each_line_match_the_oracle(R, S, per_sm, P):
    C = 50
    _check(_views(per_sm, C), R, C, 24, S, P)


@pytest.mark.parametrize('R,S,P', [
    (200, 540, 60), (200, 560, 60), (200, 1100, 60), (200, 1100, 20), (250, 1500, 60),
    (513, 700, 60), (1000, 840, 30), (1000, 880, 30),
])
def test_long_cylinders_match_the_oracle(R, S, P):
    """Staging batches of 16 and 8 pixels, and the lengths at which few of
    either's CTAs fit."""
    _check(5, R, 30, 24, S, P, few_views=3)


@pytest.mark.parametrize('R,S', [(64, 64), (128, 128), (100, 96)])
def test_few_ctas_keep_one_row_per_thread(R, S):
    """A call of few CTAs goes to the kernel of one row per thread, which
    copies aligned cylinders 16 bytes at a time and others slice by slice to
    the same bits.  (The streamed kernel, which would take the aligned ones
    only, sums in another order.)"""
    got, proj, values, pix = _check(9, R, 50, 24, S, 60)
    shifted = torch.empty(values.numel() + 1, device='cuda')[1:].view(values.shape)
    shifted.copy_(values)
    assert torch.equal(got, proj.forward(shifted, pix))


@pytest.mark.parametrize('R,S', [(200, 64), (64, 64), (120, 64)])
def test_nonfinite_voxels_in_the_streamed_kernel(R, S):
    """An infinite or NaN voxel reaches the rows whose centre slice is within
    one of it, and no others (the taps of zero weight included)."""
    N, C = 24, 40
    V = _views(25, C) if R == 64 else _views(7, C)
    _, proj, _ = _setup(V, R, C, N, S)
    idx = torch.arange(N * N, device='cuda')
    for bad in (float('inf'), float('nan')):
        x = torch.ones((N * N, S), device='cuda')
        x[N * (N // 2) + 5, 30] = bad
        got = proj.forward(x, idx)
        band = proj.forward(x[:, :40].contiguous(), idx, slice_start=0)
        band += proj.forward(x[:, 40:].contiguous(), idx, slice_start=40)
        assert torch.equal(torch.isfinite(got), torch.isfinite(band))


@pytest.mark.parametrize('R,S,P,weighted,storage', [
    (112, 112, 30, False, 'float32'), (112, 112, 60, False, 'float32'),    # n = 10 and 20
    (112, 112, 60, True, 'float32'), (112, 112, 60, True, 'float16'),
    (112, 112, 60, False, 'bfloat16'), (112, 484, 30, False, 'float32'),
    (112, 484, 60, True, 'float16'), (170, 168, 60, False, 'float32'),
    (170, 168, 60, False, 'float16'), (170, 169, 60, True, 'float32'),
    (200, 160, 20, False, 'float32'), (200, 160, 30, False, 'float32'),
    (200, 160, 60, True, 'float32'), (200, 200, 60, True, 'float32'),
    (200, 200, 40, True, 'float16'), (200, 1100, 60, False, 'float32'),
    (200, 1000, 60, False, 'float32'), (200, 1000, 60, True, 'float32'),
])
def test_subset_steps_on_both_sides_match_the_oracle(R, S, P, weighted, storage):
    N, V, C = 40, 10, 53
    ang = np.linspace(0, 2 * np.pi, V, endpoint=False)
    far = 12.0 * max(N, S)
    m = mb.ConeBeamModel((V, R, C), ang, source_detector_dist=far, source_iso_dist=far / 2)
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
    rng = np.random.default_rng(R + S + P)
    y = rng.standard_normal((V, R, C)).astype(np.float32)
    w = rng.uniform(0.5, 1.5, (V, R, C)).astype(np.float32) if weighted else None
    x0 = (0.1 * rng.random((N, N, S))).astype(np.float32)
    H = m.compute_hessian_diagonal(weights=w)
    dev = torch.device('cuda', 0)
    upd = m.create_vcd_subset_updater(H, weights=1 if w is None else torch.as_tensor(w, device=dev))
    sub = np.sort(rng.choice(mb.gen_full_indices((N, N, S)), size=P, replace=False)).astype(np.int64)
    flat = torch.as_tensor(x0.reshape(-1, S), device=dev).clone()
    err = torch.as_tensor(y, device=dev).clone()
    flat, err, _, alpha, _ = upd(flat, err, torch.as_tensor(sub, device=dev))
    prob = ovcd.Problem('cone', og, m._view_params_array().astype(np.float64), (N, N, S),
                        source_iso_dist=far / 2)
    ou = ovcd.SubsetUpdater(prob, H.reshape(-1, S), w, 0.5, 0.2,
                            dc_profile=ovcd.dc_damping_profile(prob))
    oflat, oerr = x0.reshape(-1, S).astype(np.float64), y.astype(np.float64)
    _, oalpha, _ = ou(oflat, oerr, sub)
    # 16-bit storage rounds the stored residual: 2^-11 of its size, 2^-8 in bfloat16
    bar = {'float32': max(1e-5, S * 2.0 ** -23), 'float16': 1e-3, 'bfloat16': 8e-3}[storage]
    assert abs(float(alpha) - oalpha) <= 10 * bar * abs(oalpha)
    assert rel_l2(flat.cpu().numpy(), oflat) <= bar
    assert rel_l2(err.cpu().numpy(), oerr) <= bar
