"""The streamed cone forward of a subset step where a CTA owns two channel
blocks (many views and channels): an odd number of blocks, a partial last
channel block, weights and 16-bit storage against the FP64 oracle; a block
that no pixel reaches beside one that is reached; and how many products the
line search sums in FP32 before it goes on in FP64."""

import numpy as np
import pytest
import torch

import mbirtorch_b200 as mb
import oracle
from conftest import rel_l2
from oracle import OracleGeometry
from oracle import vcd as ovcd

pytestmark = pytest.mark.gpu

R, C = 196, 491        # 31 channel blocks, the last of 11 channels


def _views():
    """Enough views that pairs of channel blocks fill the device (48 CTAs an SM)."""
    blocks = (C + 15) // 16
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return -(-2 * 48 * sms // blocks) + 1


def _model(N, S, storage='float32', sigma_y=0.5, R=R):
    V = _views()
    ang = np.linspace(0, 2 * np.pi, V, endpoint=False)
    m = mb.ConeBeamModel((V, R, C), ang, source_detector_dist=8.0 * N, source_iso_dist=4.0 * N)
    m.set_params(no_warning=True, verbose=0, delta_det_channel=2.0, delta_det_row=2.0)
    m.auto_set_recon_geometry(no_warning=True)
    m.set_params(no_warning=True, recon_shape=(N, N, S), sigma_y=sigma_y, sigma_x=0.2)
    m.set_storage_precision(storage)
    return m


def _oracle(m, N, S):
    g = m._geometry()
    R = g.num_det_rows
    og = OracleGeometry(num_det_rows=R, num_det_channels=C, num_recon_rows=N, num_recon_cols=N,
                        num_slices=S, delta_det_channel=2.0, delta_det_row=2.0,
                        delta_voxel=g.delta_voxel, delta_voxel_row=g.delta_voxel_row,
                        delta_voxel_slice=g.delta_voxel_slice, magnification=g.magnification,
                        recon_slice_offset=g.recon_slice_offset,
                        source_detector_dist=g.source_detector_dist, psf_radius=g.psf_radius,
                        bp_psf_radius=g.bp_psf_radius)
    return ovcd.Problem('cone', og, m._view_params_array().astype(np.float64), (N, N, S),
                        source_iso_dist=4.0 * N)


def _step(m, H, w, x0, err, idx):
    """One subset step on copies: (flat, err, alpha)."""
    upd = m.create_vcd_subset_updater(H, weights=1 if w is None else w)
    flat, e, _, alpha, _ = upd(x0.clone(), err.clone(), idx)
    return flat, e, float(alpha)


@pytest.mark.parametrize('R,S,weighted,storage', [
    (196, 8, False, 'float32'), (196, 200, True, 'float32'), (196, 8, True, 'float16'),
    (196, 8, False, 'bfloat16'),
    # cylinders copied slice by slice, and detectors that the streamed kernel
    # takes with two blocks a CTA only
    (140, 9, False, 'float32'), (170, 9, True, 'float32'), (170, 9, True, 'float16'),
    (176, 8, False, 'float32'),
])
def test_step_matches_oracle(R, S, weighted, storage):
    N = 470 if S < 100 else 120    # 470: the shadow reaches past both ends of the detector
    m = _model(N, S, storage, R=R)
    V = m.get_params('sinogram_shape')[0]
    gen = torch.Generator(device='cuda').manual_seed(11)
    err = torch.randn((V, R, C), generator=gen, device='cuda')
    w = torch.rand((V, R, C), generator=gen, device='cuda') + 0.5 if weighted else None
    x0 = 0.1 * torch.rand((N * N, S), generator=gen, device='cuda')
    rng = np.random.default_rng(5)
    inside = mb.gen_full_indices((N, N, S)).astype(np.int64)
    idx = np.sort(rng.choice(inside, size=250, replace=False))
    # the Hessian at the subset's pixels, and ones elsewhere (not read)
    H = torch.ones((N * N, S), device='cuda')
    ones = torch.ones_like(err) if w is None else w
    H[torch.as_tensor(idx, device='cuda')] = m.sparse_back_project(
        ones, torch.as_tensor(idx, device='cuda'), coeff_power=2)
    flat, e, alpha = _step(m, H.reshape(N, N, S), w, x0, err, torch.as_tensor(idx, device='cuda'))
    prob = _oracle(m, N, S)
    ou = ovcd.SubsetUpdater(prob, H.cpu().numpy(), None if w is None else w.cpu().numpy(), 0.5, 0.2,
                            dc_profile=ovcd.dc_damping_profile(prob))
    oflat, oerr = x0.double().cpu().numpy(), err.double().cpu().numpy()
    _, oalpha, _ = ou(oflat, oerr, idx)
    # 16-bit storage rounds the stored residual: 2^-11 of its size, 2^-8 in bfloat16
    bar = {'float32': 1e-5, 'float16': 1e-3, 'bfloat16': 8e-3}[storage]
    assert abs(alpha - oalpha) <= 10 * bar * abs(oalpha)
    assert rel_l2(flat.cpu().numpy(), oflat) <= bar
    assert rel_l2(e.cpu().numpy(), oerr) <= bar


@pytest.mark.parametrize('bad', [float('nan'), float('inf')])
def test_cells_of_a_block_that_no_pixel_reaches_are_not_counted(bad):
    """A detector edge of dead cells, beyond the volume's shadow: its channel
    block is no part of the step even where the CTA's other block is."""
    N, S = 60, 8       # shadow: channels 212 to 278 (blocks 13 to 17) at any angle
    m = _model(N, S)
    V = m.get_params('sinogram_shape')[0]
    gen = torch.Generator(device='cuda').manual_seed(12)
    err = torch.randn((V, R, C), generator=gen, device='cuda')
    x0 = 0.1 * torch.rand((N * N, S), generator=gen, device='cuda')
    idx = torch.as_tensor(mb.gen_full_indices((N, N, S)).astype(np.int64)[::7].copy(),
                          device='cuda')
    H = m.compute_hessian_diagonal(output_sharded=True)
    flat, e, alpha = _step(m, H, None, x0, err, idx)
    broken = err.clone()
    broken[:, :, :208] = bad       # blocks 0 to 12: block 12 shares its CTA with block 13
    broken[:, :, 288:] = bad       # blocks 18 on: the group of blocks 18 and 19 is all dead
    flat2, e2, alpha2 = _step(m, H, None, x0, broken, idx)
    assert alpha2 == alpha and torch.equal(flat2, flat)
    assert torch.equal(e2[:, :, 208:288], e[:, :, 208:288])


def test_line_search_sums_at_most_one_block_in_single_precision():
    """Products so large that a row's sum over one block of 16 channels fits
    FP32 and over a CTA's two does not, from eight pixels (one batch of the
    walk) that lie four channels apart."""
    N, S = 60, 4
    m = _model(N, S, sigma_y=1.0)
    m.set_params(no_warning=True, max_alpha=10.0)    # the step's alpha is about 4
    V = m.get_params('sinogram_shape')[0]
    prob = _oracle(m, N, S)
    rows, cols = np.arange(N) * N + N // 2, (N // 2) * N + np.arange(N)
    one = ovcd.Problem('cone', prob.geom, prob.view_params[:1], (N, N, S), source_iso_dist=4.0 * N)

    def centre(p):
        a = one.forward(np.ones((1, S)), np.array([p], dtype=np.int64))[0].sum(axis=0)
        return float(np.sum(a * np.arange(C)) / np.sum(a))

    line = max((rows, cols), key=lambda ps: abs(centre(ps[0]) - centre(ps[-1])))
    where = np.array([centre(p) for p in line])
    idx = np.sort([int(line[np.argmin(np.abs(where - ch))]) for ch in range(226, 256, 4)])
    assert len(set(idx)) == 8
    idx = np.asarray(idx, dtype=np.int64)
    # one view carries weight; e = 1000 there, so that products exceed gradients
    err = np.zeros((V, R, C), dtype=np.float32)
    err[0] = 1000.0
    w1 = np.zeros((1, R, C))
    w1[0] = 1.0
    H1 = np.ones((N * N, S))
    H1[idx] = one.back(w1, idx, coeff_power=2)
    probe = ovcd.SubsetUpdater(one, 1e30 * H1, 1e30 * w1, 1.0, 0.2, max_alpha=10.0,
                               dc_profile=ovcd.dc_damping_profile(prob))
    e1 = np.asarray(err[:1], dtype=np.float64)
    _, oalpha, _ = probe(np.zeros((N * N, S)), e1, idx)
    Ad = (np.asarray(err[:1], np.float64) - e1)[0] / oalpha       # (R, C)
    assert 1 < oalpha < 9
    assert np.abs(Ad[:, :224]).max() == 0 and np.abs(Ad[:, 256:]).max() == 0
    lin, quad = 1000.0 * Ad, Ad * Ad
    both = [np.abs(t[:, 224:256].sum(axis=1)).max() for t in (lin, quad)]
    each = [np.abs(t[:, a:a + 16].sum(axis=1)).max() for t in (lin, quad) for a in (224, 240)]
    top = float(np.finfo(np.float32).max)
    W = 1.4 * top / max(both)
    assert W * max(each) <= 0.8 * top
    w = torch.zeros((V, R, C), device='cuda')
    w[0] = W
    _, _, alpha = _step(m, torch.as_tensor(W * H1, dtype=torch.float32, device='cuda')
                        .reshape(N, N, S), w, torch.zeros((N * N, S), device='cuda'),
                        torch.as_tensor(err, device='cuda'), torch.as_tensor(idx, device='cuda'))
    assert abs(alpha - oalpha) <= 1e-4 * oalpha
