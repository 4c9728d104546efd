"""The workloads that this package's speed is measured on.

Each case is one call (or one short chain of calls) that a program makes:
the projector pair, the differentiable loss, one VCD iteration of a running
reconstruction, a whole one-call reconstruction, the denoiser.  `exact`
restates the projections and the VCD iteration in 64-bit torch, on its own.

Scans are ellipsoid phantoms with Poisson counts.  Their line integrals are
chords of rays through the ellipsoids, so that a case's data do not depend
on the code that is measured.
"""

import math

import numpy as np
import torch

import mbirtorch_b200 as mb
from mbirtorch_b200.vcd_engine import ResidentSinogram, storage_code

I0 = 1e4           # photons per detector cell
SIGMA_Y, SIGMA_X = 1.0, 0.05
_STORAGE = {"float32": 0, "bfloat16": 1, "float16": 2}


def _case(name, op, geom, views, rows, channels, size, slices, **more):
    case = {"op": op, "geom": geom, "views": views, "rows": rows, "channels": channels,
            "size": size, "slices": slices}
    if geom == "cone":
        case.update(mag=2.0, pitch=2.0, dist=2.0, curved=False, turns=1, row_offset=0.0)
    if geom != "image":
        case.update(channel_offset=0.0)
    case.update(more)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # The largest scan of the benchmark: a curved-detector cone scan of a
        # 512^2 x 256 volume.  Its three hot calls: projecting a volume
        # (initial error, refreshes, simulation), back projecting a scan (FDK,
        # Hessian), and one iteration of 128 subsets, the unit that a
        # reconstruction spends nearly all its time in.
        _case("forward cone 512", "forward", "cone", 720, 320, 768, 512, 256, curved=True),
        _case("back cone 512", "back", "cone", 720, 320, 768, 512, 256, curved=True),
        _case("iteration cone 512", "iteration", "cone", 720, 320, 768, 512, 256, curved=True,
              storage="float32", weighted=False, positivity=False, subsets=128),
        # The same for parallel beam (a synchrotron scan), the iteration
        # weighted, as transmission data are in earnest.
        _case("forward parallel 512", "forward", "parallel", 720, 256, 768, 512, 256),
        _case("back parallel 512", "back", "parallel", 720, 256, 768, 512, 256),
        _case("iteration parallel 512", "iteration", "parallel", 720, 256, 768, 512, 256,
              storage="float32", weighted=True, positivity=False, subsets=128),
        # A helical scan as the reconstruction server holds it: 16-bit storage,
        # weights, positivity (the subset projected twice), a short detector.
        _case("iteration helical 256 f16", "iteration", "cone", 360, 64, 384, 256, 64, turns=2,
              storage="float16", weighted=True, positivity=True, subsets=64),
        # Differentiable projectors in a training loop: loss and gradient of
        # a batch of four volumes.
        _case("loss cone 128 x4", "loss", "cone", 256, 128, 192, 128, 128, mag=1.5, pitch=1.5,
              dist=6.0, batch=4),
        _case("loss parallel 128 x4", "loss", "parallel", 256, 128, 192, 128, 128, batch=4),
        # A small reconstruction in one call, host array in and out: launches
        # and host work count.
        _case("recon parallel 128", "recon", "parallel", 180, 16, 192, 128, 16, iterations=10),
        # A few hundred cylinders projected and back projected, at odd sizes:
        # the smallest calls, where latency counts.
        _case("sparse cone 67", "sparse", "cone", 45, 19, 101, 67, 17, mag=1.7, pitch=1.0,
              dist=2.5, channel_offset=1.3, row_offset=-0.7, pixels=211),
        # The plug-and-play denoiser on a volume.
        _case("denoise 128", "denoise", "image", 1, 1, 1, 128, 96, iterations=5),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["forward", "forward", "back", "back", "iteration", "iteration", "loss",
                     "recon", "sparse", "denoise"])
    most = listed()[2]
    while True:
        size, slices = _between(rng, 24, 512), _between(rng, 8, 256)
        views = _between(rng, 30, 720)
        work = size * size * slices * views
        limit = most["size"] ** 2 * most["slices"] * most["views"]
        if op == "loss":
            limit /= 32
        if op in ("recon", "sparse"):
            limit /= 512
        if work <= limit:
            break
    if op == "denoise":
        return _case("", op, "image", 1, 1, 1, min(size, 200), slices,
                     iterations=rng.randint(2, 6))
    channels = int(1.5 * size) + rng.randint(0, 9)
    geom = rng.choice(["cone", "parallel"])
    if geom == "parallel":
        case = _case("", op, geom, views, slices, channels, size, slices,
                     channel_offset=rng.choice([0.0, round(rng.uniform(-2, 2), 2)]))
    else:
        mag = round(rng.uniform(1.3, 2.5), 2)
        case = _case("", op, geom, views, max(8, int(slices * rng.uniform(0.8, 1.3))), channels,
                     size, slices, mag=mag, pitch=rng.choice([mag, 1.0]),
                     dist=round(rng.uniform(2.0, 6.0), 2), curved=rng.random() < 0.4,
                     turns=rng.choice([1, 1, 2]),
                     channel_offset=rng.choice([0.0, round(rng.uniform(-2, 2), 2)]),
                     row_offset=rng.choice([0.0, round(rng.uniform(-2, 2), 2)]))
    if op == "iteration":
        case.update(storage=rng.choice(["float32", "float32", "float16", "bfloat16"]),
                    weighted=rng.random() < 0.5, positivity=rng.random() < 0.3,
                    subsets=rng.choice([16, 64, 128]))
    elif op == "loss":
        case.update(batch=rng.randint(1, 4))
    elif op == "recon":
        case.update(iterations=rng.randint(3, 8))
    elif op == "sparse":
        case.update(pixels=rng.randint(50, 900))
    return case


# ── what a program has in hand ─────────────────────────────────────────────
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _voxel(case):
    return case["pitch"] / case["mag"] if case["geom"] == "cone" else 1.0


def _view_params(case):
    """(V, 2) angle and z shift of each view, as the model keeps them."""
    V = case["views"]
    if case["geom"] == "parallel":
        ang, z = np.linspace(0, np.pi, V, endpoint=False), np.zeros(V)
    else:
        ang = np.linspace(0, 2 * np.pi * case["turns"], V, endpoint=False)
        span = case["slices"] * _voxel(case) / 4
        z = np.linspace(-span, span, V) if case["turns"] > 1 else np.zeros(V)
    return np.stack([ang, z], axis=1).astype(np.float32)


def _distances(case):
    """(source to detector, source to axis)."""
    sid = case["dist"] * case["size"] * _voxel(case)
    return case["mag"] * sid, sid


def _model(case):
    vp, N, S = _view_params(case), case["size"], case["slices"]
    shape = (case["views"], case["rows"], case["channels"])
    if case["geom"] == "parallel":
        m = mb.ParallelBeamModel(shape, vp[:, 0])
        m.set_params(no_warning=True, verbose=0, det_channel_offset=case["channel_offset"],
                     recon_shape=(N, N, S))
    else:
        sdd, sid = _distances(case)
        m = mb.ConeBeamModel(shape, vp[:, 0], source_detector_dist=sdd, source_iso_dist=sid,
                             helical_z_shifts=vp[:, 1], use_curved_detector=case["curved"])
        m.set_params(no_warning=True, verbose=0, delta_det_channel=case["pitch"],
                     delta_det_row=case["pitch"], det_channel_offset=case["channel_offset"],
                     det_row_offset=case["row_offset"])
        m.auto_set_recon_geometry(no_warning=True)
        m.set_params(no_warning=True, recon_shape=(N, N, S), recon_slice_offset=0.0)
    m.set_params(no_warning=True, sigma_y=SIGMA_Y, sigma_x=SIGMA_X,
                 positivity_flag=bool(case.get("positivity", False)))
    return m


def _ellipsoids(seed, count=8):
    """(centre, semi-axes, in-plane angle, density) on [-1, 1]^3."""
    r = np.random.RandomState(seed)
    return [(r.uniform(-0.4, 0.4, 3), r.uniform(0.1, 0.5, 3), r.uniform(0, np.pi),
             r.uniform(0.1, 1.0)) for _ in range(count)]


def _volume(shape, seed):
    """The phantom on a voxel grid."""
    dev = _device()
    axes = [torch.linspace(-1, 1, max(n, 2), device=dev)[:n] for n in shape]
    Y, X = torch.meshgrid(axes[0], axes[1], indexing="ij")
    vol = torch.zeros(shape, device=dev)
    for c, a, ang, dens in _ellipsoids(seed):
        ca, sa = math.cos(ang), math.sin(ang)
        xr, yr = ca * (X - c[0]) + sa * (Y - c[1]), -sa * (X - c[0]) + ca * (Y - c[1])
        r2 = ((xr / a[0]) ** 2 + (yr / a[1]) ** 2)[:, :, None] + ((axes[2] - c[2]) / a[2]) ** 2
        vol += dens * (r2 <= 1).float()
    return vol


def _scan(case, seed):
    """(V, R, C) noisy line integrals of the phantom, and the counts' share
    of I0, the usual weights of such data."""
    dev, vp = _device(), _view_params(case)
    V, R, C, N, S = (case[k] for k in ("views", "rows", "channels", "size", "slices"))
    dv, pitch = _voxel(case), case.get("pitch", 1.0)
    half = [0.5 * N * dv, 0.5 * N * dv, 0.5 * S * dv]
    u = (torch.arange(C, device=dev) - (C - 1) / 2) * pitch - case["channel_offset"]
    w = (torch.arange(R, device=dev) - (R - 1) / 2) * pitch - case.get("row_offset", 0.0)
    y = torch.empty((V, R, C), device=dev)
    for v0 in range(0, V, 60):
        ang = torch.as_tensor(vp[v0:v0 + 60], device=dev)
        cos, sin = torch.cos(ang[:, :1]), torch.sin(ang[:, :1])   # (v, 1)
        z0 = ang[:, 1].view(-1, 1, 1)
        if case["geom"] == "parallel":   # rays along -y', at x' = u and z = w
            sx, sy = cos * u + sin * 0, -sin * u
            dx, dy = -sin.expand_as(sx), -cos.expand_as(sx)
            sz, dz = w.view(1, R, 1), torch.zeros((1, R, 1), device=dev)
        else:                            # from the source at y' = sid to the cell
            sdd, sid = _distances(case)
            fx, fy = ((sdd * torch.sin(u / sdd), -sdd * torch.cos(u / sdd)) if case["curved"]
                      else (u, torch.full_like(u, -sdd)))
            sx, sy = (sin * sid).expand(-1, C), (cos * sid).expand(-1, C)
            dx, dy = cos * fx + sin * fy, -sin * fx + cos * fy
            sz, dz = z0, w.view(1, R, 1)
        total = torch.zeros((sx.shape[0], R, C), device=dev)
        for c, a, tilt, dens in _ellipsoids(seed):
            ca, sa = math.cos(tilt), math.sin(tilt)
            ax = [a[k] * half[k] for k in range(3)]
            ox, oy = sx - c[0] * half[0], sy - c[1] * half[1]
            px, py = (ca * ox + sa * oy) / ax[0], (-sa * ox + ca * oy) / ax[1]
            qx, qy = (ca * dx + sa * dy) / ax[0], (-sa * dx + ca * dy) / ax[1]
            pz, qz = (sz - c[2] * half[2]) / ax[2], dz / ax[2]
            A = (qx * qx + qy * qy)[:, None] + qz * qz
            B = (px * qx + py * qy)[:, None] + pz * qz
            D = B * B - A * ((px * px + py * py)[:, None] + pz * pz - 1)
            total += 2 * dens * torch.sqrt(D.clamp_min(0)) / A
        length = torch.sqrt((dx * dx + dy * dy)[:, None] + dz * dz)
        y[v0:v0 + 60] = total * length
    mu = 3.0 / max(float(y.max()), 1e-6)
    gen = torch.Generator(device=dev).manual_seed(seed)
    counts = torch.poisson(I0 * torch.exp(-mu * y), generator=gen).clamp_min(1.0)
    return (-torch.log(counts / I0) / mu).contiguous(), (counts / I0).contiguous()


def _residual(case, seed):
    """An error sinogram in mid-reconstruction: what is left of the scan,
    and its noise."""
    gen = torch.Generator(device=_device()).manual_seed(seed + 1)
    y, _ = _scan(case, seed)
    y.mul_(0.1)
    return y.add_(torch.randn(y.shape, generator=gen, device=y.device), alpha=0.5)


def _field(shape, seed):
    """A batch of smoothed normal fields."""
    gen = torch.Generator(device=_device()).manual_seed(seed)
    x = torch.randn((shape[0], 1) + tuple(shape[1:]), generator=gen, device=_device())
    return torch.nn.functional.avg_pool3d(x, 3, stride=1, padding=1)[:, 0].contiguous()


def _sparse_inputs(case, seed):
    """Pixel indices, their cylinders, and a sinogram."""
    dev, N = _device(), case["size"]
    inside = _ror(N)
    r = np.random.RandomState(seed)
    idx = np.sort(r.choice(inside, size=min(case["pixels"], inside.size), replace=False))
    idx = torch.as_tensor(idx, device=dev)
    vals = _volume((N, N, case["slices"]), seed).reshape(N * N, -1)[idx].contiguous()
    gen = torch.Generator(device=dev).manual_seed(seed)
    vals += 0.1 * torch.randn(vals.shape, generator=gen, device=dev)
    sino = torch.rand((case["views"], case["rows"], case["channels"]), generator=gen, device=dev)
    return idx, vals, sino


def _loss_inputs(case, seed):
    shape = (case["batch"], case["size"], case["size"], case["slices"])
    gen = torch.Generator(device=_device()).manual_seed(seed + 1)
    x = _field(shape, seed)
    y = torch.randn((case["batch"], case["views"], case["rows"], case["channels"]),
                    generator=gen, device=_device()) * math.sqrt(case["size"])
    w = 0.5 + torch.rand(y.shape, generator=gen, device=_device())
    return x, y, w


def _iteration_inputs(case, seed):
    """Volume, error sinogram, weights (or None) and the pixel partition."""
    N, S = case["size"], case["slices"]
    x = 0.9 * _volume((N, N, S), seed)
    e = _residual(case, seed)
    w = _scan(case, seed)[1] if case["weighted"] else None
    inside = np.random.RandomState(seed).permutation(_ror(N))
    per = inside.size // min(case["subsets"], inside.size)
    part = np.sort(inside[:per * (inside.size // per)].reshape(-1, per), axis=1)
    return x, e, w, part[:case["subsets"]]


def prepare(case, seed):
    op, N, S = case["op"], case["size"], case["slices"]
    if op == "denoise":
        gen = torch.Generator(device=_device()).manual_seed(seed)
        x = _volume((N, N, S), seed)
        x += 0.1 * torch.randn(x.shape, generator=gen, device=x.device)
        d = mb.QGGMRFDenoiser((N, N, S))
        d.set_params(no_warning=True, verbose=0)
        return {"op": op, "model": d, "x": x, "iterations": case["iterations"], "seed": seed}
    if op == "recon":
        y, w = _scan(case, seed)
        return {"op": op, "case": case, "y": y.cpu().numpy(), "seed": seed,
                "angles": _view_params(case)[:, 0], "model": _model(case)}
    m = _model(case)
    state = {"op": op, "model": m}
    if op == "forward":
        state["x"] = _volume((N, N, S), seed)
    elif op == "back":
        state["y"] = _scan(case, seed)[0]
    elif op == "sparse":
        state["idx"], state["vals"], state["y"] = _sparse_inputs(case, seed)
    elif op == "loss":
        x, state["y"], state["w"] = _loss_inputs(case, seed)
        state["x"] = x.requires_grad_(True)
    elif op == "iteration":
        m.set_storage_precision(case["storage"])
        x, e, w, part = _iteration_inputs(case, seed)
        H = m.compute_hessian_diagonal(weights=w, output_sharded=True)
        state["updater"] = m.create_vcd_subset_updater(H, weights=1 if w is None else w)
        state["flat"] = x.reshape(N * N, S).contiguous()
        state["err"] = ResidentSinogram.from_vrc(e, storage_code(case["storage"]))
        state["partition"] = torch.as_tensor(part, dtype=torch.int64, device=e.device)
        state["seed"] = seed % (1 << 31)
    if op in ("forward", "back", "sparse", "loss"):
        m.full_indices_device()   # the model keeps its index list
    return state


def run(state):
    op, m = state["op"], state["model"]
    if op == "forward":
        return m.forward_project(state["x"], output_sharded=True)
    if op == "back":
        return m.back_project(state["y"], output_sharded=True)
    if op == "sparse":
        return [m.sparse_forward_project(state["vals"], state["idx"]),
                m.sparse_back_project(state["y"], state["idx"])]
    if op == "loss":
        state["x"].grad = None
        loss = mb.weighted_residual_loss(m, state["x"], state["y"], state["w"])
        loss.backward()
        return [loss.detach(), state["x"].grad]
    np.random.seed(state["seed"] % (1 << 31))
    if op == "iteration":
        flat, err, ell1, alpha, sumsq = m.vcd_partition_iterator(
            state["updater"], state["flat"], state["err"], state["partition"])
        return [flat, err.data, ell1, alpha, sumsq]
    if op == "denoise":
        out, info = m.denoise(state["x"], sigma_noise=0.1, max_iterations=state["iterations"],
                              stop_threshold_change_pct=0, logfile_path=None, print_logs=False,
                              output_sharded=True)
        return out
    case = state["case"]
    kw = dict(max_iterations=case["iterations"], stop_threshold_change_pct=0, logfile_path=None,
              print_logs=False)
    out, info = m.recon(state["y"], **kw)
    return [out, np.asarray(info["recon_params"]["fm_rmse"])]


# ── what a pass cannot do without ──────────────────────────────────────────
def work(case):
    op, N, S = case["op"], case["size"], case["slices"]
    if op == "denoise":
        # per sweep: image and residual read and written; about 15 operations
        # for each of the six neighbours
        n = N * N * S
        return {"bytes": 16 * n * case["iterations"], "flops": 90 * n * case["iterations"]}
    V, sino = case["views"], case["views"] * case["rows"] * case["channels"]
    P = int(_ror(N).size) if op != "sparse" else case["pixels"]
    # multiply-adds per (voxel, view): two channel taps, and two row taps for cone
    per = (8 if case["geom"] == "cone" else 4) * V * S
    one = {"bytes": 4 * (sino + P * S), "flops": per * P}
    if op in ("forward", "back"):
        return one
    if op == "sparse":
        return {k: 2 * v for k, v in one.items()}
    if op == "loss":   # the residual and its gradient; x, y, w in, the gradient out
        return {"bytes": case["batch"] * 4 * (2 * sino + 2 * P * S),
                "flops": case["batch"] * 2 * one["flops"]}
    width = 4 if case.get("storage", "float32") == "float32" else 2
    arrays = 3 if case.get("weighted") else 2    # e in and out, weights in
    reach = min(1.0, 1.1 * N / case["channels"])  # channels that the volume covers
    if op == "recon":
        sweeps, steps = case["iterations"], 4 + 16 + 64 + 128 * max(0, case["iterations"] - 3)
    else:
        sweeps, steps = 1, case["subsets"]
    return {"bytes": int(steps * arrays * width * sino * reach) + 16 * P * S * sweeps,
            "flops": sweeps * 2 * one["flops"]}


def tolerance(case):
    op = case["op"]
    if op in ("forward", "back", "sparse"):
        # 32-bit sums and 32-bit geometry: 1e-7 to 3e-6 off `exact`
        return {"rel": 1e-5, "max": 4e-4}
    if op == "loss":
        return {"rel": 2e-5, "max": 8e-4}   # both in a row: 3e-6 to 5e-6 off
    if op == "denoise":
        return {"rel": 1e-5, "max": 1e-3}
    if case.get("storage", "float32") != "float32":
        return {"rel": 1e-2, "max": 0.5}    # the stored residual's own rounding
    # each step's size is a ratio of sums over all that came before it
    return {"rel": 1e-4, "max": 1e-2}


# ── the same in 64 bits ────────────────────────────────────────────────────
def _ror(N):
    """Indices of the pixels inside the inscribed circle of an N x N grid."""
    t = ((np.arange(N) - (N - 1) / 2) / max((N - 1) / 2, 1e-9)) ** 2
    return np.flatnonzero((t[:, None] + t[None, :] <= 1.0).reshape(-1))


class _Exact:
    """The projector pair in float64: footprints of rectangles on detector
    cells, separable over channels and rows."""

    def __init__(self, case):
        self.case, self.dev = case, _device()
        self.vp = torch.as_tensor(_view_params(case), device=self.dev).double()
        self.V, self.R, self.C, self.S = (case[k] for k in ("views", "rows", "channels",
                                                            "slices"))
        self.cone = case["geom"] == "cone"
        self.dv, self.pitch = _voxel(case), case.get("pitch", 1.0)

    def _chunks(self, P):
        n = max(1, int(2.5e7 // (P * max(self.R, self.S))))
        return [(v, min(self.V, v + n)) for v in range(0, self.V, n)]

    def _footprints(self, v0, v1, idx):
        """Channel centre and width (in cells), weight scale, and for cone the
        rows' magnification of each (view, pixel)."""
        N = self.case["size"]
        ang = self.vp[v0:v1, :1]
        x = ((idx % N).double() - (N - 1) / 2) * self.dv
        y = (torch.div(idx, N, rounding_mode="floor").double() - (N - 1) / 2) * self.dv
        c, s = torch.cos(ang), torch.sin(ang)
        xr, yr = c * x - s * y, s * x + c * y
        mag = torch.ones_like(xr)
        if not self.cone:
            u, theta = xr, torch.zeros_like(xr)
        else:
            sdd, sid = _distances(self.case)
            mag = 1 / (1 / self.case["mag"] - yr / sdd)
            if self.case["curved"]:
                theta = torch.atan2(xr, sid - yr)
                u = sdd * theta
            else:
                u = mag * xr
                theta = torch.atan2(u, torch.full_like(u, sdd))
        side = torch.maximum(torch.cos(ang - theta).abs(), torch.sin(ang - theta).abs()) * self.dv
        width = mag * side / self.pitch
        if self.cone and not self.case["curved"]:
            width = width / torch.cos(theta)
        n = (u + self.case["channel_offset"]) / self.pitch + (self.C - 1) / 2
        return n, width, self.dv * self.dv / side, mag

    @staticmethod
    def _overlap(centre, width, cell):
        """Length of [centre -+ width / 2] inside cell -+ 1/2."""
        a = (width + 1) / 2 - (centre - cell).abs()
        return torch.minimum(a.clamp_min(0), width.clamp_max(1))

    def _rows(self, v0, v1, mag):
        """Row of slice 0, rows per slice, and t(k) = t0 + t1 k, the tangent of
        the ray's slope."""
        z0 = -self.vp[v0:v1, 1:] - self.dv * (self.S - 1) / 2
        sdd, _ = _distances(self.case)
        step = mag * self.dv / self.pitch
        m0 = (mag * z0 + self.case["row_offset"]) / self.pitch + (self.R - 1) / 2
        return m0, step, mag * z0 / sdd, mag * self.dv / sdd

    def forward(self, values, idx):
        """(P, S) -> (V, C, R)."""
        P, R, C, S = idx.numel(), self.R, self.C, self.S
        out = torch.zeros((self.V, C, R), dtype=torch.float64, device=self.dev)
        rows = torch.arange(R, device=self.dev, dtype=torch.float64)
        pad = torch.zeros((P, S + 2), dtype=torch.float64, device=self.dev)
        pad[:, 1:-1] = values
        for v0, v1 in self._chunks(P):
            n, width, scale, mag = self._footprints(v0, v1, idx)
            if self.cone:
                m0, step, t0, t1 = (t[:, :, None] for t in self._rows(v0, v1, mag))
                k0 = torch.round((rows - m0) / step)
                det = torch.zeros((v1 - v0, P, R), dtype=torch.float64, device=self.dev)
                for o in (-1, 0, 1):
                    k = k0 + o
                    a = self._overlap(m0 + step * k, step, rows) * torch.sqrt(1 + (t0 + t1 * k) ** 2)
                    at = k.clamp(-1, S).long() + 1
                    det += a * torch.gather(pad[None].expand(v1 - v0, P, S + 2), 2, at)
            else:
                det = values[None].expand(v1 - v0, P, S)
            c0 = torch.round(n)
            base = torch.arange(v0, v1, device=self.dev)[:, None] * C
            for o in (-1, 0, 1):
                c = c0 + o
                on = (c >= 0) & (c < C)
                w = torch.where(on, self._overlap(n, width, c) * scale, 0.0)
                at = (base + c.clamp(0, C - 1).long()).reshape(-1)
                out.view(-1, R).index_add_(0, at, (w[:, :, None] * det).reshape(-1, R))
        return out

    def back(self, sino, idx, power=1):
        """(V, C, R) -> (P, S)."""
        P, R, C, S = idx.numel(), self.R, self.C, self.S
        out = torch.zeros((P, S), dtype=torch.float64, device=self.dev)
        k = torch.arange(S, device=self.dev, dtype=torch.float64)
        for v0, v1 in self._chunks(P):
            n, width, scale, mag = self._footprints(v0, v1, idx)
            c0 = torch.round(n)
            base = torch.arange(v0, v1, device=self.dev)[:, None] * C
            col = torch.zeros((v1 - v0, P, R), dtype=torch.float64, device=self.dev)
            flat = sino.reshape(-1, R)
            for o in (-1, 0, 1):
                c = c0 + o
                on = (c >= 0) & (c < C)
                w = torch.where(on, self._overlap(n, width, c) * scale, 0.0) ** power
                at = base + c.clamp(0, C - 1).long()
                col += w[:, :, None] * flat[at]
            if not self.cone:
                out += col.sum(0)
                continue
            m0, step, t0, t1 = (t[:, :, None] for t in self._rows(v0, v1, mag))
            m = m0 + step * k
            mc = torch.round(m)
            got = torch.zeros((v1 - v0, P, S), dtype=torch.float64, device=self.dev)
            for o in (-1, 0, 1):
                r = mc + o
                a = torch.where((r >= 0) & (r < R), self._overlap(m, step, r), 0.0) ** power
                got += a * torch.gather(col, 2, r.clamp(0, R - 1).long())
            out += (got * torch.sqrt(1 + (t0 + t1 * k) ** 2) ** power).sum(0)
        return out


def _prior(flat, N, idx, S):
    """Gradient and curvature of the qGGMRF surrogate (p = 2, q = 1.2, T = 1,
    equal neighbour weights; edges reflect) at the cylinders idx."""
    def influence(d):
        a = (d.abs().clamp_min(SIGMA_X * float(np.finfo(np.float32).eps)) / SIGMA_X) ** (1.2 - 2)
        return a * (0.6 + a) / (2 * SIGMA_X ** 2 * (1 + a) ** 2)

    x = flat[idx]
    row, col = torch.div(idx, N, rounding_mode="floor"), idx % N
    near = [flat[(row + i).clamp(0, N - 1) * N + (col + j).clamp(0, N - 1)]
            for i, j in ((1, 0), (-1, 0), (0, 1), (0, -1))]
    near += [torch.cat([x[:, 1:], x[:, -1:]], 1), torch.cat([x[:, :1], x[:, :-1]], 1)]
    g, h = torch.zeros_like(x), torch.zeros_like(x)
    for other in near:
        d = x - other
        b = influence(d) * (2 / 6)
        g, h = g + b * d, h + b
    return g, h


def _damping(case):
    """Per-slice damping of the subset's mean direction (cone beam)."""
    a, b, p, c = 0.25, 100.0, 0.7, 0.5
    dv, S = _voxel(case), case["slices"]
    z = (np.arange(S) - (S - 1) / 2) * dv
    zs = _view_params(case)[:, 1].astype(np.float64)
    if np.ptp(zs) == 0:
        zs = zs[:1]
    t = case["size"] * np.abs(z[:, None] - zs[None, :]) / _distances(case)[1]
    return ((c * t ** p + a * b ** p) / (t ** p + b ** p)).mean(axis=1)


def _exact_iteration(case, seed):
    A = _Exact(case)
    dev, N, S = A.dev, case["size"], case["slices"]
    x, e, w, part = _iteration_inputs(case, seed)
    flat = x.reshape(N * N, S).double()
    e = e.double().transpose(1, 2).contiguous()
    w = torch.ones_like(e) if w is None else w.double().transpose(1, 2).contiguous()
    every = torch.as_tensor(_ror(N), device=dev)
    H = torch.zeros_like(flat)
    H[every] = A.back(w, every, power=2)
    s = torch.as_tensor(_damping(case), device=dev) if A.cone else None
    ell1 = alphas = 0.0
    sumsq = torch.zeros(S, dtype=torch.float64, device=dev)
    np.random.seed(seed % (1 << 31))
    fm = 1 / SIGMA_Y ** 2
    for k in np.random.permutation(part.shape[0]):
        idx = torch.as_tensor(part[int(k)], device=dev)
        gp, hp = _prior(flat, N, idx, S)
        g = gp - fm * A.back(w * e, idx)
        inv = 1 / (hp + fm * H[idx])
        if s is not None:
            g = g - (1 - s) * ((inv * g).sum(0) / inv.sum(0))
        step = -g * inv
        Ad = A.forward(step, idx)
        alpha = ((fm * (w * e * Ad).sum() - (gp * step).sum())
                 / (fm * (w * Ad * Ad).sum() + (hp * step * step).sum())).clamp(1e-7, 1.5)
        if case["positivity"]:
            step = torch.maximum(-flat[idx] / alpha, step)
            Ad = A.forward(step, idx)
        flat[idx] += alpha * step
        e -= alpha * Ad
        ell1 = ell1 + (alpha * step).abs().sum()
        sumsq += ((alpha * step) ** 2).sum(0)
        alphas = alphas + alpha
    stored = e if case["storage"] == "float32" else None   # 16 bits: in units of its own
    return [flat, stored, ell1, alphas / part.shape[0], sumsq]


def exact(case, seed):
    op, N, S = case["op"], case["size"], case["slices"]
    if op in ("recon", "denoise"):
        # Host-side statistics, hundreds of steps on partitions drawn inside
        # the call: the iteration cases stand for their arithmetic.
        return None
    cost = N * N * max(S, case["rows"]) * case["views"]
    if cost > (1.5e10 if op == "iteration" else 8e10):
        return None   # over about 20 seconds
    if op == "iteration":
        return _exact_iteration(case, seed)
    A = _Exact(case)
    every = torch.as_tensor(_ror(N), device=A.dev)
    if op == "forward":
        x = _volume((N, N, S), seed).reshape(N * N, S)[every].double()
        return A.forward(x, every).transpose(1, 2)
    if op == "back":
        vol = torch.zeros((N * N, S), dtype=torch.float64, device=A.dev)
        vol[every] = A.back(_scan(case, seed)[0].double().transpose(1, 2).contiguous(), every)
        return vol.reshape(N, N, S)
    if op == "sparse":
        idx, vals, y = _sparse_inputs(case, seed)
        return [A.forward(vals.double(), idx).transpose(1, 2),
                A.back(y.double().transpose(1, 2).contiguous(), idx)]
    x, y, w = _loss_inputs(case, seed)
    loss, grad = 0.0, torch.zeros(x.shape, dtype=torch.float64, device=A.dev)
    for b in range(case["batch"]):
        r = A.forward(x[b].reshape(N * N, S)[every].double(), every) - y[b].double().transpose(1, 2)
        wr = w[b].double().transpose(1, 2) * r
        loss = loss + (wr * r).sum()
        grad[b].view(N * N, S)[every] = A.back((2 * wr).contiguous(), every)
    return [loss, grad]
