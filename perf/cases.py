"""Timed cases of the package: what a ptychographic reconstruction has it do, through its
public entry points.

Every case is a dict of plain values; ``prepare`` makes the inputs a program has in hand (the
current object and probe, the measured patterns, the scan) from a seed, ``run`` is one call and
``exact`` the same outputs in 64 bits from plain torch. The inputs follow the package's
synthetic workloads: objects of random Gaussian atoms, a defocused aperture probe with
incoherent modes centred in its window, a jittered raster scan, Poisson patterns. The calls are
those in the middle of a reconstruction: the object carries half the specimen's phase and the
probe's defocus is off (20 of 50 A; 40 of 100 A at 64 px). The losses are the amplitude and the
least-squares losses.

The loss and the squared error are sums of float32 terms per detector pixel; the passes hand
them out as float32, as a program logs them.
"""
import ctypes
import math

import numpy as np
import torch

from pypty_gb300 import _lib
from pypty_gb300.autograd import multislice_loss
from pypty_gb300.engine import Geometry, default_engine, make_problem
from pypty_gb300.fft import fft2, ifft2, ifft2_ishift, shift_fft2
from pypty_gb300.optim import fourier_clean_

PI, TWO_PI = 3.141592654, 6.2831855      # the truncated constants of the method's definition
CUTOFF, DISTANCE = 2 / 3, 2.0            # band limit (of Nyquist), slice distance (Angstrom)
MODE_POWERS = (0.45, 0.2, 0.12, 0.08, 0.06, 0.04, 0.03, 0.02)


# ---------------------------------------------------------------------- cases
def _scan(name, call, W, Z, modes, rows, cols, batch, step=4.0, algorithm="lsq_sqrt", distances=False,
          rolloff=0.0, checkpoint=1, variant="", margin=7):
    return dict(name=name, call=call, W=W, Z=Z, modes=modes, rows=rows, cols=cols, batch=batch, step=step,
                algorithm=algorithm, distances=distances, rolloff=rolloff, checkpoint=checkpoint, variant=variant,
                margin=margin)


def listed():
    return [
        # one epoch of a thin specimen: the package's single-slice workload (16 x 16 scan, 64 px)
        _scan("single slice 64", "gradient", 64, 1, 1, 16, 16, 256, step=2.5, margin=26),
        # one mini-batch of an incremental solver: few positions, intensity loss, odd object extents
        _scan("mini-batch 64", "gradient", 64, 4, 2, 5, 7, 35, step=9.0, algorithm="lsq", margin=10),
        # one full iteration of the package's headline multislice workload (512 x 512 x 20, 32 x 32 scan)
        _scan("multislice 128", "gradient", 128, 20, 3, 32, 32, 256, margin=260),
        # a refinement with its own distance per slice, a smooth band limit and a ragged last batch
        _scan("per-slice distances 128", "gradient", 128, 7, 2, 11, 13, 64, algorithm="lsq_sqrt_2", distances=True,
              rolloff=0.1),
        # a large-window, many-slice call that keeps every 8th wave and recomputes the others
        _scan("checkpointed 256", "gradient", 256, 24, 5, 14, 20, 70, checkpoint=8),
        # refinement of one specimen tilt per position (the tilted propagators differ by position)
        _scan("tilts 128", "gradient", 128, 10, 2, 12, 12, 72, variant="tilt"),
        # in-line (near-field) imaging of a thick specimen
        _scan("near field 64", "gradient", 64, 6, 3, 9, 15, 135, variant="near"),
        # a torch program that differentiates the loss: forward and backward as two calls
        _scan("autograd 128", "autograd", 128, 8, 3, 8, 12, 96),
        # the patterns of one training specimen of the learned warm start
        _scan("simulate 128", "simulate", 128, 20, 3, 32, 32, 256, margin=260),
        # the window transforms on their own: plain and centred, forward and back
        dict(name="window FFTs 128", call="fft", W=128, batch=1536),
        # the band limit of a trial object x + step * dx inside a line search
        dict(name="band limit 512x512x20", call="clean", ny=512, nx=512, Z=20),
        # one training step's share of a layer of the warm-start network: output, data and weight gradients
        dict(name="convolution 64-64", call="conv", N=4, Ci=64, Co=64, H=128, Wd=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["64", "64", "128", "128", "256", "tilt", "near", "autograd", "simulate", "fft", "clean", "conv"])
    if kind == "fft":
        W = rng.choice([64, 128, 256])
        return dict(call="fft", W=W, batch=_log(rng, 5, 1536 * 128 * 128 // (W * W)))
    if kind == "clean":
        ny, nx = rng.choice([(256, 256), (256, 512), (512, 512), (1024, 512)])
        return dict(call="clean", ny=ny, nx=nx, Z=_log(rng, 1, 20 * 512 * 512 // (ny * nx)))
    if kind == "conv":
        Ci, Co = 8 * rng.randint(1, 16), 8 * rng.randint(1, 12)
        H, Wd = 32 * rng.randint(1, 4), 32 * rng.randint(1, 4)
        return dict(call="conv", N=rng.randint(1, 4), Ci=Ci, Co=Co, H=H, Wd=Wd)
    W = {"64": 64, "256": 256, "near": rng.choice([64, 128])}.get(kind, 128)
    Z = _log(rng, 1 if W < 256 else 2, {64: 8, 128: 20, 256: 24}[W])
    modes = rng.randint(1, {64: 4, 128: 3, 256: 5}[W])
    if kind in ("tilt", "near", "autograd"):
        Z = max(2, min(Z, 10))
    most = {64: 24, 128: 20, 256: 12}[W]
    rows, cols = _log(rng, 3, most), _log(rng, 3, most)
    step = round(rng.uniform(2.0, 8.0 if W < 256 else 5.0), 2)
    call = kind if kind in ("autograd", "simulate") else "gradient"
    # a distance per slice and a smooth band limit are options of the far-field calls
    plain = kind in ("64", "128")
    batch = max(1, min(rows * cols, _log(rng, 16, 256 if W < 256 else 64)))
    c = _scan("", call, W, Z, modes, rows, cols, batch, step, rng.choice(["lsq_sqrt", "lsq_sqrt", "lsq", "lsq_sqrt_2"]),
              plain and Z > 2 and rng.random() < 0.3, 0.1 if plain and rng.random() < 0.3 else 0.0,
              rng.choice([1, 1, 8]) if W == 256 else 1, kind if kind in ("tilt", "near") else "", rng.randint(0, 60))
    del c["name"]
    return c


# ---------------------------------------------------------------------- inputs
def _optics(c):
    """(wavelength in A, aperture in rad, pixel in A): 200 kV at 64 px, 300 kV above."""
    kv, alpha, px = (200.0, 25e-3, 0.2) if c["W"] == 64 else (300.0, 30e-3, 0.1)
    return 12.398 / math.sqrt((2 * 511.0 + kv) * kv), alpha, px


def _probe(c, defocus, dose=1e5):
    """A defocused aperture probe, its modes orthogonal, centred in the window (W, W, modes)."""
    W, modes, (lam, alpha, px) = c["W"], c["modes"], _optics(c)
    f = np.fft.fftfreq(W, px)
    kx, ky = np.meshgrid(f, f, indexing="xy")
    k2, kmax = kx ** 2 + ky ** 2, alpha / lam
    base = (k2 <= kmax ** 2) * np.exp(-1j * math.pi * lam * defocus * px * k2)
    polys = [1, kx / kmax, ky / kmax, (kx ** 2 - ky ** 2) / kmax ** 2, kx * ky / kmax ** 2]
    found = []
    for p in polys[:modes]:
        m = np.fft.fftshift(np.fft.ifft2(base * p))
        for q in found:
            m = m - np.vdot(q, m) * q
        found.append(m / np.sqrt(np.vdot(m, m).real))
    w = np.array(MODE_POWERS[:modes]) / sum(MODE_POWERS[:modes])
    return np.stack([m * math.sqrt(dose * modes / W ** 2 * a) for m, a in zip(found, w)], axis=-1)


def _specimen(c, ny, nx, rng, dev):
    """Phases (ny, nx, Z) of Gaussian atoms (sigma 0.35 A, one per 4 A^2 of every slice, peaks of 0.4 to
    2 rad)."""
    Z, px = c["Z"], _optics(c)[2]
    n = int(ny * nx * px * px / 4)
    v = np.zeros((Z, ny, nx))
    z = np.repeat(np.arange(Z), n)
    np.add.at(v, (z, rng.integers(0, ny, Z * n), rng.integers(0, nx, Z * n)), rng.uniform(0.4, 2.0, Z * n))
    s = 0.35 / px
    fy = torch.fft.fftfreq(ny, dtype=torch.float64, device=dev)[:, None]
    fx = torch.fft.rfftfreq(nx, dtype=torch.float64, device=dev)[None]
    g = 2 * math.pi * s * s * torch.exp(-2 * math.pi ** 2 * s * s * (fy ** 2 + fx ** 2))
    t = torch.fft.irfft2(torch.fft.rfft2(torch.from_numpy(v).to(dev)) * g, s=(ny, nx))
    return t.permute(1, 2, 0).contiguous()


def _scan_inputs(c, seed, dev="cuda"):
    rng = np.random.default_rng(seed)
    W = c["W"]
    yy, xx = np.meshgrid(np.arange(c["rows"]) * c["step"], np.arange(c["cols"]) * c["step"], indexing="ij")
    pos = np.stack([yy.ravel(), xx.ravel()], 1)
    pos = pos + rng.uniform(-0.3, 0.3, pos.shape) * c["step"]
    pos -= pos.min(axis=0)
    whole = np.round(pos)
    ny, nx = (math.ceil((k - 0.4) * c["step"]) + W + c["margin"] for k in (c["rows"], c["cols"]))
    phase = _specimen(c, ny, nx, rng, dev)
    x = dict(whole=whole.astype(np.int32), corr=(pos - whole).astype(np.float32))
    x["obj"] = torch.polar(torch.ones_like(phase), 0.5 * phase).to(torch.complex64)[..., None].contiguous()
    x["probe"], true_probe = (torch.from_numpy(_probe(c, f)).to(dev).to(torch.complex64) for f in (200.0, 500.0))
    d = DISTANCE * (1 + 0.2 * rng.uniform(-1, 1, max(1, c["Z"] - 1)))
    x["distances"] = d.astype(np.float32) if c["distances"] else np.full(max(1, c["Z"] - 1), DISTANCE, np.float32)
    x["tilts"] = np.zeros((len(pos), 6), np.float32)
    if c["variant"] == "tilt":
        x["tilts"][:, 2:4] = rng.normal(size=(len(pos), 2)) * 2e-3
    truth = torch.polar(torch.ones_like(phase), phase).to(torch.complex64)[..., None]
    gen = torch.Generator(device=dev).manual_seed(seed)
    parts = []
    with torch.no_grad():
        for b in _batches(c, len(pos), 64 if W == 256 else 256):
            parts.append(_patterns(c, x, truth, true_probe, torch.from_numpy(x["corr"]).to(dev), None, b))
        x["measured"] = torch.poisson(torch.cat(parts).float().clamp_min(0), generator=gen)
    return x


def _network_inputs(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    N, Ci, Co, H, Wd = (c[k] for k in ("N", "Ci", "Co", "H", "Wd"))
    return dict(x=r(N, Ci, H, Wd).clamp_min(0).bfloat16(), w=r(Co, Ci, 3, 3) * (2 / (9 * Ci)) ** 0.5, b=0.1 * r(Co),
                dy=(1e-2 * r(N, Co, H, Wd)).bfloat16())


def _complex_inputs(shape, seed, n=1):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.view_as_complex(torch.randn((*shape, 2), generator=gen, device="cuda")) for _ in range(n)]


# ---------------------------------------------------------------------- the calls
_kept = {}


def _gradients(x):
    """The loss and gradient buffers of a program's calls: allocated once for each problem size and
    kept, as the engine with its workspace is."""
    key = (tuple(x["obj"].shape), tuple(x["probe"].shape), len(x["whole"]))
    if key not in _kept:
        _kept[key] = (torch.empty(2, dtype=torch.float64, device="cuda"), torch.empty_like(x["obj"]),
                      torch.empty_like(x["probe"]), torch.empty((key[2], 2), device="cuda"))
    return _kept[key]


def _c_ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    c = case
    if c["call"] == "fft":
        return dict(c=c, x=_complex_inputs((c["batch"], c["W"], c["W"]), seed)[0])
    if c["call"] == "clean":
        noise, dx = _complex_inputs((c["ny"], c["nx"], c["Z"], 1), seed, 2)
        return dict(c=c, x=1 + 0.3 * noise, dx=0.1 * dx, out=torch.empty_like(dx), engine=default_engine())
    if c["call"] == "conv":
        s = dict(_network_inputs(c, seed), c=c)
        n = ctypes.c_int64(0)
        _lib.check(_lib.lib().pty_nn_conv3x3_wgrad_workspace_floats(c["N"], c["Ci"], c["Co"], c["H"], c["Wd"],
                                                                   ctypes.byref(n)), "workspace")
        s.update(ws=torch.empty(n.value, device="cuda"), y=torch.empty_like(s["dy"]), dx=torch.empty_like(s["x"]),
                 dw=torch.empty_like(s["w"]), db=torch.empty_like(s["b"]))
        return s
    x = _scan_inputs(c, seed)
    geo = Geometry.make(x["whole"], x["corr"])
    lam, _, px = _optics(c)
    options = dict(algorithm=c["algorithm"], wavelength=lam, pixel_size_x=px, pixel_size_y=px, slice_distance=DISTANCE,
                   damping_cutoff=CUTOFF, smooth_rolloff=c["rolloff"])
    s = dict(c=c, x=x, geo=geo, options=options, engine=default_engine(), out=_gradients(x))
    s["problem"] = make_problem(c["W"], tuple(x["obj"].shape), c["modes"], geo, compute_batch=c["batch"], step_pos=True,
                                checkpoint_every=c["checkpoint"],
                                slice_distances=x["distances"] if c["distances"] else None, **options)
    if c["call"] == "autograd":
        s["leaves"] = [x["obj"].clone().requires_grad_(True), x["probe"].clone().requires_grad_(True),
                       torch.from_numpy(x["corr"]).cuda().requires_grad_(True)]
    return s


def run(state):
    s, c = state, state["c"]
    if c["call"] == "fft":
        a, b = fft2(s["x"], axes=(1, 2)), shift_fft2(s["x"], axes=(1, 2))
        return a, b, ifft2(a, axes=(1, 2)), ifft2_ishift(b, axes=(1, 2))
    if c["call"] == "clean":
        return fourier_clean_(s["x"], CUTOFF, 0.0, out=s["out"], dx=s["dx"], step=0.3, engine=s["engine"])
    if c["call"] == "conv":
        return _conv(s)
    x, e = s["x"], s["engine"]
    if c["call"] == "simulate":
        return e.simulate(s["problem"], x["obj"], x["probe"], s["geo"])
    if c["call"] == "autograd":
        loss = multislice_loss(*s["leaves"], x["whole"], x["measured"], engine=e, **s["options"])
        return [loss.detach().float(), *torch.autograd.grad(loss, s["leaves"])]
    if c["variant"]:
        kw = dict(recon_type="near_field", defocus=60.0, cs=1e5) if c["variant"] == "near" else \
            dict(tilts=x["tilts"], tilt_mode=0, step_tilts=True)
        r = e.loss_and_direction_variants(s["problem"], x["obj"], x["probe"], s["geo"], x["measured"], **kw)
        return [r[0].float(), *r[1:4]] + ([r[6][:, 2:4]] if c["variant"] == "tilt" else [])
    loss, *grads = e.loss_and_direction(s["problem"], x["obj"], x["probe"], s["geo"], x["measured"], out=s["out"])
    return [loss.float(), *grads]


def _conv(s):
    """A 3x3 layer of the network in training: ReLU(conv(x)), then the gradients of an upstream dy."""
    c, lib = s["c"], _lib.lib()
    N, Ci, Co, H, Wd = (c[k] for k in ("N", "Ci", "Co", "H", "Wd"))
    st = torch.cuda.current_stream().cuda_stream
    p = {k: _c_ptr(v) for k, v in s.items() if isinstance(v, torch.Tensor)}
    _lib.check(lib.pty_nn_conv3x3(p["x"], p["w"], p["b"], p["y"], N, Ci, Co, H, Wd, 1, 0, st), "conv3x3")
    _lib.check(lib.pty_nn_conv3x3_wgrad(p["dy"], p["x"], p["dw"], p["db"], N, Ci, Co, H, Wd, p["ws"], st), "wgrad")
    _lib.check(lib.pty_nn_conv3x3(p["dy"], p["w"], None, p["dx"], N, Co, Ci, H, Wd, 0, 1, st), "data gradient")
    return s["y"], s["dw"], s["db"], s["dx"]


# ---------------------------------------------------------------------- the work
def work(case):
    """Bytes: inputs read once, outputs written once (by each of the four transforms). Flops: 5 n log2 n per transform (the probe
    shift once per position and mode, a transform pair per slice step, mode and direction, the band
    limit of every object and gradient window) and the convolutions' multiply-adds."""
    c = case
    if c["call"] == "fft":
        n = c["W"] ** 2
        return dict(bytes=8 * 8 * c["batch"] * n, flops=4 * c["batch"] * 5 * n * math.log2(n))
    if c["call"] == "clean":
        n = c["ny"] * c["nx"]
        return dict(bytes=24 * n * c["Z"], flops=2 * c["Z"] * 5 * n * math.log2(n))
    if c["call"] == "conv":
        px, w = c["N"] * c["H"] * c["Wd"], 9 * c["Ci"] * c["Co"]
        return dict(bytes=2 * px * 2 * (c["Ci"] + c["Co"]) + 8 * w, flops=3 * 2 * px * w)
    W, Z, M, n = c["W"], c["Z"], c["modes"], c["rows"] * c["cols"]
    ny, nx = (W + c["margin"] + c["step"] * (k - 0.4) for k in (c["rows"], c["cols"]))
    both = 1 if c["call"] == "simulate" else 2
    ffts = both * (2 * Z + 2 * (Z - 1) * M + 2 * M)
    return dict(bytes=both * 8 * (ny * nx * Z + W * W * M) + 4 * n * W * W, flops=n * ffts * 5 * W * W * 2 * math.log2(W))


# ---------------------------------------------------------------------- 64-bit results
def _batches(c, n, size):
    return [np.arange(i, min(n, i + size)) for i in range(0, n, size)]


def _frequencies(c, dev):
    """(qx, qy) in 1/A, the pixel size a float32 number, and the band limit, whose edge is a test of
    float32 frequencies; unshifted (ky, kx) order, float64."""
    W, px = c["W"], np.float32(_optics(c)[2])
    k = np.where(np.arange(W) < W // 2, np.arange(W), np.arange(W) - W)
    f32 = (k * np.float64(np.float32(1) / (np.float32(W) * px))).astype(np.float32)
    q2 = (f32 ** 2)[None, :] + (f32 ** 2)[:, None]
    cut, roll = np.float32(CUTOFF), np.float32(c["rolloff"])
    r1, r0 = (f32.max() * cut) ** 2, (f32.max() * (cut - roll)) ** 2
    mask = (q2 <= r1).astype(np.float64)
    if c["rolloff"]:
        mask *= np.where(q2 > r0, 0.5 * (1 + np.cos(PI * (q2.astype(np.float64) - r0) / (float(r1) - float(r0)))), 1.0)
    f = torch.from_numpy(f32.astype(np.float64)).to(dev)
    return f[None, :].expand(W, W), f[:, None].expand(W, W), torch.from_numpy(mask).to(dev)


def _patterns(c, x, obj, probe, corr, tilts, b):
    """Model patterns (B, W, W) of the positions b in the precision of `obj`, detector order."""
    dev, cplx = obj.device, obj.dtype
    W, Z = c["W"], c["Z"]
    lam = float(np.float32(_optics(c)[0]))
    qx, qy, mask = _frequencies(c, dev)
    r = torch.arange(W, device=dev)
    y = torch.from_numpy(x["whole"][b, 0].astype(np.int64)).to(dev)[:, None] + r
    xx = torch.from_numpy(x["whole"][b, 1].astype(np.int64)).to(dev)[:, None] + r
    m = mask.to(obj.real.dtype)
    ob = obj[y[:, :, None], xx[:, None, :], :, 0].permute(3, 0, 1, 2)          # (Z, B, W, W)
    ob = torch.fft.ifft2(torch.fft.fft2(ob) * m)
    k = torch.from_numpy(np.fft.fftfreq(W) * -TWO_PI).to(dev)
    th = corr[b, 1, None, None].double() * k[None, None, :] + corr[b, 0, None, None].double() * k[None, :, None]
    ramp = (torch.polar(torch.ones_like(th), th * (mask != 0)) * mask if not c["rolloff"]
            else torch.polar(torch.ones_like(th), th * mask) * mask).to(cplx)
    psi = torch.fft.ifft2(torch.fft.fft2(probe.permute(2, 0, 1))[None] * ramp[:, None])
    for z in range(Z):
        psi = psi * ob[z][:, None]
        if z + 1 < Z:
            t = lam * (qx ** 2 + qy ** 2)[None]
            if c["variant"] == "tilt":
                tt = (torch.from_numpy(x["tilts"][:, 2:4]).to(dev) if tilts is None else tilts)[b].double()
                t = t + 2 * (qx * tt[:, 1, None, None] + qy * tt[:, 0, None, None])
            ph = -PI * float(x["distances"][z]) * t
            psi = torch.fft.ifft2(torch.fft.fft2(psi) * (torch.polar(torch.ones_like(ph), ph) * mask).to(cplx)[:, None])
    far = torch.fft.fft2(psi)
    if c["variant"] == "near":
        q2 = qx ** 2 + qy ** 2
        ph = -PI * (lam * q2 * 60.0 + 0.5 * 1e5 * lam ** 3 * q2 ** 2)
        return torch.fft.ifft2(far * (torch.polar(torch.ones_like(ph), ph) * mask).to(cplx)).abs().square().mean(1)
    wave = far * m
    if c["rolloff"]:      # the method's adjoint takes the masked wave, and not the mask a second time
        wave = far + (wave - far).detach()
    return torch.fft.fftshift((wave.real ** 2 + wave.imag ** 2).mean(1), dim=(-2, -1))


def _loss(kind, I, M):
    """(loss, squared error) of patterns I against the measured M."""
    sse = ((I - M) ** 2).sum()
    if kind == "lsq":
        return sse, sse
    if kind == "lsq_sqrt":
        lit = I > 0
        return torch.where(lit, (torch.sqrt(torch.where(lit, I, 1.0)) - M.sqrt()) ** 2, M).sum(), sse
    big = M > 0.5
    return torch.where(big, 0.5 * (I - M) ** 2 / torch.where(big, M, 1.0), I).sum(), sse


def exact(case, seed):
    c = case
    if c["call"] == "fft":
        x = _complex_inputs((c["batch"], c["W"], c["W"]), seed)[0].to(torch.complex128)
        f = torch.fft.fft2(x)
        return f, torch.fft.fftshift(f, dim=(1, 2)), x, x
    if c["call"] == "clean":
        noise, dx = _complex_inputs((c["ny"], c["nx"], c["Z"], 1), seed, 2)
        ky, kx = (torch.fft.fftfreq(n, dtype=torch.float64, device="cuda") for n in (c["ny"], c["nx"]))
        keep = (ky[:, None] ** 2 + kx[None] ** 2 <= (0.5 * float(np.float32(CUTOFF))) ** 2)[..., None, None]
        t = (1 + 0.3 * noise).to(torch.complex128) + 0.3 * (0.1 * dx).to(torch.complex128)
        return torch.fft.ifft2(torch.fft.fft2(t, dim=(0, 1)) * keep, dim=(0, 1))
    if c["call"] == "conv":
        s = {k: v.double() for k, v in _network_inputs(c, seed).items()}
        x, w, b = (s[k].requires_grad_(True) for k in "xwb")
        y = torch.nn.functional.conv2d(x, w, b, padding=1)
        dx, dw, db = torch.autograd.grad(y, (x, w, b), s["dy"])
        return y.detach().relu(), dw, db, dx
    x = _scan_inputs(c, seed)
    dev = x["obj"].device
    obj, probe = (x[k].to(torch.complex128).requires_grad_(True) for k in ("obj", "probe"))
    corr = torch.from_numpy(x["corr"]).to(dev).double().requires_grad_(True)
    tilts = torch.from_numpy(x["tilts"][:, 2:4]).to(dev).double().requires_grad_(True)
    n, W = len(x["whole"]), c["W"]
    size = max(1, min(64, int(2 ** 31 // (W * W * 16 * c["modes"] * (c["Z"] + 1) * 4))))
    if c["call"] == "simulate":
        with torch.no_grad():
            return torch.cat([_patterns(c, x, obj, probe, corr, tilts, b) for b in _batches(c, n, size)])
    leaves = [obj, probe, corr] + ([tilts] if c["variant"] == "tilt" else [])
    total, grads = torch.zeros(2, dtype=torch.float64, device=dev), [torch.zeros_like(v) for v in leaves]
    for b in _batches(c, n, size):
        loss, sse = _loss(c["algorithm"], _patterns(c, x, obj, probe, corr, tilts, b), x["measured"][b].double())
        total += torch.stack([loss, sse]).detach()
        for g, d in zip(grads, torch.autograd.grad(loss, leaves)):
            g += d
    mask = _frequencies(c, dev)[2]
    grads[1] = torch.fft.ifft2(torch.fft.fft2(grads[1], dim=(0, 1)) * mask[..., None], dim=(0, 1))
    if c["call"] == "autograd":
        return [total[0], *grads]
    # the package's gradients of complex arrays are dL/dz*, half of torch's
    return [total, grads[0] / 2, grads[1] / 2, *grads[2:]]
