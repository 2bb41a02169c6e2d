"""The work a user of this framework has it do, as measurable cases.

One imaging problem is set up once and evaluated many times: an optimiser
calls objective + gradient (or the objective alone, in its line search)
hundreds of times.  Around that stand the dirty image and PSF, the learned
start, and the visibility weighting and gridding on the way in.  Sizes follow
the configurations in gpuvmem_gb300/synth.py, from the smallest test problem
to a quarter of the visibilities of the 2048 x 2048, 8-channel one.

exact() restates each result in 64 bits with numpy and torch alone.
"""

from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

import gpuvmem_gb300 as gv
from gpuvmem_gb300 import synth, unet, warmstart

RPDEG = math.pi / 180.0
LIGHT = np.float32(2.99792458e8)

ENTROPY, TSV, ETA, MINPIX = 0.01, 1e-4, -1.0, 0.001


def listed():
    return [
        # the smallest problem of the tests: launches and latency decide
        dict(name="evaluate-64", kind="evaluate", n=64, nchan=1, n_ant=8, n_times=40, mfs=False),
        # plain MEM 256^2 (104,400 visibilities), one optimiser evaluation
        dict(name="evaluate-256", kind="evaluate", n=256, nchan=1, n_ant=30, n_times=240,
             mfs=False),
        # plain MEM 2048^2 x 8 channels, a quarter of its integrations
        dict(name="evaluate-2048-8ch", kind="evaluate", n=2048, nchan=8, n_ant=50, n_times=900,
             mfs=False),
        # two-image fit: both planes' evaluations, uneven flagging per channel
        dict(name="mfs-1024-8ch", kind="evaluate", n=1024, nchan=8, n_ant=30, n_times=97,
             mfs=True),
        # the objective alone, as a host-side line search calls it
        dict(name="objective-1024-4ch", kind="objective", n=1024, nchan=4, n_ant=40, n_times=720,
             mfs=False),
        # candidate starts scored by the solver's objective, one synchronisation
        # (a whole solve is not compared: its steps hang on the last bits of f)
        dict(name="score-256", kind="score", n=256, nchan=1, n_ant=30, n_times=240, mfs=False,
             count=12),
        # independent small problems of uneven size in one launch
        dict(name="batch-16", kind="batch", count=16, lo=20000, hi=500000),
        # the warm start's inputs: dirty image and PSF of one sky
        dict(name="dirty-psf-256", kind="dirty", n=256, nchan=1, n_ant=30, n_times=240,
             mfs=False),
        # the shipped network on one sky
        dict(name="unet-forward-256", kind="unet", height=256, base=16, levels=5, batch=1,
             train=False),
        # one training step of the same network
        dict(name="unet-train-256", kind="unet", height=256, base=16, levels=5, batch=8,
             train=True),
        # robust weighting of ragged channels, host arrays in and out
        dict(name="briggs-1024-16ch", kind="weights", n=1024, nchan=16, n_ant=40, n_times=120,
             scheme="briggs"),
        # convolutional gridding with the 7 x 7 spheroidal kernel, host arrays in and out
        dict(name="grid-pswf-512-4ch", kind="grid", n=512, nchan=4, n_ant=30, n_times=160,
             kernel="PSWF"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "evaluate", "objective", "score", "batch", "dirty",
                       "unet", "weights", "grid"])
    if kind in ("evaluate", "objective", "score", "dirty"):
        n = rng.choice([64, 128, 256, 512, 1024, 2048])
        mfs = kind == "evaluate" and rng.random() < 0.3
        nchan = rng.randint(2 if mfs else 1, 9)
        n_ant = rng.randint(7, 50)
        nbl = n_ant * (n_ant - 1) // 2
        vis = _log(rng, 1000, 400000)
        d = dict(kind=kind, n=n, nchan=nchan, n_ant=n_ant, n_times=max(3, vis // nbl), mfs=mfs)
        if kind == "score":
            d["count"] = rng.randint(2, 12)
        return d
    if kind == "batch":
        lo = _log(rng, 5000, 50000)
        return dict(kind=kind, count=rng.randint(3, 16), lo=lo, hi=lo * rng.randint(2, 8))
    if kind == "unet":
        train = rng.random() < 0.5
        return dict(kind=kind, height=rng.choice([64, 128, 256]), base=rng.choice([8, 16]),
                    levels=rng.randint(3, 5), batch=rng.randint(1, 8 if train else 3), train=train)
    n_ant = rng.randint(10, 45)
    nbl = n_ant * (n_ant - 1) // 2
    d = dict(kind=kind, n=rng.choice([256, 512, 1024]), nchan=rng.randint(1, 12), n_ant=n_ant,
             n_times=max(3, _log(rng, 5000, 90000) // nbl))
    if kind == "weights":
        d["scheme"] = rng.choice(["uniform", "briggs"])
    else:
        d["kernel"] = rng.choice(["PillBox2D", "Gaussian2D", "PSWF"])
    return d


# ---- inputs -------------------------------------------------------------------

def _config(case, seed):
    """The array, sky and sampling of a case: the antenna disk and cell size
    of the 256, 1024 and 2048 pixel configurations, scaled for the sizes in
    between, flagged visibilities and uneven weights as real data have."""
    n, nchan = case["n"], case["nchan"]
    if n >= 2048:
        cell, disk, fwhm, hours = 0.01, 2000.0, 25.0, 4.0
        freqs = list(np.linspace(225e9, 235e9, nchan))
    elif n >= 1024:
        cell, disk, fwhm, hours = 0.05, 1000.0, 40.0, 2.0
        freqs = list(np.linspace(85e9, 115e9, nchan))
    elif n >= 256:
        cell, disk, fwhm, hours = 12.8 / n, 500.0 * n / 256, 25.0, 4.0
        freqs = list(np.linspace(228e9, 232e9, nchan))
    else:
        cell, disk, fwhm, hours = 0.05, 150.0 * n / 64, 0.45 * n * 0.05, 4.0
        freqs = list(np.linspace(229e9, 231e9, nchan))
    if nchan == 1:
        freqs = [230e9]
    return synth.SynthConfig(
        name="case", n=n, cell_arcsec=cell, n_ant=case["n_ant"], disk_radius_m=disk,
        freqs_hz=freqs, dec_deg=-30.0, ha_start_h=-hours / 2, ha_stop_h=hours / 2,
        dt_s=hours * 3600.0 / case["n_times"], n_sources=20, pb_fwhm_arcsec=fwhm, seed=seed,
        source_radius_frac=0.2, flag_fraction_range=(0.0, 0.4) if case.get("mfs") else (0.0, 0.0),
        alpha_range=(-1.0, 3.0) if case.get("mfs") else None,
        # gridded data have one visibility per occupied cell: one array for all seeds
        array_seed=1 if case.get("kind") == "grid" else None)


def _data(case, seed):
    data = synth.generate(_config(case, seed), device="cuda")
    rng = np.random.default_rng([seed, 77])
    w = data.weight * rng.uniform(0.5, 1.5, data.weight.size).astype(np.float32)
    if case.get("kind") != "grid":
        w[rng.random(w.size) < 0.02] = 0.0
    return dataclasses.replace(data, weight=w)


def _terms(case):
    t = [gv.term("Chi2", 1.0), gv.term("Entropy", ENTROPY, prior_value=MINPIX, eta=ETA)]
    if not case.get("mfs"):
        t.append(gv.term("TotalSquaredVariation", TSV))
    return t


def _sky_image(n, seed, peak, mfs):
    """A partly converged image: the positivity floor, a few extended
    components and faint structure, in units of fg_scale."""
    g = torch.Generator().manual_seed(seed * 7 + 1)
    ax = torch.arange(n, dtype=torch.float64)
    img = torch.zeros(2, n, n, dtype=torch.float64)
    for _ in range(8):
        r = torch.rand(4, generator=g, dtype=torch.float64)
        cx, cy = n * (0.3 + 0.4 * r[0]), n * (0.3 + 0.4 * r[1])
        s = n * (0.01 + 0.03 * r[2])
        img[0] += peak * (0.05 + r[3]) * torch.outer(torch.exp(-0.5 * ((ax - cy) / s) ** 2),
                                                     torch.exp(-0.5 * ((ax - cx) / s) ** 2))
    img[0] += 0.01 * peak * torch.rand(n, n, generator=g, dtype=torch.float64) ** 4 + MINPIX
    if mfs:
        img[1] = torch.rand(n, n, generator=g, dtype=torch.float64) * 2 - 0.5
    return img.float()


def _image(case, data, seed):
    # flux of the components spread over the beam, in units of fg_scale
    return _sky_image(case["n"], seed, 200.0, case.get("mfs", False))


def _candidates(case, data, seed):
    """One image about the positivity floor at several scales, as the learned
    start's policy tries them."""
    img = _image(case, data, seed)
    k = torch.linspace(0.5, 1.5, case["count"])[:, None, None, None]
    return (MINPIX + k * (img[None] - MINPIX)) * torch.tensor([1.0, 0.0])[None, :, None, None]


def _batch_parts(case, seed):
    rng = np.random.default_rng([seed, 5])
    parts = []
    for k in range(case["count"]):
        n = int([128, 256, 512][k % 3])
        n_ant = int(rng.integers(10, 41))
        vis = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
        parts.append(dict(n=n, nchan=1, n_ant=n_ant, mfs=False,
                          n_times=max(4, int(vis / (n_ant * (n_ant - 1) // 2)))))
    return parts


def _unet_inputs(case, seed):
    g = torch.Generator().manual_seed(seed)
    H, B = case["height"], case["batch"]
    ax = torch.arange(H, dtype=torch.float32) - H / 2
    r2 = ax[:, None] ** 2 + ax[None, :] ** 2
    psf = torch.exp(-r2 / 18.0) * torch.cos(torch.sqrt(r2) / 3.0)
    x, t = torch.zeros(B, 2, H, H), torch.zeros(B, 1, H, H)
    F = torch.fft.rfft2(torch.fft.ifftshift(psf))
    for b in range(B):
        sky = torch.zeros(H, H)
        for _ in range(12):
            r = torch.rand(4, generator=g)
            cy, cx, s = H * (r[0] * 0.6 - 0.3), H * (r[1] * 0.6 - 0.3), 1.0 + 4.0 * r[2]
            sky += (0.1 + r[3]) * torch.exp(-((ax[:, None] - cy) ** 2 + (ax[None, :] - cx) ** 2)
                                            / (2 * s * s))
        d = torch.fft.irfft2(torch.fft.rfft2(sky) * F, s=(H, H))
        d += 0.02 * d.abs().max() * torch.randn(H, H, generator=g)
        x[b, 0], x[b, 1], t[b, 0] = d / d.abs().max(), psf, sky / sky.max()
    return x, t


LR = 1e-3


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("evaluate", "objective", "score", "dirty"):
        data = _data(case, seed)
        prob = gv.Problem(data, _terms(case))
        st = dict(case=case, prob=prob)
        if kind == "score":
            prob.set_iteration(1)
            st["imgs"] = _candidates(case, data, seed).cuda()
        elif kind != "dirty":
            prob.set_iteration(1)
            st["img"] = _image(case, data, seed).cuda()
            st["xi"] = [torch.zeros_like(st["img"]) for _ in range(2 if case["mfs"] else 1)]
        return st
    if kind == "batch":
        probs, imgs = [], []
        for k, p in enumerate(_batch_parts(case, seed)):
            data = _data(p, 100 * seed + k)
            prob = gv.Problem(data, _terms(p))
            prob.set_iteration(1)
            probs.append(prob)
            imgs.append(_image(p, data, 100 * seed + k).cuda())
        return dict(case=case, batch=gv.Batch(probs), imgs=imgs,
                    xis=[torch.zeros_like(i) for i in imgs])
    if kind == "unet":
        x, t = _unet_inputs(case, seed)
        if case["train"] or (case["height"], case["base"], case["levels"]) != (256, 16, 5):
            net = unet.UNet(case["height"], in_channels=2, base_channels=case["base"],
                            levels=case["levels"], max_batch=case["batch"], seed=seed)
        else:
            net, _ = warmstart.load_network(warmstart.NETWORK_PATH, max_batch=case["batch"])
        return dict(case=case, net=net, x=x.cuda(), t=t.cuda())
    data = _data(case, seed)
    st = dict(case=case, data=data)
    if kind == "grid":
        st["table"], st["support"], _ = gv.ckernel_build(case["kernel"], data.M, data.N,
                                                         data.DELTAX, data.DELTAY)
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "evaluate":
        prob, img, out = state["prob"], state["img"], []
        for flag, xi in enumerate(state["xi"]):
            f, fi, _ = prob.evaluate(img, 1, flag_opt=flag, xi=xi)
            out.append({"f": f, "terms": fi, "gradient": xi})
        return out
    if kind == "objective":
        f, fi = state["prob"].objective(state["img"])
        return {"f": f, "terms": fi, "image": state["img"]}
    if kind == "score":
        return state["prob"].objective_many(state["imgs"])
    if kind == "dirty":
        return {"dirty": state["prob"].dirty_image(), "psf": state["prob"].psf_image()}
    if kind == "batch":
        f = state["batch"].evaluate(state["imgs"], state["xis"], 1)
        return {"f": f, "gradients": state["xis"]}
    if kind == "unet":
        net = state["net"]
        if not case["train"]:
            return net.forward(state["x"])
        loss = net.train_step(state["x"], state["t"], LR)
        return {"loss": loss, "grads": net.grads(), "params": net.params()}
    d = state["data"]
    if kind == "weights":
        return gv.apply_weighting(case["scheme"], 0.0, d.M, d.N, d.DELTAX, d.DELTAY, d.freqs,
                                  d.chan_off, d.uvw_m, d.weight)
    off, uvw, vo, w = gv.grid_visibilities(state["table"], state["support"], d.M, d.N, d.DELTAX,
                                           d.DELTAY, d.freqs, d.chan_off, d.uvw_m, d.vo, d.weight)
    return {"off": off, "uvw": uvw, "vo": vo, "weight": w}


# ---- necessary work -------------------------------------------------------------

def _nvis(case):
    v = case["nchan"] * case["n_times"] * (case["n_ant"] * (case["n_ant"] - 1) // 2)
    return v * 0.8 if case.get("mfs") else v * 1.0


def _conv_flops(case):
    c = [case["base"] << l for l in range(case["levels"])]
    px, L, f = case["height"] ** 2, case["levels"], 0
    for l in range(L):
        f += (px >> 2 * l) * 18 * ((2 if l == 0 else c[l - 1]) * c[l] + c[l] * c[l])
    for l in range(L - 1):
        f += (px >> 2 * l) * 18 * ((c[l + 1] + c[l]) * c[l] + c[l] * c[l])
    return case["batch"] * (f + 2.0 * px * c[0])


def work(case):
    """Inputs once, outputs once.  A visibility is (u, v, w) as three floats,
    its complex value and its weight (24 bytes); the transforms between image
    and visibilities need an FFT per channel and direction and a local
    interpolation (16 multiply-adds) per visibility."""
    kind = case["kind"]
    if kind == "batch":
        vis = sum(_nvis(p) for p in _batch_parts(case, 0))
        px = sum(p["n"] ** 2 for p in _batch_parts(case, 0))
        fft = sum(10.0 * p["n"] ** 2 * math.log2(p["n"]) for p in _batch_parts(case, 0))
        return dict(bytes=24.0 * vis + 16.0 * px, flops=2 * fft + 64.0 * vis)
    if kind == "unet":
        f = _conv_flops(case)
        px = case["batch"] * case["height"] ** 2
        return dict(bytes=12.0 * px, flops=3 * f if case["train"] else f)
    vis, px = _nvis(case), float(case["n"] ** 2)
    fft = 10.0 * px * math.log2(case["n"]) * case["nchan"]
    if kind == "evaluate":
        k = 2 if case["mfs"] else 1
        return dict(bytes=k * (24.0 * vis + 16.0 * px), flops=k * (2 * fft + 64.0 * vis))
    if kind == "objective":
        return dict(bytes=24.0 * vis + 8.0 * px, flops=fft + 32.0 * vis)
    if kind == "score":
        k = case["count"]
        return dict(bytes=24.0 * vis + k * 8.0 * px, flops=k * (fft + 32.0 * vis))
    if kind == "dirty":
        return dict(bytes=2 * (24.0 * vis + 4.0 * px), flops=2 * (fft + 32.0 * vis))
    if kind == "weights":
        return dict(bytes=28.0 * vis + 4.0 * vis, flops=10.0 * vis)
    taps = 1 if case["kernel"] == "PillBox2D" else 49
    return dict(bytes=36.0 * vis + 36.0 * min(vis, px * case["nchan"]), flops=16.0 * vis * taps)


# ---- 64-bit restatements -----------------------------------------------------------

def _lam(freq):
    return float(LIGHT / np.float32(freq))


def _atten32(n, data, freq):
    """The primary beam in single precision (it decides the mask)."""
    f = np.float32
    x = ((np.arange(n) - int(data.xobs)) * data.DELTAX * RPDEG).astype(f)
    y = ((np.arange(n) - int(data.yobs)) * data.DELTAY * RPDEG).astype(f)
    arc = np.sqrt(x[None, :] * x[None, :] + y[:, None] * y[:, None])
    fwhm = f(data.pb_factor) * f(LIGHT / f(freq)) / f(data.antenna_diameter)
    r = arc / fwhm
    a = np.exp(-(f(4.0) * f(np.log(f(2.0)))) * r * r)
    return np.where(arc <= f(data.pb_cutoff), a, f(0.0))


class _Setup:
    """Wavelengths, flips, noise image, mask and scale of a problem."""

    def __init__(self, data):
        f = np.float32
        n, self.data, self.n = data.N, data, data.N
        C = len(data.freqs)
        sw, mom = f(0.0), np.zeros(3)
        for c in range(C):
            o, e = data.chan_off[c], data.chan_off[c + 1]
            if e == o:
                continue
            u, v = (data.uvw_m[o:e, k] / _lam(data.freqs[c]) for k in (0, 1))
            w = data.weight[o:e].astype(np.float64)
            mom += [np.sum(u * u * w), np.sum(v * v * w), np.sum(u * v * w)]
            sw = f(sw + np.cumsum(data.weight[o:e], dtype=f)[-1])  # summed in order, 32 bits
        uu, vv, uv = mom / float(sw)
        sq = math.sqrt((uu - vv) ** 2 + 4.0 * uv * uv)
        bmaj = 1.0 / math.sqrt(2.0) / math.pi / math.sqrt(uu + vv - sq) / RPDEG
        bmin = 1.0 / math.sqrt(2.0) / math.pi / math.sqrt(uu + vv + sq) / RPDEG
        vis_noise = f(0.5) * np.sqrt(f(1.0) / sw)
        area = math.pi * (bmaj / abs(data.DELTAX)) * (bmin / abs(data.DELTAX))
        jypix = f(float(vis_noise) / (area / float(f(4.0) * f(np.log(f(2.0))))))
        a = _atten32(n, data, data.nu_0)
        w = a * a
        with np.errstate(divide="ignore"):
            noise = np.sqrt(f(1.0) / ((w / w.max()) / (jypix * jypix)))
        self.fg = float(noise.min())
        cut = f(10.0) * noise.min()
        self.inside = torch.from_numpy(noise < cut).cuda()
        self.outside = torch.from_numpy(noise > cut).cuda()

    def channel(self, c):
        """u, v, w (wavelengths, u flipped to be non-positive), Vo, weight."""
        d = self.data
        o, e = d.chan_off[c], d.chan_off[c + 1]
        uvw = torch.from_numpy(d.uvw_m[o:e]).cuda()
        vo = torch.complex(*(torch.from_numpy(d.vo[o:e, k].astype(np.float64)).cuda()
                             for k in (0, 1)))
        wt = torch.from_numpy(d.weight[o:e].astype(np.float64)).cuda()
        flip = uvw[:, 0] > 0
        s = torch.where(flip, -1.0, 1.0).double()
        lam = _lam(d.freqs[c])
        vo = torch.where(flip, vo.conj(), vo)
        return uvw[:, 0] * s / lam, uvw[:, 1] * s / lam, uvw[:, 2] / lam, vo, wt

    def beam(self, freq):
        d, n = self.data, self.n
        x = (torch.arange(n, device="cuda").double() - int(d.xobs)) * d.DELTAX * RPDEG
        y = (torch.arange(n, device="cuda").double() - int(d.yobs)) * d.DELTAY * RPDEG
        r2 = x[None, :] ** 2 + y[:, None] ** 2
        fwhm = d.pb_factor * _lam(freq) / d.antenna_diameter
        a = torch.exp(-4.0 * math.log(2.0) * r2 / fwhm ** 2)
        return torch.where(torch.from_numpy(_atten32(n, d, freq) > 0).cuda(), a, 0.0)

    def clip(self, img, flag):
        i0, al = img[0].double(), img[1].double()
        i0 = torch.where(self.outside, float(np.float32(MINPIX)), i0)
        al = torch.where(self.outside, 0.0, al)
        if flag > 0:
            al = torch.where(~self.outside & (i0 < 0.0), 0.0, al)
        return i0, al

    def model(self, i0, al, c):
        """The grid's cells as complex128, interpolated at the visibilities;
        (Vo - Vm, weights with those off the grid set to 0)."""
        d, n = self.data, self.n
        u, v, w, vo, wt = self.channel(c)
        nud = float(np.float32(d.freqs[c]) / np.float32(d.nu_0))
        inu = torch.clamp(i0 * nud ** al, min=float(np.float32(MINPIX)))
        grid = torch.fft.ifft2((inu * self.beam(d.freqs[c]) * self.fg).to(torch.complex128),
                               norm="forward")
        k = torch.arange(n, device="cuda").double()
        k = torch.where(k < n // 2, k, k - n)
        ru, rv = d.xobs / n * k, d.yobs / n * k
        grid = grid * torch.exp(-2j * math.pi * (ru[None, :] + rv[:, None]))
        ux = u * (n * (RPDEG * d.DELTAX))
        uy = v * (n * (RPDEG * d.DELTAY))
        ux = torch.where(ux < 0, ux + n, ux)
        uy = torch.where(uy < 0, uy + n, uy)
        i1, j1 = torch.floor(ux).long(), torch.floor(uy).long()
        ok = (i1 >= 0) & (i1 < n) & (j1 >= 0) & (j1 < n)
        fu, fv = ux - i1, uy - j1
        i1, j1 = i1.clamp(0, n - 1), j1.clamp(0, n - 1)
        i2, j2 = (i1 + 1) % n, (j1 + 1) % n
        vm = ((1 - fu) * (1 - fv) * grid[j1, i1] + (1 - fu) * fv * grid[j2, i1]
              + fu * (1 - fv) * grid[j1, i2] + fu * fv * grid[j2, i2])
        return u, v, w, vo - torch.where(ok, vm, 0.0), torch.where(ok, wt, 0.0)

    def adjoint(self, u, v, w, val):
        """sum_k Re(conj(val_k) e^{2 pi i (x u + y v + (z - 1) w)}) per pixel."""
        d, n = self.data, self.n
        x = (torch.arange(n, device="cuda").double() - int(d.xobs)) * d.DELTAX * RPDEG
        y = (torch.arange(n, device="cuda").double() - int(d.yobs)) * d.DELTAY * RPDEG
        r2 = x[None, :] ** 2 + y[:, None] ** 2
        z = torch.sqrt(1.0 - r2)
        rho = -r2 * r2 / (2.0 * (1.0 + z) ** 2)  # (z - 1) + r^2 / 2, first order below
        g0 = torch.zeros(n, n, dtype=torch.complex128, device="cuda")
        g1 = torch.zeros_like(g0)
        step = max(1024, (1 << 25) // n)
        for k in range(0, u.numel(), step):
            uu, vv, ww, cc = (t[k:k + step] for t in (u, v, w, val))
            def ph(a, t):
                q = a[:, None] * t[None, :] - 0.5 * a[:, None] ** 2 * ww[None, :]
                q = 2 * math.pi * (q - torch.round(q))
                return torch.complex(torch.cos(q), torch.sin(q))
            A, B = ph(y, vv) * cc.conj()[None, :], ph(x, uu).T
            g0 += A @ B
            g1 += (A * ww[None, :]) @ B
        return (g0 + 2j * math.pi * rho * g1).real

    def priors(self, i0, terms_n):
        g, m = float(np.float32(MINPIX)), self.inside
        lam_e, lam_t = float(np.float32(ENTROPY)), float(np.float32(TSV))
        lg = torch.log(i0 / g)
        vals = [torch.where(m, i0 * lg, 0.0).sum().item()]
        grad = lam_e * (lg + 1.0)
        if terms_n > 2:
            t = i0.clone()
            t[:-1, :-1] = (i0[:-1, :-1] - i0[:-1, 1:]) ** 2 + (i0[:-1, :-1] - i0[1:, :-1]) ** 2
            vals.append(torch.where(m, t, 0.0).sum().item())
            t = i0.clone()
            t[1:-1, 1:-1] = 8 * i0[1:-1, 1:-1] - 2 * (i0[:-2, 1:-1] + i0[1:-1, :-2]
                                                     + i0[2:, 1:-1] + i0[1:-1, 2:])
            grad = grad + lam_t * t
        return vals, torch.where(m, grad, 0.0)

    def evaluate(self, img, flag, terms_n, gradient):
        d, n = self.data, self.n
        i0, al = self.clip(img.cuda(), flag)
        chi2, plane = 0.0, torch.zeros(n, n, dtype=torch.float64, device="cuda")
        for c in range(len(d.freqs)):
            u, v, w, vr, wt = self.model(i0, al, c)
            chi2 += 0.5 * (wt * (vr.real ** 2 + vr.imag ** 2)).sum().item()
            if gradient:
                s = -self.adjoint(u, v, w, wt * vr) * self.fg * self.beam(d.freqs[c])
                nud = float(np.float32(d.freqs[c]) / np.float32(d.nu_0))
                s = s * nud ** al
                if flag % 2:
                    s = torch.where(i0 > 0.0, s * i0 * self.fg * math.log(nud), 0.0)
                plane += torch.where(self.inside, s, 0.0)
        vals, pg = self.priors(i0, terms_n)
        lams = [float(np.float32(ENTROPY)), float(np.float32(TSV))]
        f = chi2 + sum(a * b for a, b in zip(lams, vals))
        xi = torch.zeros(2, n, n, dtype=torch.float64, device="cuda")
        xi[flag % 2] = plane
        if flag % 2 == 0:
            xi[0] += pg
        return f, [chi2] + vals, xi, torch.stack([i0, al])


def _exact_unet(case, seed):
    st = prepare(case, seed)
    th = st["net"].params().double().requires_grad_(case["train"])
    x, t, L = st["x"].double(), st["t"].double(), case["levels"]
    C, at = [case["base"] << l for l in range(L)], 0

    def conv(h, co, k, relu):
        nonlocal at
        ci = h.shape[1]
        w = th[at:at + co * ci * k * k].reshape(co, ci, k, k)
        b = th[at + co * ci * k * k:at + co * ci * k * k + co]
        at += co * ci * k * k + co
        # a sum over taps: plain matrix products
        p = torch.nn.functional.pad(h, (k // 2,) * 4)
        H = h.shape[-1]
        y = b[None, :, None, None] + sum(
            torch.einsum("bchw,oc->bohw", p[:, :, i:i + H, j:j + H], w[:, :, i, j])
            for i in range(k) for j in range(k))
        return torch.relu(y) if relu else y

    h, skips = x, []
    for l in range(L):
        if l:
            h = torch.nn.functional.avg_pool2d(h, 2)
        h = conv(conv(h, C[l], 3, True), C[l], 3, True)
        skips.append(h)
    for l in range(L - 2, -1, -1):
        up = h.repeat_interleave(2, 2).repeat_interleave(2, 3)
        h = conv(conv(torch.cat([up, skips[l]], 1), C[l], 3, True), C[l], 3, True)
    y = conv(h, 1, 1, False)
    if not case["train"]:
        return y
    loss = ((y - t) ** 2).mean()
    (g,) = torch.autograd.grad(loss, th)
    return {"loss": loss.item(), "grads": g, "params": None}


def _exact_weights(case, data):
    n, out, cells = data.N, [], []
    du = 1.0 / (data.M * (RPDEG * data.DELTAX))
    dv = 1.0 / (data.N * (RPDEG * data.DELTAY))
    g, sq = np.zeros(n * n), 0.0
    for c in range(len(data.freqs)):
        o, e = data.chan_off[c], data.chan_off[c + 1]
        u, v = (data.uvw_m[o:e, k] / _lam(data.freqs[c]) for k in (0, 1))
        neg = u < 0
        u, v = np.where(neg, -u, u), np.where(neg, -v, v)
        x = np.trunc(u / abs(du) + n // 2 + 0.5).astype(np.int64)
        y = np.trunc(v / abs(dv) + n // 2 + 0.5).astype(np.int64)
        ok = (x >= 0) & (y >= 0) & (x < n) & (y < n)
        w = data.weight[o:e].astype(np.float64)
        gc = np.bincount(np.where(ok, n * y + x, 0), weights=w * ok, minlength=n * n)
        cells.append((np.where(ok, n * y + x, 0), ok, w, gc))
        g += gc
        sq += float(np.sum(g.reshape(n, n)[:, n // 2:] ** 2))
    f2 = 25.0 / (sq / float(data.weight.sum(dtype=np.float64)))
    for cell, ok, w, gc in cells:
        with np.errstate(divide="ignore", invalid="ignore"):
            r = w / gc[cell] if case["scheme"] == "uniform" else w / (1.0 + gc[cell] * f2)
        out.append(np.where(ok, r, 0.0))
    return np.concatenate(out)


def _exact_grid(case, data, table, support):
    n, off, ouvw, ovo, ow = data.N, [0], [], [], []
    du = 1.0 / (data.M * (RPDEG * data.DELTAX))
    dv = 1.0 / (data.N * (RPDEG * data.DELTAY))
    tab = table.astype(np.float64)
    for c in range(len(data.freqs)):
        o, e = data.chan_off[c], data.chan_off[c + 1]
        lam = _lam(data.freqs[c])
        u = np.concatenate([data.uvw_m[o:e, 0], -data.uvw_m[o:e, 0]]) / lam
        v = np.concatenate([data.uvw_m[o:e, 1], -data.uvw_m[o:e, 1]]) / lam
        re = np.tile(data.vo[o:e, 0].astype(np.float64), 2)
        im = np.concatenate([data.vo[o:e, 1], -data.vo[o:e, 1]]).astype(np.float64)
        w = np.tile(data.weight[o:e].astype(np.float64), 2)
        j = np.trunc(u / du + n // 2 + 0.5).astype(np.int64)
        k = np.trunc(v / dv + n // 2 + 0.5).astype(np.int64)
        acc = np.zeros((4, n * n))
        for a in range(-support[1], support[1] + 1):
            for b in range(-support[0], support[0] + 1):
                ka, kb = a + support[1], b + support[0]
                if ka >= tab.shape[0] or kb >= tab.shape[1]:
                    continue
                ok = (k + a >= 0) & (k + a < n) & (j + b >= 0) & (j + b < n)
                cell, t = np.where(ok, n * (k + a) + j + b, 0), tab[ka, kb] * ok
                for q, val in enumerate((w * t, w * t * t, w * re * t, w * im * t)):
                    acc[q] += np.bincount(cell, weights=val, minlength=n * n)
        occ = np.nonzero((acc[0] > 0) & (acc[1] > 0))[0]
        g = acc[:, occ]
        off.append(off[-1] + occ.size)
        ouvw.append(np.stack([(occ % n - n // 2) * du * lam, (occ // n - n // 2) * dv * lam,
                              np.zeros(occ.size)], 1))
        ovo.append(np.stack([g[2] / g[0], g[3] / g[0]], 1))
        ow.append(g[0] ** 2 / g[1])
    return {"off": None, "uvw": np.concatenate(ouvw), "vo": np.concatenate(ovo),
            "weight": np.concatenate(ow)}


#: complex multiply-adds in 64 bits that fit the time an exact value may take
MOST = 1.2e12


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None
    if kind == "unet":
        return _exact_unet(case, seed)
    if kind in ("evaluate", "dirty") and 2 * _nvis(case) * case["n"] ** 2 * (
            2 if kind == "dirty" or case["mfs"] else 1) > MOST:
        return None
    data = _data(case, seed)
    if kind == "weights":
        return _exact_weights(case, data)
    if kind == "grid":
        table, support, _ = gv.ckernel_build(case["kernel"], data.M, data.N, data.DELTAX,
                                             data.DELTAY)
        return _exact_grid(case, data, table, support)
    s = _Setup(data)
    if kind == "dirty":
        out = torch.zeros(2, data.N, data.N, dtype=torch.float64, device="cuda")
        zero = torch.zeros(data.N, data.N, dtype=torch.float64, device="cuda")
        for c in range(len(data.freqs)):
            u, v, w, _, wt = s.model(zero, zero, c)
            vo = s.channel(c)[3]
            out[0] += s.adjoint(u, v, w, wt * vo)
            out[1] += s.adjoint(u, v, w, wt.to(torch.complex128))
        return {"dirty": out[0], "psf": out[1]}
    nt = len(_terms(case))
    if kind == "score":
        return [s.evaluate(i, 0, nt, False)[0] for i in _candidates(case, data, seed)]
    img = _image(case, data, seed)
    if kind == "objective":
        f, fi, _, cl = s.evaluate(img, 0, nt, False)
        return {"f": f, "terms": fi, "image": cl}
    out = []
    for flag in range(2 if case["mfs"] else 1):
        f, fi, xi, cl = s.evaluate(img, flag, nt, True)
        out.append({"f": f, "terms": fi, "gradient": xi})
        img = cl.float().cpu()
    return out
