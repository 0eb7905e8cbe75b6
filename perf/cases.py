"""Workloads of the engine with their inputs and float64 references, for timing and comparing builds.

Every case goes through the package's public entry points: per-box plans (``engine``), the
persistent batch (``batch``), delta_T and P(k), initial conditions (``initial``), density evolution
(``perturb``) and the learned surrogate (``surrogate``).  Densities are Gaussian random fields of the
benchmark cosmology drawn on the GPU; parameters are those of the benchmark configurations or, in
drawn cases, of the same ranges.
"""
import importlib
import math

import numpy as np
import torch

PKG = "21cmpy_gb300"
SQRT_2PI2 = 2.0 * math.pi ** 2


def _mod(name):
    return importlib.import_module(PKG + "." + name)


# ------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the 64^3 / 100 Mpc single box: ~95 short launches, where launch latency counts
        dict(name="box_64", kind="box", n=64, L=100.0, z=8.0, zeta=30.0, R_max=15.0, log_tvir=4.0, filter=0,
             update=0, bins=20),
        # one box of the reference's default parameters: HII_DIM 128, 128 Mpc, k-space top hat, 100 bins
        dict(name="box_128", kind="box", n=128, L=128.0, z=9.0, zeta=40.0, R_max=30.0, log_tvir=4.0, filter=1,
             update=0, bins=100),
        # one box of the 52-box 256^3 redshift sweep, the headline workload
        dict(name="box_256", kind="box", n=256, L=300.0, z=8.5, zeta=30.0, R_max=15.0, log_tvir=4.0, filter=0,
             update=0, bins=20),
        # the large single box: 512^3, 600 Mpc, 40 radii
        dict(name="box_512", kind="box", n=512, L=600.0, z=7.5, zeta=20.0, R_max=30.0, log_tvir=4.0, filter=0,
             update=0, bins=20),
        # sphere painting (FIND_BUBBLE_ALGORITHM 1) on a size that is no power of two
        dict(name="sphere_96", kind="box", n=96, L=144.0, z=8.0, zeta=25.0, R_max=15.0, log_tvir=4.0, filter=0,
             update=1, bins=20),
        # parameter sweep over uneven boxes (64, 96, 128, 160) in one persistent launch, with delta_T and P(k)
        dict(name="batch_16", kind="batch", count=16, params=12345, bins=20),
        # delta_T.py alone on a stored x_HI box: brightness temperature and its power spectrum
        dict(name="products_256", kind="products", n=256, L=300.0, z=8.0, bins=100),
        # initialize.py at the reference's default sizes: DIM 512 and its HII_DIM 128 copies
        dict(name="ic_512", kind="ic", dim=512, hii=128, L=128.0),
        # perturb_field.py's Zel'dovich move at the same sizes
        dict(name="move_512", kind="move", dim=512, hii=128, L=128.0, z=8.0, cells=2.0),
        # perturb_field.py's velocity boxes at z from the evolved 512^3 density
        dict(name="velocities_512", kind="velocities", dim=512, hii=128, L=128.0, z=8.0),
        # one surrogate prediction: input features and the network's forward pass
        dict(name="surrogate_128", kind="surrogate", n=128, L=200.0, z=8.0, zeta=30.0, R_max=15.0, log_tvir=4.0,
             train=False),
        # one surrogate training step up to its gradients: features, forward, backward
        dict(name="train_128", kind="surrogate", n=128, L=200.0, z=8.0, zeta=30.0, R_max=15.0, log_tvir=4.0,
             train=True),
    ]


def _zeta_for(z, log_tvir, q):
    """Ionising efficiency that ionises about the fraction q at z, within the configurations' 10-80."""
    cos = _mod("cosmology")
    sigma_min, delta_c = cos.sig_del(10.0 ** log_tvir, z, cos.BASELINE_COSMO)
    return round(min(80.0, max(10.0, q / float(cos.collapse_fraction(sigma_min, delta_c)))), 3)


def draw(rng):
    kind = rng.choice(["box"] * 6 + ["batch", "products", "products", "ic", "move", "move", "velocities", "surrogate",
                                     "surrogate"])
    z = round(rng.uniform(6.0, 11.0), 3)
    log_tvir = round(rng.uniform(4.0, 5.0), 3)
    if kind == "box":
        n = rng.choice([16, 32, 48, 64, 96, 128, 128, 160, 256, 256, 512])
        L = round(n * rng.uniform(1.0, 1.8), 2)
        return dict(kind=kind, n=n, L=L, z=z, zeta=_zeta_for(z, log_tvir, rng.uniform(0.1, 0.8)),
                    R_max=round(min(math.exp(rng.uniform(math.log(4.0), math.log(40.0 if n < 512 else 25.0))), 0.4 * L), 3),
                    log_tvir=log_tvir, filter=rng.choice([0, 0, 1, 2]),
                    update=rng.choice([0, 0, 0, 1]) if n <= 96 else 0, bins=rng.choice([20, 33, 64, 100]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 16), params=rng.randrange(1 << 20), bins=rng.choice([20, 50]))
    if kind == "products":
        n = rng.choice([16, 32, 48, 64, 96, 128, 160, 256, 512])
        return dict(kind=kind, n=n, L=round(n * rng.uniform(0.8, 2.0), 2), z=z, bins=rng.choice([15, 20, 64, 100]))
    if kind in ("ic", "velocities"):
        dim, hii = rng.choice([(128, 32), (128, 64), (160, 48), (160, 32), (256, 64), (256, 100), (256, 128), (512, 128),
                               (512, 256)])
        c = dict(kind=kind, dim=dim, hii=hii, L=round(hii * rng.uniform(0.8, 2.0), 2))
        return c if kind == "ic" else dict(c, z=z)
    if kind == "move":
        dim, hii = rng.choice([(64, 64), (100, 64), (128, 32), (192, 64), (200, 100), (256, 64), (256, 128), (384, 128),
                               (400, 256), (512, 128), (512, 256)])
        return dict(kind=kind, dim=dim, hii=hii, L=round(hii * rng.uniform(0.8, 2.0), 2), z=z,
                    cells=round(math.exp(rng.uniform(math.log(0.3), math.log(5.0))), 3))
    n = rng.choice([32, 64, 128, 128])
    return dict(kind=kind, n=n, L=round(n * rng.uniform(1.2, 1.8), 2), z=min(z, 10.0), zeta=round(rng.uniform(10.0, 80.0), 3),
                R_max=round(rng.uniform(5.0, 50.0), 3), log_tvir=log_tvir, train=rng.random() < 0.5)


# ------------------------------------------------------------------------------------ inputs
def _k2(n, dtype=torch.int64):
    m = torch.arange(n, device="cuda")
    m = torch.where(m > n // 2, m - n, m)
    i = torch.arange(n // 2 + 1, device="cuda")
    return (m[:, None, None] ** 2 + m[None, :, None] ** 2 + i[None, None, :] ** 2).to(dtype)


def _field(n, L, seed, growth, smooth=0.0):
    """Gaussian random density of the benchmark cosmology times `growth`, float32 on the GPU."""
    cos = _mod("cosmology")
    k = 2.0 * math.pi / L * np.sqrt(np.arange(3 * (n // 2) ** 2 + 1))
    amp = np.zeros_like(k)
    amp[1:] = growth * np.sqrt(cos.power_spectrum_z0(k[1:], cos.BASELINE_COSMO) * n ** 3 / L ** 3)
    amp *= np.exp(-0.5 * (k * smooth) ** 2)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    white = torch.randn((n, n, n), device="cuda", generator=g)
    W = torch.fft.rfftn(white)
    W *= torch.from_numpy(amp.astype(np.float32)).cuda()[_k2(n)]
    return torch.fft.irfftn(W, s=(n, n, n)).contiguous()


def _growth(z):
    cos = _mod("cosmology")
    return float(cos.growth_factor(z, cos.BASELINE_COSMO))


def _setup(c):
    cos, sch = _mod("cosmology"), _mod("schedule")
    return sch.ionize_setup(c["n"], c["L"], c["z"], zeta=c["zeta"], t_vir_min=10.0 ** c["log_tvir"], R_max=c["R_max"],
                            cosmo=cos.BASELINE_COSMO, filter_type=c["filter"], update=c["update"])


def _c_factor(z):
    cos = _mod("cosmology")
    return float(cos.brightness_temperature_factor(z, cos.BASELINE_COSMO))


def _batch_specs(c):
    return _mod("grf").uneven_batch(c["count"], param_seed=c["params"])


def _batch_setup(s):
    cos, sch = _mod("cosmology"), _mod("schedule")
    return sch.ionize_setup(s.n, s.box_len, s.z, zeta=s.zeta, t_vir_min=s.t_vir_min, R_max=s.R_max,
                            cosmo=cos.BASELINE_COSMO)


def _normals(c, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    shape = (c["dim"], c["dim"], c["dim"] // 2 + 1)
    return torch.randn(shape, device="cuda", generator=g), torch.randn(shape, device="cuda", generator=g)


def _move_inputs(c, seed):
    """Density at z = 0 and displacement boxes whose rms move at z is c["cells"] HII cells, coherent
    over tens of Mpc as Zel'dovich displacements are."""
    cos = _mod("cosmology")
    g0 = float(np.float32(cos.growth_factor(300.0, cos.BASELINE_COSMO)))
    ds = float(np.float32((_growth(c["z"]) - g0) / c["L"]))
    d = _field(c["dim"], c["L"], seed, 1.0)
    v = []
    for a in range(3):
        f = _field(c["hii"], c["L"], seed * 3 + a + 7, 1.0, smooth=4.0)
        v.append((f * (c["cells"] / c["hii"] / ds / float(f.std()))).contiguous())
    return d, v, g0, ds, float(np.float32((c["dim"] / c["hii"]) ** 3))


def _growth_rate(z):
    cos = _mod("cosmology")
    return float(cos.growth_rate(z, cos.BASELINE_COSMO))


def _target_map(delta):
    """A neutral-fraction-like training target: 0 inside overdense regions of a few cells, 1 outside."""
    n = delta.shape[0]
    s = torch.fft.irfftn(torch.fft.rfftn(delta) * torch.exp(-0.5 * (_k2(n, torch.float32) * (2 * math.pi * 3.0 / n) ** 2)),
                         s=(n, n, n))
    return torch.sigmoid(-12.0 * (s / s.std() - 0.3)).contiguous()


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    s = dict(case=c)
    if kind == "box":
        # a program keeps one plan per box size and hands it every box's density and schedule
        s["setup"] = _setup(c)
        s["delta"] = _field(c["n"], c["L"], seed, _growth(c["z"]))
        s["plan"] = _mod("engine").ExcursionSetPlan(c["n"], c["L"])
        s["edges"] = _mod("schedule").pk_edges(c["n"], c["L"], c["bins"])
        s["c"] = _c_factor(c["z"])
    elif kind == "batch":
        specs = _batch_specs(c)
        boxes = [(_field(b.n, b.box_len, seed + 1000 * i, _growth(b.z)), _batch_setup(b)) for i, b in enumerate(specs)]
        s["batch"] = _mod("batch").BatchedExcursionSet(
            boxes, t_factors=[_c_factor(b.z) for b in specs],
            pk_edges=[_mod("schedule").pk_edges(b.n, b.box_len, c["bins"]) for b in specs])
    elif kind == "products":
        s["delta"] = _field(c["n"], c["L"], seed, _growth(c["z"]))
        s["xH"] = _target_map(s["delta"])
        s["plan"] = _mod("engine").ExcursionSetPlan(c["n"], c["L"])
        s["edges"] = _mod("schedule").pk_edges(c["n"], c["L"], c["bins"])
        s["c"] = _c_factor(c["z"])
    elif kind == "ic":
        s["ic"] = _mod("initial").InitialConditions(c["dim"], c["hii"], c["L"], cosmo=_mod("cosmology").BASELINE_COSMO)
        s["normals"] = _normals(c, seed)
    elif kind == "move":
        s["inputs"] = _move_inputs(c, seed)
        s["plan"] = _mod("perturb").PerturbPlan(c["dim"], c["hii"])
    elif kind == "velocities":
        s["delta"] = _field(c["dim"], c["L"], seed, _growth(c["z"]))
        s["rate"] = _growth_rate(c["z"])
    else:
        s["delta"] = _field(c["n"], c["L"], seed, _growth(c["z"]))
        s["net"] = _mod("surrogate").SurrogateNet(seed=int(seed))
        s["target"] = _target_map(s["delta"]) if c["train"] else None
    return s


# ------------------------------------------------------------------------------------ one pass
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "box":
        p = s["plan"]
        xh, nf = p.run(s["delta"], s["setup"])
        dT, ave = p.delta_T(xh, s["delta"], s["c"])
        return dict(xH=xh, nf=nf, dT=dT, ave=ave, pk=p.power_spectrum(dT, ave, s["edges"]))
    if kind == "batch":
        b = s["batch"]
        out, nf = b.run()
        return dict(xH=out, nf=nf, dT=b.dT, ave=b.ave, pk=b.pk)
    if kind == "products":
        p = s["plan"]
        dT, ave = p.delta_T(s["xH"], s["delta"], s["c"])
        return dict(dT=dT, ave=ave, pk=p.power_spectrum(dT, ave, s["edges"]))
    if kind == "ic":
        return s["ic"].generate(normals=s["normals"])
    if kind == "move":
        d, v, g0, ds, mf = s["inputs"]
        return s["plan"].move_mass(d, *v, init_growth=g0, disp_scale=ds, mass_factor=mf)
    if kind == "velocities":
        return _mod("perturb").updated_velocities(s["delta"], c["hii"], c["L"], s["rate"])
    net = s["net"]
    f = net.features(s["delta"], c["z"], c["zeta"], c["R_max"], 10.0 ** c["log_tvir"])
    if not c["train"]:
        return net.forward(f)[0]
    pred, acts = net.forward(f, keep=True)
    dws, dbs = net.backward(acts, pred, s["target"])
    return dict(pred=pred, dw=dws, db=dbs)


# ------------------------------------------------------------------------------------ work of a pass
def _fft_flops(n):
    return 2.5 * n ** 3 * math.log2(n ** 3)


def _half(n):
    return 8.0 * n * n * (n // 2 + 1)


def _layer_flops(n, train):
    f = [2.0 * 27 * ci * co * n ** 3 for ci, co in [(16, 32)] + [(32, 32)] * 6 + [(32, 16)]]
    return sum(f) + (sum(f) + sum(f[1:]) if train else 0.0)


def work(case):
    """Bytes of the inputs and outputs, each once, and the floating-point operations of the
    transforms (2.5 N^3 log2 N^3 for a real one), windows, erfc sums (25 a voxel) and convolutions."""
    c = dict(case)
    kind = c["kind"]
    if kind == "box":
        n3, nr = float(c["n"]) ** 3, _setup(c).n_radii
        return dict(bytes=12 * n3, flops=(nr + 2) * _fft_flops(c["n"]) + nr * 29 * n3 + 40 * n3)
    if kind == "batch":
        b = f = 0.0
        for s in _batch_specs(c):
            n3, nr = float(s.n) ** 3, _batch_setup(s).n_radii
            b += 12 * n3
            f += (nr + 2) * _fft_flops(s.n) + nr * 29 * n3 + 40 * n3
        return dict(bytes=b, flops=f)
    if kind == "products":
        n3 = float(c["n"]) ** 3
        return dict(bytes=12 * n3, flops=_fft_flops(c["n"]) + 15 * n3)
    if kind == "ic":
        n, m3 = c["dim"], float(c["hii"]) ** 3
        return dict(bytes=2 * _half(n) + 4.0 * n ** 3 + 16 * m3, flops=_fft_flops(n) + 10.0 * n ** 3 + 4 * _fft_flops(c["hii"]))
    if kind == "move":
        return dict(bytes=4.0 * c["dim"] ** 3 + 16.0 * c["hii"] ** 3, flops=12.0 * c["dim"] ** 3)
    if kind == "velocities":
        n = c["dim"]
        return dict(bytes=4.0 * n ** 3 + 12.0 * c["hii"] ** 3, flops=_fft_flops(n) + 10.0 * n ** 3 + 3 * _fft_flops(c["hii"]))
    n = c["n"]
    n3 = float(n) ** 3
    weights = 4.0 * 27 * sum(ci * co for ci, co in [(16, 32)] + [(32, 32)] * 6 + [(32, 16)])
    return dict(bytes=(12 if c["train"] else 8) * n3 + weights * (2 if c["train"] else 1),
                flops=_layer_flops(n, c["train"]) + 5 * _fft_flops(n))


# ------------------------------------------------------------------------------------ float64 references
def _tophat(x):
    y = np.ones_like(x)
    b = x > 1e-2
    y[b] = 3.0 * (np.sin(x[b]) - x[b] * np.cos(x[b])) / x[b] ** 3
    s = x[~b] ** 2
    y[~b] = 1.0 - s / 10.0 + s * s / 280.0
    return y


def _dk(L):
    return float(np.float32(2.0 * math.pi / float(np.float32(L))))


def _window(n, dk, R, filt):
    x = dk * np.sqrt(np.arange(3 * (n // 2) ** 2 + 1, dtype=np.float64)) * R
    if filt == 0:
        return _tophat(x)
    return (x * 0.413566994 <= 1.0).astype(np.float64) if filt == 1 else np.exp(-0.5 * (0.643 * x) ** 2)


def _ball_paint(flags, R, scale):
    n = flags.shape[0]
    m = torch.arange(n, device="cuda")
    m = torch.minimum(m, n - m)
    r2 = m[:, None, None] ** 2 + m[None, :, None] ** 2 + m[None, None, :] ** 2
    ball = (r2.double() < (R / scale) ** 2).double()
    return torch.fft.irfftn(torch.fft.rfftn(flags.double()) * torch.fft.rfftn(ball), s=(n, n, n)) > 0.5


def _exact_box(delta, st):
    n = delta.shape[0]
    X = torch.fft.rfftn(delta.double()) * float(st.growth_scale)
    k2, dk = _k2(n), _dk(st.box_len)
    dc, inv_zeta = float(st.deltac32), float(np.float32(1.0 / float(np.float32(st.zeta))))
    ion = torch.zeros((n, n, n), dtype=torch.bool, device="cuda")
    for i, step in enumerate(st.steps):
        W = torch.from_numpy(_window(n, dk, float(step.R), st.filter_type)).cuda()
        f = torch.erfc((dc - torch.fft.irfftn(X * W[k2], s=(n, n, n))) / float(step.denom))
        if st.normalize_mean:
            f *= float(st.fc_mean_ps) / f.mean()
        over = f >= inv_zeta
        if i + 1 < st.n_radii:
            ion |= _ball_paint(over, float(step.R), st.scale) if st.update else over
    return 1.0 - torch.where(ion | over, torch.ones_like(f), f * float(np.float32(st.zeta)))


def _exact_products(xH, delta, cfac, L, bins):
    n = delta.shape[0]
    dT = float(np.float32(cfac)) * xH.double() * (1.0 + delta.double())
    ave = dT.mean()
    L = float(np.float32(L))
    k2, dk = _k2(n).reshape(-1), _dk(L)
    G = torch.fft.rfftn((dT / ave - 1.0) * (L ** 3 / n ** 3)).reshape(-1)
    k = dk * torch.sqrt(k2.double())
    edges = np.float32(np.logspace(np.log10(dk), np.log10(dk * np.sqrt(3.0) * n), bins)).astype(np.float64)
    b = torch.searchsorted(torch.from_numpy(edges).cuda(), k)
    i = torch.arange(n // 2 + 1, device="cuda")
    w = torch.where((i > 0) & (i < n // 2), 2.0, 1.0).double().repeat(n * n)
    w = torch.where((k2 > 0) & (b < bins), w, torch.zeros_like(w))
    b = b.clamp(max=bins - 1)
    sums = [torch.zeros(bins, dtype=torch.float64, device="cuda").index_add_(0, b, w * q)
            for q in (k ** 3 * G.abs() ** 2 / (SQRT_2PI2 * L ** 3), k, torch.ones_like(k))]
    cnt = sums[2].clamp(min=1.0)
    return dT, ave.reshape(1), torch.stack([sums[0] / cnt, sums[1] / cnt, sums[2]])


def _subsample(x, m):
    n = x.shape[0]
    pf = np.float32(n) / np.float32(m)
    i = np.floor(np.arange(m, dtype=np.float32) * pf + np.float32(0.5)).astype(np.int64).clip(0, n - 1)
    i = torch.from_numpy(i).cuda()
    return x[i][:, i][:, :, i].clone()


def _exact_velocities(H, n, hii, L, norm):
    m = torch.arange(n, device="cuda")
    m = torch.where(m > n // 2, m - n, m).double()
    i = torch.arange(n // 2 + 1, device="cuda").double()
    m, i = torch.where(m == n // 2, 0.0, m), torch.where(i == n // 2, 0.0, i)
    k2, dk = _k2(n), float(np.float32(2.0 * math.pi / float(np.float32(L))))
    R = float(np.float32(np.float32(0.620350491) * np.float32(L) / np.float32(hii)))
    W = _window(n, dk, R, 0)
    smooth = torch.from_numpy(W).cuda()[k2]
    W[1:] /= np.arange(1, len(W)) * dk
    W[0] = 0.0
    f = torch.from_numpy(W).cuda()[k2]
    out = {"smoothed": _subsample(torch.fft.irfftn(H * smooth, s=(n, n, n)) * float(n) ** 3, hii) * norm}
    for name, kc in (("vx", m[:, None, None]), ("vy", m[None, :, None]), ("vz", i[None, None, :])):
        out[name] = _subsample(torch.fft.irfftn(H * (1j * kc * f), s=(n, n, n)) * float(n) ** 3, hii) * norm
    return out


def _exact_spectrum(c, nre, nim):
    n, dk = c["dim"], float(np.float32(2.0 * math.pi / float(np.float32(c["L"]))))
    K, P = _mod("initial").pk_table(n, float(np.float32(c["L"])), _mod("cosmology").BASELINE_COSMO)
    k = dk * np.sqrt(np.arange(3 * (n // 2) ** 2 + 1, dtype=np.float64))
    amp = np.sqrt(np.interp(k, K.astype(np.float64), P.astype(np.float64)) * float(np.float32(c["L"])) ** 3)
    amp[0] = 0.0
    X = torch.complex(nre.double(), nim.double())
    i = (-torch.arange(n, device="cuda")) % n
    for plane in (0, n // 2):
        X[:, :, plane] = 0.5 * (X[:, :, plane] + X[:, :, plane].conj()[i][:, i])
    X[:, :, 1:n // 2] *= math.sqrt(0.5)
    return X * torch.from_numpy(amp).cuda()[_k2(n)]


def _exact_move(c, seed):
    d, v, g0, ds, mf = _move_inputs(c, seed)
    n, sw = c["dim"], c["hii"]
    pos = torch.from_numpy(((np.arange(n) + 0.5) / n).astype(np.float32)).cuda()
    h = torch.from_numpy(np.floor(np.arange(n, dtype=np.float32) / np.float32(np.float32(n) / np.float32(sw))).astype(np.int64)).cuda()
    out = torch.zeros(sw ** 3, dtype=torch.float64, device="cuda")
    for a in range(0, n, 16):                    # which cell a mass lands in is decided in float32
        cell = torch.zeros((min(16, n - a), n, n), dtype=torch.int64, device="cuda")
        for axis in range(3):
            p = pos[a:a + 16, None, None] if axis == 0 else (pos[None, :, None] if axis == 1 else pos[None, None, :])
            f = (p + v[axis][h[a:a + 16]][:, h][:, :, h] * ds) * float(sw)
            for _ in range(64):
                f = torch.where(f >= sw, f - float(sw), f)
                f = torch.where(f < 0, f + float(sw), f)
            cell = cell * sw + (f.to(torch.int64) % sw)
        out.index_add_(0, cell.reshape(-1), (1.0 + g0 * d[a:a + 16].double()).reshape(-1))
    return out.reshape(sw, sw, sw) / mf - 1.0


def _shifts():
    return [(t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1) for t in range(27)]


def _conv64(x, w):
    """out[v] = sum over taps of x[v + tap] w[tap]^T, channels last, circular."""
    out = None
    for t, sh in enumerate(_shifts()):
        y = torch.roll(x, tuple(-q for q in sh), (0, 1, 2)) @ w[t].T
        out = y if out is None else out.add_(y)
    return out


def _exact_surrogate(s):
    c, net = s["case"], s["net"]
    n = c["n"]
    cos = _mod("cosmology")
    x = torch.zeros((n, n, n, 16), dtype=torch.float64, device="cuda")
    scale = 1.0 / (4.0 * cos.growth_factor(c["z"], cos.BASELINE_COSMO))
    x[..., 0] = s["delta"].double() * scale
    for i, q in enumerate((c["zeta"] / 80.0, c["R_max"] / 50.0, c["log_tvir"] - 4.0, (c["z"] - 6.0) / 4.0)):
        x[..., 1 + i] = q
    X, k2 = torch.fft.rfftn(s["delta"].double()), _k2(n)
    for j, R in enumerate(net.smoothing):
        W = torch.from_numpy(_window(n, 2.0 * math.pi / n, R, 0)).cuda()
        x[..., 5 + j] = torch.fft.irfftn(X * W[k2], s=(n, n, n)) * scale
    w = [q.double() for q in net.w]
    acts = [x]
    for i in range(len(w) - 1):
        acts.append(torch.relu_(_conv64(acts[-1], w[i]) + net.b[i].double()))
    pred = torch.sigmoid(_conv64(acts[-1], w[-1][:, :1]) + net.b[-1][:1].double())[..., 0]
    if not c["train"]:
        return pred
    dz = torch.zeros((n, n, n, w[-1].shape[1]), dtype=torch.float64, device="cuda")
    dz[..., 0] = pred - s["target"].double()
    dws, dbs = [], []
    for i in range(len(w) - 1, -1, -1):
        flat = dz.reshape(-1, dz.shape[-1]).T.contiguous()
        dws.append(torch.stack([flat @ torch.roll(acts[i], tuple(-q for q in sh), (0, 1, 2)).reshape(-1, w[i].shape[2])
                                for sh in _shifts()]))
        dbs.append(dz.sum((0, 1, 2)))
        if i:
            dz = _conv64(dz, w[i].flip(0).transpose(1, 2)) * (acts[i] > 0)
    dws[-1][:, :, net.n_in:] = 0.0
    return dict(pred=pred, dw=dws[::-1], db=dbs[::-1])


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "box":
        d = _field(c["n"], c["L"], seed, _growth(c["z"]))
        xH = _exact_box(d, _setup(c))
        dT, ave, pk = _exact_products(xH, d, _c_factor(c["z"]), c["L"], c["bins"])
        return dict(xH=xH, nf=xH.mean().reshape(1), dT=dT, ave=ave, pk=pk)
    if kind == "batch":
        got = dict(xH=[], nf=[], dT=[], ave=[], pk=[])
        for i, b in enumerate(_batch_specs(c)):
            d = _field(b.n, b.box_len, seed + 1000 * i, _growth(b.z))
            xH = _exact_box(d, _batch_setup(b))
            dT, ave, pk = _exact_products(xH, d, _c_factor(b.z), b.box_len, c["bins"])
            for key, q in zip(("xH", "nf", "dT", "ave", "pk"), (xH, xH.mean().reshape(1), dT, ave, pk)):
                got[key].append(q)
        return dict(got, nf=torch.cat(got["nf"]), ave=torch.cat(got["ave"]))
    if kind == "products":
        d = _field(c["n"], c["L"], seed, _growth(c["z"]))
        dT, ave, pk = _exact_products(_target_map(d), d, _c_factor(c["z"]), c["L"], c["bins"])
        return dict(dT=dT, ave=ave, pk=pk)
    if kind == "ic":
        H = _exact_spectrum(c, *_normals(c, seed))
        n = c["dim"]
        norm = 1.0 / float(np.float32(c["L"])) ** 3
        return dict(_exact_velocities(H, n, c["hii"], c["L"], norm), spectrum=H,
                    deltax=torch.fft.irfftn(H, s=(n, n, n)) * (float(n) ** 3 * norm))
    if kind == "move":
        return _exact_move(c, seed)
    if kind == "velocities":
        n = c["dim"]
        H = torch.fft.rfftn(_field(n, c["L"], seed, _growth(c["z"])).double())
        got = _exact_velocities(H, n, c["hii"], c["L"], _growth_rate(c["z"]) / float(n) ** 3)
        got.pop("smoothed")
        return got
    return _exact_surrogate(prepare(case, seed))
