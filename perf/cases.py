"""Performance cases of the framework: one pass of each public path on seeded synthetic boxes.

A case is a dict of plain values; ``prepare`` builds what a user's program holds before the call (the
boxes or the catalogue and a context of the library), ``run`` makes one pass through the public entry
points, ``exact`` gives the same outputs in float64 with plain torch, ``work`` the bytes and operations
the pass cannot do without.  The kinds of case:

  hii    the bubble filter bank, device boxes (FilterBank.run_z_device), one or more parameter sets,
         one redshift or a short series of them on one context
  host   the same through host boxes (FilterBank.run_z), as the executable sf21_hii calls it
  grad   the continuous criterion and its vector-Jacobian product
  halo   the halo finder of one redshift, catalogue on the host, with or without the subgrid cycle
  sfr    the star-formation-rate box of a halo catalogue on the device
  pk     the power spectrum of a device box
  t21    the 21-cm brightness temperature, host boxes, with or without the spin boxes
"""
import ctypes
import math

import numpy as np
import torch

from simfast21_gb300 import halos, hii, sfr, synth

HUBBLE = 0.71
PI2 = 2.0 * math.pi
# sides the drawn cases take besides powers of two: products of 2, 3 and 5 that 8 divides
RAGGED = [24, 40, 48, 72, 80, 96, 120, 144, 160, 200, 216, 240, 288, 320, 360, 400, 432, 480, 600]


# ---- the cases ---------------------------------------------------------------------------------
def listed():
    return [
        # the smallest box of the tests: a call is a few dozen short launches
        dict(name="hii-32", kind="hii", N=32, L=25.0, z=8.0, nz=1, src="sfrd", sets=1, zeta=30.0, rmax=12.0,
             factor=1.1),
        # the reference's plain method: 128^3, zeta 30, Rmax 50 Mpc/h, radius factor 1.1
        dict(name="hii-128", kind="hii", N=128, L=100.0, z=8.0, nz=1, src="sfrd", sets=1, zeta=30.0, rmax=50.0,
             factor=1.1),
        # part of a redshift series on one context, as a simulation visits it: every redshift has boxes of its own
        dict(name="hii-256-series", kind="hii", N=256, L=200.0, z=12.0, nz=3, src="sfrd", sets=1, zeta=30.0,
             rmax=60.0, factor=1.05),
        # the batched form at 512^3: eight parameter sets share one forward transform
        dict(name="hii-512-batched", kind="hii", N=512, L=300.0, z=7.0, nz=1, src="sfrd", sets=8, zeta=0.0,
             rmax=60.0, factor=1.05),
        # the reference's default N_smoothed
        dict(name="hii-600", kind="hii", N=600, L=106.5, z=7.0, nz=1, src="sfrd", sets=1, zeta=30.0, rmax=35.5,
             factor=1.05),
        # a ragged side with the halo branch's source box (Rion after the block average)
        dict(name="hii-360-rion", kind="hii", N=360, L=150.0, z=7.5, nz=1, src="rion", sets=2, zeta=0.0, rmax=40.0,
             factor=1.1),
        # host boxes in and out with the neutral fraction: the call the executable makes per redshift
        dict(name="host-256", kind="host", N=256, L=150.0, z=7.0, nz=1, src="sfrd", sets=1, zeta=30.0, rmax=30.0,
             factor=1.05),
        # criterion and gradient of the differentiation configuration
        dict(name="grad-256", kind="grad", N=256, L=200.0, z=8.0, src="sfrd", zeta=30.0, rmax=60.0, factor=1.05),
        # halo finder with the subgrid cycle at the benchmark's cell size
        dict(name="halo-512-subgrid", kind="halo", N=512, cell=100.0 / 512, z=7.0, sigma=4.0, subgrid=True),
        # star-formation-rate stage at the default grids
        dict(name="sfr-1200-600", kind="sfr", N_halo=1200, N=600, L=105.0, z=8.0, n=20_000_000),
        # power spectrum of a large box
        dict(name="pk-512", kind="pk", N=512, dl=0.3, window=1),
        # brightness temperature with the spin-temperature boxes
        dict(name="t21-256-spin", kind="t21", N=256, L=150.0, z=9.0, axis=3, spin=True),
    ]


def _side(rng, lo, hi):
    """A supported side, spread over the logarithm of [lo, hi], powers of two and ragged ones alike."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    pool = [1 << k for k in range(4, 11)] if rng.random() < 0.5 else RAGGED
    return min((s for s in pool if lo <= s <= hi), key=lambda s: abs(math.log(s / n)))


def draw(rng):
    kind = rng.choice(["hii"] * 7 + ["host", "grad", "grad", "halo", "halo", "sfr", "pk", "t21"])
    z = round(rng.uniform(6.0, 12.0), 3)
    if kind in ("hii", "host", "grad"):
        # the filtered-field gradient takes boxes up to 320, the host calls up to 400
        N = _side(rng, 16, {"hii": 600, "host": 400, "grad": 320}[kind])
        L = N * round(rng.uniform(0.2, 0.9), 4)
        case = dict(kind=kind, N=N, L=L, z=z, src=rng.choice(["sfrd", "rion"]),
                    zeta=round(math.exp(rng.uniform(math.log(10.0), math.log(100.0))), 3),
                    rmax=round(max(L * rng.uniform(0.08, 0.5), 4.0 * L / N), 3), factor=round(rng.uniform(1.05, 1.2), 3))
        if kind == "hii":
            case["sets"] = rng.randint(1, 4 if N <= 512 else 1)
            case["nz"] = rng.choice([1, 1, 2]) if N <= 256 else 1
        if kind == "host":
            case["sets"], case["nz"] = rng.randint(1, 2), 1
        return case
    if kind == "halo":
        N = _side(rng, 32, 480)
        return dict(kind="halo", N=N, cell=round(rng.uniform(0.18, 0.25), 4), z=round(rng.uniform(6.0, 9.0), 3),
                    sigma=round(rng.uniform(3.0, 4.0), 3), subgrid=rng.random() < 0.5)
    if kind == "sfr":
        N = _side(rng, 24, 600)
        n_halo = N * rng.choice([1, 2, 2, 3]) if N <= 400 else 2 * N
        most = min(2e7, 0.1 * n_halo ** 3)  # the halo finder leaves up to a tenth of a halo per cell
        return dict(kind="sfr", N_halo=n_halo, N=N, L=N * round(rng.uniform(0.15, 0.5), 4), z=z,
                    n=int(math.exp(rng.uniform(math.log(1e3), math.log(most)))))
    N = _side(rng, 32, 512 if kind == "pk" else 400)
    if kind == "pk":
        return dict(kind="pk", N=N, dl=round(rng.uniform(0.1, 1.0), 4), window=rng.randint(0, 2))
    return dict(kind="t21", N=N, L=N * round(rng.uniform(0.2, 0.9), 4), z=z, axis=rng.randint(1, 3),
                spin=rng.random() < 0.5)


# ---- inputs ------------------------------------------------------------------------------------
def _sets(case):
    """(zeta, Rmax, Nbins) of each set.  With zeta = 0 in the case the sets follow the benchmark's ranges: zeta
    log-uniform on [10, 100], Rmax uniform on [rmax/6, rmax]; several sets of a drawn case lie around its own."""
    dx = case["L"] / case["N"]
    n = case.get("sets", 1)
    rng = np.random.default_rng(1236)
    out = []
    for s in range(n):
        zeta, rmax = case["zeta"], case["rmax"]
        u, v = rng.random(2)
        if case["zeta"] == 0.0:
            zeta, rmax = 10.0 * 10.0 ** u, rmax * (1.0 + 5.0 * v) / 6.0
        elif s:
            zeta, rmax = zeta * (0.5 + u), rmax * (0.3 + 0.7 * v)
        rmax = max(min(rmax, case["L"] / 2.0), 1.5 * dx)
        out.append((zeta, rmax, max(1, int(round(math.log(rmax / dx) / math.log(case["factor"]))))))
    return out


def _redshifts(case):
    return [case["z"] - 0.3 * i for i in range(case.get("nz", 1))]


def _n_halo(case):
    return 2 * case["N"] if case["src"] == "rion" else case["N"]


def _boxes(case, z, seed):
    """(density, source) boxes of one redshift on the GPU: a lognormal density and one-halo-per-cell sources."""
    N, L = case["N"], case["L"]
    sigma = 0.8 * synth.growth(z) / synth.growth(8.0)
    delta, src = synth.make_boxes_torch(N, L, z, seed, sigma=sigma)
    if case["src"] == "rion":  # the ionisation rate itself, before the factor (dx / dx_halo)^3
        src = (src.double() * (L / N) ** 3 * synth.qion(z) / (_n_halo(case) / N) ** 3).float()
    return delta, src


def _gaussian(N, seed, sigma):
    """A Gaussian density box with P(k) ~ k^-2 and the given rms per cell, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    w = torch.fft.rfftn(torch.randn((N, N, N), generator=g, device="cuda"))
    f = torch.fft.fftfreq(N, 1.0 / N, device="cuda")
    h = torch.arange(N // 2 + 1, device="cuda", dtype=torch.float32)
    k2 = f[:, None, None] ** 2 + f[None, :, None] ** 2 + h ** 2
    w *= torch.where(k2 > 0, k2.clamp(min=1.0) ** -0.5, torch.zeros_like(k2))
    d = torch.fft.irfftn(w, s=(N, N, N))
    return ((d - d.mean()) * (sigma / d.std())).contiguous()


def _catalogue(case, seed):
    """(n, 4) halo records on the GPU: the halo finder's mass schedule (1e8 Msun up, 0.2 dex apart), abundance
    falling as M^-0.9, uniform positions in cells of the fine grid."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    m = 1e8 * 10.0 ** (0.2 * torch.arange(21, dtype=torch.float64, device="cuda"))
    cut = torch.cumsum(m ** -0.9, 0)
    u = torch.rand(case["n"], generator=g, device="cuda", dtype=torch.float64) * cut[-1]
    cat = torch.rand((case["n"], 4), generator=g, device="cuda", dtype=torch.float32) * case["N_halo"]
    cat.clamp_(max=float(np.nextafter(np.float32(case["N_halo"]), np.float32(0))))
    cat[:, 0] = m[torch.searchsorted(cut, u).clamp(max=20)].float()
    return cat


def _t21_boxes(case, seed):
    N = case["N"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    delta = torch.exp(_gaussian(N, seed, 0.8) - 0.32) - 1.0
    rand = lambda: torch.rand((N, N, N), generator=g, device="cuda")  # noqa: E731
    boxes = dict(delta=delta, xhii=(1.6 * rand() - 0.3).clamp(0.0, 1.0))
    if case["spin"]:
        boxes.update(xc=0.1 * rand(), xalpha=5.0 * rand() ** 2, tempx=10.0 * 100.0 ** rand())
    return boxes


def _bank(case, sets):
    return hii.FilterBank(case["N"], case["L"], HUBBLE, sets, N_halo=_n_halo(case))


def prepare(case, seed):
    kind, N = case["kind"], case.get("N")
    st = dict(case=case)
    if kind in ("hii", "host"):
        st["zs"] = _redshifts(case)
        boxes = [_boxes(case, z, seed * 16 + i) for i, z in enumerate(st["zs"])]
        st["kind"] = hii.SF21_SRC_SFRD if case["src"] == "sfrd" else hii.SF21_SRC_RION
        st["bank"] = _bank(case, _sets(case))
        if kind == "host":
            st["boxes"] = [(d.cpu().numpy(), s.cpu().numpy()) for d, s in boxes]
            st["out"] = np.empty((case["sets"], N, N, N), np.float32)
        else:
            st["boxes"] = boxes
            st["out"] = torch.empty((len(st["zs"]), case["sets"], N, N, N), device="cuda")
            st["stream"] = torch.cuda.Stream()
    elif kind == "grad":
        st["boxes"] = _boxes(case, case["z"], seed)
        st["g"] = _weights(N, seed)
        st["kind"] = hii.SF21_SRC_SFRD if case["src"] == "sfrd" else hii.SF21_SRC_RION
        st["bank"] = _bank(case, _sets(case))
        st["C"], st["gd"], st["gs"] = (torch.empty((N, N, N), device="cuda") for _ in range(3))
        st["A"] = torch.empty((N, N, N), dtype=torch.uint8, device="cuda")
        st["stream"] = torch.cuda.Stream()
    elif kind == "halo":
        w = synth.HaloWorkload(N=N, L_mpc=N * case["cell"], subgrid=case["subgrid"])
        cfg = halos.config_from_ini(halos.parse_ini(synth.halo_ini_text(w, case["z"], case["z"], 1.0)))
        st["finder"] = halos.HaloFinder(cfg)
        st["finder"].set_density(_gaussian(N, seed, case["sigma"]).cpu().numpy())
        st["records"] = np.zeros((N ** 3 // 6, 4), np.float32)  # room for the records of one redshift
    elif kind == "sfr":
        st["cat"] = _catalogue(case, seed)
        st["box"] = sfr.SFRBox(case["N_halo"], N, case["L"])
        st["out"] = torch.empty((N, N, N), device="cuda")
        st["stream"] = torch.cuda.Stream()
    elif kind == "pk":
        st["delta"] = torch.exp(_gaussian(N, seed, 0.8) - 0.32) - 1.0
        st["bank"] = hii.FilterBank(N, N * case["dl"], HUBBLE, [(1.0, N * case["dl"] / 4, 1)], kmax=1, path=1)
        st["stream"] = torch.cuda.Stream()
    else:
        st["boxes"] = {k: v.cpu().numpy() for k, v in _t21_boxes(case, seed).items()}
        st["bank"] = hii.FilterBank(N, case["L"], HUBBLE, [(1.0, case["L"] / 4, 1)], kmax=1, path=1)
    return st


def _weights(N, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 7)
    return torch.rand((N, N, N), generator=g, device="cuda")


# ---- one pass ----------------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "hii":
        for i, (z, (delta, src)) in enumerate(zip(st["zs"], st["boxes"])):
            st["bank"].run_z_device(z, delta.data_ptr(), src.data_ptr(), st["out"][i].data_ptr(), st["kind"],
                                    stream=st["stream"].cuda_stream)
        return st["out"]
    if kind == "host":
        return st["bank"].run_z(st["zs"][0], *st["boxes"][0], st["kind"], out=st["out"])
    if kind == "grad":
        p = [t.data_ptr() for t in st["boxes"]]
        s = st["stream"].cuda_stream
        st["bank"].criterion_device(case["z"], *p, st["C"].data_ptr(), st["A"].data_ptr(), src_kind=st["kind"], stream=s)
        gz = st["bank"].vjp_device(case["z"], *p, st["g"].data_ptr(), st["gd"].data_ptr(), st["gs"].data_ptr(),
                                   src_kind=st["kind"], stream=s)
        return dict(C=st["C"], A=st["A"], ddelta=st["gd"], dsrc=st["gs"], dzeta=gz)
    if kind == "halo":
        # the C calls, with a record buffer that the program keeps; every pass is the first redshift of a run
        hf, lib, n = st["finder"], halos.load_library(), ctypes.c_long(0)
        hf.set_rng()
        hf._check(lib.sf21_halo_find_z(hf._h, case["z"], ctypes.byref(n)))
        if n.value:
            hf._check(lib.sf21_halo_fetch(hf._h, st["records"].ctypes.data, 0, min(n.value, len(st["records"]))))
        return st["records"], n.value
    if kind == "sfr":
        st["box"].box_device(case["z"], case["n"], st["cat"].data_ptr(), st["out"].data_ptr(), st["stream"].cuda_stream)
        return st["out"]
    if kind == "pk":
        return st["bank"].power_spectrum_device(st["delta"].data_ptr(), case["dl"], case["window"],
                                                st["stream"].cuda_stream)
    b = st["boxes"]
    tb, mean, ts = st["bank"].t21(case["z"], b["delta"], b["xhii"], vel_comp=case["axis"], xc=b.get("xc"),
                                  xalpha=b.get("xalpha"), tempx=b.get("tempx"))
    return [tb, mean] + ([ts] if case["spin"] else [])


# ---- the same in 64 bits -------------------------------------------------------------------------
def _radii(rmax, dx, nbins):
    """Descending radii and how many of them are at least two cells."""
    b, R, out = 10.0 ** (math.log10(rmax / dx) / nbins), rmax, []
    while R >= dx:
        out.append(R)
        R /= b
    return out, sum(r >= 2 * dx for r in out)


def _axes(N):
    f = torch.fft.fftfreq(N, 1.0 / N, device="cuda", dtype=torch.float64)
    return f, torch.arange(N // 2 + 1, device="cuda", dtype=torch.float64)


def _kmag(N, L):
    f, h = _axes(N)
    return (PI2 / L) * torch.sqrt(f[:, None, None] ** 2 + f[None, :, None] ** 2 + h ** 2)


def _tophat(x):
    s = torch.where(x < 0.03, torch.ones_like(x), x)
    return torch.where(x < 0.03, 1.0 - x * x / 10.0, 3.0 * (torch.sin(s) / s - torch.cos(s)) / (s * s))


def _rec(od, case, z):
    """Recombination rate of a cell of overdensity od."""
    cell = (case["L"] * 3.0857e24 / case["N"] / HUBBLE / (1.0 + z)) ** 3
    q = (od / 1.76105133) ** 0.81722878
    return 1e-24 * 9.84815696 * (1.0 + z) ** 5.06773134 * (q / (1.0 + q)) ** 4 * cell / 1e45


def _ion_scale(case, z):
    """Ionisation rate per unit of the source box, without the efficiency."""
    dx = case["L"] / case["N"]
    return dx ** 3 * synth.qion(z) if case["src"] == "sfrd" else float(_n_halo(case) / case["N"]) ** 3


def _neutral_residual(od, z):
    lo = -4.37152818e-05 * z ** 5 + 1.64394635e-03 * z ** 4 - 2.03044756e-02 * z ** 3
    hi = 7.18335221e-02 * z ** 2 - 8.85791388e-02 * z - 1.20887500e+01
    r = od * 1.881e-7 * (1.0 + z) ** 3 * 4.19232273531e-13 / 10.0 ** (lo + hi)
    s = 2.0 * r + 1.0
    return 2.0 * r / (s + torch.sqrt(s * s - 4.0 * r * r))  # = (s - sqrt(s^2 - 4 r^2)) / (2 r) for r > 0


def _xhii(case, z, delta, src):
    """xHII of every set: centres per radius, the discrete balls around them, the single-cell fill, the cap."""
    N, L = case["N"], case["L"]
    dx, n3, size = L / N, float(N) ** 3, (N, N, N)
    od = 1.0 + delta.double()
    rec, ion = _rec(od, case, z), src.double() * _ion_scale(case, z)
    cap = 1.0 - _neutral_residual(od, z)
    k, fr, fi = _kmag(N, L), torch.fft.rfftn(rec), torch.fft.rfftn(ion)
    f = torch.fft.fftfreq(N, 1.0 / N, device="cuda", dtype=torch.float64)
    dist = torch.sqrt(f[:, None, None] ** 2 + f[None, :, None] ** 2 + f ** 2) * dx
    out = []
    for zeta, rmax, nbins in _sets(case):
        x = (ion * zeta / rec).clamp(max=1.0)
        for R in _radii(rmax, dx, nbins)[0]:
            w = _tophat(k * R)
            h = torch.fft.irfftn(fi * w, s=size) * (n3 * zeta)
            centre = (h > 0) & (h >= torch.fft.irfftn(fr * w, s=size) * n3)
            if bool(src.any()) and bool(centre.any()):
                ball = torch.fft.rfftn((dist <= R).double())
                near = torch.fft.irfftn(torch.fft.rfftn(centre.double()) * ball, s=size)
                x[near > 0.5] = 1.0
        out.append(torch.minimum(x, cap))
    return torch.stack(out)


def _criterion_grad(case, delta, src, g):
    N, L, z = case["N"], case["L"], case["z"]
    dx, n3, size = L / N, float(N) ** 3, (N, N, N)
    (zeta, rmax, nbins), = _sets(case)
    radii, n_fft = _radii(rmax, dx, nbins)
    od = (1.0 + delta.double()).requires_grad_()
    rec = _rec(od, case, z)
    scale = _ion_scale(case, z)
    k = _kmag(N, L)
    fr, fi = torch.fft.rfftn(rec.detach()), torch.fft.rfftn(src.double() * scale)

    def fields(R):
        w = _tophat(k * R)
        return w, torch.fft.irfftn(fr * w, s=size) * n3, torch.fft.irfftn(fi * w, s=size) * (n3 * zeta)

    best = torch.zeros(size, dtype=torch.float64, device="cuda")
    arg = torch.full(size, 255, dtype=torch.uint8, device="cuda")
    for i, R in enumerate(radii[:n_fft]):
        _, d, h = fields(R)
        c = torch.where(d > 0, h / d, torch.full_like(d, -1.0))
        up = (d > 0) & ((arg == 255) | (c > best))
        best = torch.where(up, c, best)
        arg[up] = i
    gg = g.double()
    ar, ai = torch.zeros_like(fr), torch.zeros_like(fi)
    for i, R in enumerate(radii[:n_fft]):
        w, d, _ = fields(R)
        q = torch.where(arg == i, gg / d, torch.zeros_like(d))
        ai += torch.fft.rfftn(q) * w
        ar -= torch.fft.rfftn(q * best) * w
    grec = torch.fft.irfftn(ar, s=size) * n3
    gsrc = torch.fft.irfftn(ai, s=size) * (n3 * zeta * scale)
    gdelta, = torch.autograd.grad(rec, od, grec)
    return dict(C=best, A=None, ddelta=gdelta, dsrc=gsrc, dzeta=(gg * best).sum() / zeta)


def _sfr_box(case, cat):
    z, Nh, N = case["z"], case["N_halo"], case["N"]
    m = cat[:, 0].double()
    rate = 1.575e39 * m * (1.0 + z) ** 2.27044695 * (m / 9.367608e07) ** 0.44 * torch.exp(-((9.367608e07 / m) ** 3))
    rate = rate / 1e45 / synth.qion(z)
    pos = cat[:, 1:].double()
    cell, grid = pos.floor().long(), torch.zeros(Nh ** 3, dtype=torch.float64, device="cuda")
    frac = pos - cell
    for corner in range(8):
        at, wt = 0, rate
        for ax in range(3):
            up = (corner >> (2 - ax)) & 1
            at = at * Nh + (cell[:, ax] + up) % Nh
            wt = wt * (frac[:, ax] if up else 1.0 - frac[:, ax])
        grid.index_add_(0, at, wt)
    sm = int(round(Nh / N))
    sm -= N * sm > Nh
    grid = grid.view(Nh, Nh, Nh)[:N * sm, :N * sm, :N * sm]
    mean = grid.reshape(N, sm, N, sm, N, sm).mean(dim=(1, 3, 5))
    return mean / (case["L"] / Nh) ** 3


def _power(case, box):
    N, dl = case["N"], case["dl"]
    x = torch.arange(N, dtype=torch.float64, device="cuda")
    u = (x - (N - 1) / 2.0) / (N - 1) * 2.0
    w = {0: torch.ones_like(x), 1: 1.0 - u.abs(), 2: 1.0 - u * u}[case["window"]]
    w = w[:, None, None] * w[None, :, None] * w
    F = torch.fft.rfftn(box.double() * w)
    f, h = _axes(N)
    f = torch.where(f == -(N // 2), -f, f)
    b = torch.floor(torch.sqrt(f[:, None, None] ** 2 + f[None, :, None] ** 2 + h ** 2) + 0.5).long().reshape(-1)
    nk = int(round(math.sqrt(3.0 * (N // 2) ** 2))) + 1
    p = (F.real ** 2 + F.imag ** 2).reshape(-1)
    total = torch.zeros(nk, dtype=torch.float64, device="cuda").index_add_(0, b, p)
    count = torch.bincount(b, minlength=nk).clamp(min=1)
    return (torch.arange(nk, device="cuda") * (PI2 / (N * dl)), total / count / (w * w).sum() * dl ** 3)


def _brightness(case, b):
    N, L, z, om, ob, ol = case["N"], case["L"], case["z"], 0.27, 0.046, 0.73
    hz = lambda x: HUBBLE * 3.24078e-18 * np.sqrt(om * (1.0 + x) ** 3 + ol)  # noqa: E731

    def growth(x):
        part = lambda y: float(np.sum((1.0 + y) / (hz(y) / hz(0.0)) ** 3)) * 1e-3  # noqa: E731
        steps = 5e-4 + 1e-3 * np.arange(100000)
        return float(hz(x) / hz(0.0)) * part(x + steps) / part(steps)

    rate = -(growth(z + 5e-4) - growth(z - 5e-4)) / 1e-3 * float(hz(z)) * (1.0 + z)
    f, h = _axes(N)
    axes = [f[:, None, None] ** 2, f[None, :, None] ** 2, h ** 2]
    k2 = axes[0] + axes[1] + axes[2]
    ratio = torch.where(k2 > 0, axes[case["axis"] - 1] / k2.clamp(min=1.0), torch.zeros_like(k2))
    delta = b["delta"].double()
    dv = torch.fft.irfftn(torch.fft.rfftn(delta) * ratio, s=(N, N, N)) * (-rate / float(hz(z)) / growth(z))
    t, out = torch.ones_like(delta), []
    if case["spin"]:
        x = b["xc"].double() + b["xalpha"].double()
        tcmb = 2.725 * (1.0 + z)
        t = x / (1.0 + x) * (1.0 - tcmb / b["tempx"].double())
        out = [(tcmb / (1.0 - t)).mean()]
    pref = 0.023 * (0.7 / HUBBLE) * (ob * HUBBLE ** 2 / 0.02) * math.sqrt(0.15 / om / HUBBLE ** 2 * (1.0 + z) / 10.0)
    tb = pref * (1.0 + delta) * t / (1.0 + dv.clamp(-0.5, 1.0)) * (1.0 - b["xhii"].double())
    return [tb, tb.mean()] + out


def exact(case, seed):
    kind, N = case["kind"], case["N"]
    if kind in ("hii", "host"):
        dx = case["L"] / N
        radii = sum(len(_radii(r, dx, b)[0]) for _, r, b in _sets(case)) * len(_redshifts(case))
        if N ** 3 * radii > 6e9:  # would take too long in 64 bits
            return None
        x = torch.stack([_xhii(case, z, *_boxes(case, z, seed * 16 + i)) for i, z in enumerate(_redshifts(case))])
        if kind == "hii":
            return x
        return x[0], (1.0 - x[0]).mean(dim=(1, 2, 3))
    if kind == "grad":
        return _criterion_grad(case, *_boxes(case, case["z"], seed), _weights(N, seed))
    if kind == "halo":
        return None  # a catalogue of decisions, masses and cell positions
    if kind == "sfr":
        return _sfr_box(case, _catalogue(case, seed))
    if kind == "pk":
        return _power(case, torch.exp(_gaussian(N, seed, 0.8) - 0.32) - 1.0)
    return _brightness(case, _t21_boxes(case, seed))


# ---- what a pass cannot do without -------------------------------------------------------------
def work(case):
    kind = case["kind"]
    n3 = float(case["N"]) ** 3
    fft = 5.0 * n3 * math.log2(n3)  # one complex transform of the box
    if kind in ("hii", "host", "grad"):
        dx = case["L"] / case["N"]
        counts = [_radii(r, dx, b) for _, r, b in _sets(case)]
        if kind == "grad":
            n = counts[0][1]
            return {"bytes": n3 * (2 * 8 + 4 + 1 + 4 + 8), "flops": fft * (2 + 2 * n)}
        nz = len(_redshifts(case))
        radii = sum(len(c[0]) for c in counts)
        return {"bytes": nz * n3 * (8 + 4 * len(counts)), "flops": nz * fft * (1 + radii)}
    if kind == "halo":
        # the density in and a few percent of the cells as records; one transform per pair of some 20 masses
        return {"bytes": n3 * 8, "flops": 10 * fft}
    if kind == "sfr":
        return {"bytes": 16.0 * case["n"] + 4.0 * n3, "flops": 60.0 * case["n"]}
    if kind == "pk":
        return {"bytes": 4.0 * n3, "flops": 0.5 * fft}
    return {"bytes": n3 * 4 * (6 if case["spin"] else 3), "flops": fft}
