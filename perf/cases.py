"""The renders, batches, served requests, spectra and snapshot loads whose speed matters, as measurable cases.

A case is a dict of plain values.  Renders run on synthetic block-AMR snapshots with the shapes and value distributions
of GRMHD data (a torus with log-normal turbulence, a poloidal field, Keplerian rotation with perturbations; base grid in
8^3 blocks, refined around the torus), made on the GPU from the seed.  The seed also draws the camera azimuth and small
offsets of inclination and accretion rate, so two seeds are two observations of two snapshots.

FP32 and mixed renders accumulate their images in FP32 and the C ABI widens them to doubles; `run` returns those
records as the FP32 numbers they are (lossless), FP64 renders and spectra as FP64.
"""
from __future__ import annotations

import math
import os
import subprocess
import tempfile

import numpy as np
import torch

import phoenix_b200 as P

GEN = os.path.join(os.path.dirname(os.path.abspath(P.__file__)), "_build", "phx_gen_snapshot")

SPIN, HSLOPE, GAM = 0.9375, 0.25, 13.0 / 9.0
X_LO, X_HI = (math.log(1.2), 0.0, 0.0), (math.log(1000.0), math.pi, 2.0 * math.pi)
BLOCK = 8

# Rays march about 3,000 steps at a field of view of 40 M, and about 40% of the points emit; the flops of a step, an
# emitting sample and a sample-frequency are those of the reference's algorithm (bench.py).
STEPS_PER_RAY, EMITTING = 3000.0, 0.4
FLOPS_STEP, FLOPS_SAMPLE, FLOPS_FREQ = 3445.0, 870.0, 1224.0


def listed():
    return [
        # a quick look: the smallest image that is still looked at, one frequency, on a small snapshot
        dict(name="image 64 fp32", kind="image", W=64, H=64, nfreqs=1, precision="fp32", grid=64, levels=3,
             incl=10.0, freq=230e9, m_unit=1.2e18),
        # the command-line renderer's default image
        dict(name="image 200 fp32", kind="image", W=200, H=200, nfreqs=1, precision="fp32", grid=64, levels=3,
             incl=50.0, freq=230e9, m_unit=1e18),
        # a figure-quality image on a production-size snapshot (bench.py's workload), left on the device
        dict(name="device 512 fp32", kind="device", W=512, H=512, nfreqs=1, precision="fp32", grid=192, levels=3,
             incl=60.0, freq=230e9, m_unit=1.2e18),
        # the largest: a three-frequency image of optically and Faraday-thick plasma
        dict(name="image 1024 3f fp32", kind="image", W=1024, H=1024, nfreqs=3, precision="fp32", grid=192, levels=3,
             incl=60.0, freq=86e9, m_unit=1e19),
        # the mixed mode, which holds the flux error bar at every frequency
        dict(name="device 512 mixed", kind="device", W=512, H=512, nfreqs=1, precision="mixed", grid=192, levels=3,
             incl=163.0, freq=230e9, m_unit=1.2e18),
        # an odd, non-square image of three frequencies
        dict(name="device 333x217 3f mixed", kind="device", W=333, H=217, nfreqs=3, precision="mixed", grid=96,
             levels=3, incl=75.0, freq=86e9, m_unit=1e19),
        # a reference-precision image for validation
        dict(name="image 128 fp64", kind="image", W=128, H=128, nfreqs=1, precision="fp64", grid=64, levels=3,
             incl=60.0, freq=230e9, m_unit=1.2e18),
        # a frequency sweep (config key frequency_logspace) of a small image
        dict(name="device 129x96 8f fp32", kind="device", W=129, H=96, nfreqs=8, precision="fp32", grid=64, levels=2,
             incl=30.0, freq=86e9, m_unit=3e18),
        # a parameter survey: images of several sizes, cameras and accretion rates in one captured launch
        dict(name="batch 24 fp32", kind="batch", n=24, precision="fp32", grid=64, levels=3),
        # a request mix of the render server: a few images from 64^2 to 256^2, 1-4 frequencies
        dict(name="serve 8 fp32", kind="serve", n=8, precision="fp32", grid=96, levels=3),
        # the flux line of an image that stays on the device
        dict(name="spectrum 1024 4f", kind="spectrum", W=1024, H=1024, nfreqs=4),
        # reading a dump: file, decode on the GPU, resident primitives
        dict(name="load 96", kind="load", grid=96, levels=3),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["image", "device", "device", "image", "device", "batch", "serve", "spectrum", "load"])
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(4, 32), precision=rng.choice(["fp32", "fp32", "mixed"]),
                    grid=rng.choice([32, 64, 96]), levels=rng.randint(1, 3))
    if kind == "serve":
        return dict(kind=kind, n=rng.randint(2, 12), precision=rng.choice(["fp32", "fp32", "mixed"]),
                    grid=rng.choice([32, 64, 96]), levels=rng.randint(1, 3))
    if kind == "load":
        return dict(kind=kind, grid=rng.choice([32, 48, 64, 80, 96]), levels=rng.randint(1, 3))
    if kind == "spectrum":
        return dict(kind=kind, W=int(log(64, 1400)), H=int(log(64, 1400)), nfreqs=rng.randint(1, 6))
    precision = rng.choice(["fp32", "fp32", "mixed", "mixed", "fp64"])
    top = 200 if precision == "fp64" else 640
    # more than four frequencies are a frequency sweep
    nf = rng.choice([1, 1, 1, 2, 3, 4, 8] if precision == "fp32" else [1, 1, 3])
    if nf > 4:
        top = 200
    return dict(kind=kind, W=int(log(40, top)), H=int(log(40, top)), nfreqs=nf, precision=precision,
                grid=rng.choice([32, 64, 96, 192]), levels=rng.randint(1, 3), incl=rng.uniform(5.0, 175.0),
                freq=log(86e9, 345e9), m_unit=log(1e17, 1e19))


# ---- synthetic snapshots ------------------------------------------------------------------------------------------


def _leaves(grid, levels):
    """Leaf level and block index, block origins, cell sizes and the per-level leaf maps of the refined mesh."""
    ng = np.array([grid // BLOCK, grid // 2 // BLOCK, grid // 2 // BLOCK])
    lo, width = np.array(X_LO), (np.array(X_HI) - np.array(X_LO)) / ng
    idx = np.stack(np.meshgrid(*[np.arange(n) for n in ng], indexing="ij"), -1).reshape(-1, 3)
    level, index, maps = [], [], []
    for L in range(levels):
        centre = lo + (idx + 0.5) * width / 2**L
        th = centre[:, 1] + 0.5 * HSLOPE * np.sin(2.0 * centre[:, 1])
        r = np.exp(centre[:, 0])
        split = (r >= 3.5) & (r <= 25.0) & (np.abs(th - 0.5 * np.pi) < 0.55) & (L + 1 < levels)
        here = idx[~split]
        m = np.full(tuple(ng << L), -1, dtype=np.int32)
        first = sum(len(x) for x in index)
        m[here[:, 0], here[:, 1], here[:, 2]] = first + np.arange(len(here))
        maps.append(m)
        index.append(here)
        level.append(np.full(len(here), L))
        child = np.stack(np.meshgrid([0, 1], [0, 1], [0, 1], indexing="ij"), -1).reshape(1, 8, 3)
        idx = (2 * idx[split][:, None, :] + child).reshape(-1, 3)
    level, index = np.concatenate(level), np.concatenate(index)
    scale = (1.0 / 2.0**level)[:, None]
    return ng, maps, lo + index * width * scale, width / BLOCK * scale


def _torus(r, th):
    """Torus density without noise: constant angular momentum, inner edge 6 M, pressure maximum 12 M."""
    l2, r_in = 12.0, 6.0
    hmax = 0.5 / l2 - (1.0 / r_in - l2 / (2.0 * r_in * r_in))
    h = 1.0 / r - l2 / (2.0 * r * r * torch.sin(th) ** 2) - (1.0 / r_in - l2 / (2.0 * r_in * r_in))
    return torch.clamp(h / hmax, min=0.0) ** (1.0 / (GAM - 1.0)) * torch.exp(-((r / 40.0) ** 2)), hmax


def _theta(x2):
    return x2 + 0.5 * HSLOPE * torch.sin(2.0 * x2)


def _field(x1, x2):
    """B^1, B^2 (unscaled) from the curl of A_phi = max(rho - 0.2, 0)."""
    def aphi(a, b):
        return torch.clamp(_torus(torch.exp(a), _theta(b))[0] - 0.2, min=0.0)

    d, r, th = 1e-5, torch.exp(x1), _theta(x2)
    sqrtg = (r * r + (SPIN * torch.cos(th)) ** 2) * torch.sin(th) * r * (1.0 + HSLOPE * torch.cos(2.0 * x2))
    return (aphi(x1, x2 + d) - aphi(x1, x2 - d)) / (2.0 * d) / sqrtg, \
        -(aphi(x1 + d, x2) - aphi(x1 - d, x2)) / (2.0 * d) / sqrtg


def _metric(x1, x2):
    r, th = torch.exp(x1), _theta(x2)
    s2, tp = torch.sin(th) ** 2, 1.0 + HSLOPE * torch.cos(2.0 * x2)
    sig = r * r + (SPIN * torch.cos(th)) ** 2
    q = 2.0 * r / sig
    return dict(tt=q - 1.0, t3=-SPIN * s2 * q, x11=(1.0 + q) * r * r, x13=-SPIN * s2 * (1.0 + q) * r,
                x22=sig * tp * tp, x33=s2 * (sig + SPIN**2 * s2 * (1.0 + q)), shift=2.0 / sig / (1.0 + q))


def _arrays(grid, levels, seed):
    """The arguments of Snapshot.from_arrays for one synthetic snapshot (FP64 primitives beside the FP32 ones)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    ng, maps, lb, dxc = _leaves(grid, levels)
    tlb, tdx = torch.from_numpy(lb).cuda(), torch.from_numpy(dxc).cuda()
    c = torch.arange(BLOCK, device="cuda", dtype=torch.float64) + 0.5
    n = len(lb)
    x1 = (tlb[:, 0, None] + c * tdx[:, 0, None])[:, None, None, :].expand(n, BLOCK, BLOCK, BLOCK)
    x2 = (tlb[:, 1, None] + c * tdx[:, 1, None])[:, None, :, None].expand(n, BLOCK, BLOCK, BLOCK)
    r, th = torch.exp(x1), _theta(x2)

    def noise():
        return torch.randn(r.shape, generator=g, device="cuda", dtype=torch.float64)

    rt, hmax = _torus(r, th)
    kappa = (GAM - 1.0) * hmax / GAM
    rho_t = rt * torch.exp(0.5 * noise() - 0.125)
    prim = torch.empty(n, BLOCK, BLOCK, BLOCK, 8, device="cuda", dtype=torch.float64)
    prim[..., 0] = rho_t + 1e-5 * r**-1.5
    prim[..., 1] = kappa * rho_t**GAM / (GAM - 1.0) + 1e-7 * r**-2.5
    # field strength: <p_gas> / <p_mag> = 100 over the torus body, plus a weak monopole
    l1 = X_LO[0] + (torch.arange(512, device="cuda", dtype=torch.float64) + 0.5) * (X_HI[0] - X_LO[0]) / 512
    l2 = (torch.arange(256, device="cuda", dtype=torch.float64) + 0.5) * math.pi / 256
    l1, l2 = torch.meshgrid(l1, l2, indexing="ij")
    body = _torus(torch.exp(l1), _theta(l2))[0]
    b1, b2 = _field(l1, l2)
    m = _metric(l1, l2)
    on = body > 0.2
    scale = torch.sqrt((kappa * body**GAM)[on].sum() / (100.0 * (0.5 * (m["x11"] * b1 * b1 + m["x22"] * b2 * b2))[on].sum()))
    b1, b2 = _field(x1, x2)
    prim[..., 5] = b1 * scale + 0.05 / ((r * r + (SPIN * torch.cos(th)) ** 2) * r)
    prim[..., 6] = b2 * scale
    prim[..., 7] = 0.0
    # Keplerian rotation inside the torus, 10% perturbations
    m = _metric(x1, x2)
    om = 1.0 / ((r * torch.sin(th)) ** 1.5 + SPIN)
    norm = -(m["tt"] + 2.0 * m["t3"] * om + m["x33"] * om * om)
    ok = (rt > 0.0) & (norm > 0.0)
    ut = torch.where(ok, torch.rsqrt(torch.where(ok, norm, torch.ones_like(norm))), torch.zeros_like(norm))
    v1, v3 = ut * m["shift"], ut * om
    mag = torch.sqrt(torch.clamp(m["x11"] * v1 * v1 + 2.0 * m["x13"] * v1 * v3 + m["x33"] * v3 * v3, min=0.0))
    prim[..., 2] = v1 + 0.1 * mag * noise()
    prim[..., 3] = 0.1 * mag * noise()
    prim[..., 4] = v3 + 0.1 * mag * noise()
    prim = prim.reshape(n, BLOCK**3, 8)
    return dict(nx=[BLOCK] * 3, ng=[int(v) for v in ng], nlevels=levels, a=SPIN, hslope=HSLOPE, gam=GAM, x_lo=X_LO,
                x_hi=X_HI, lb=lb, dxc=dxc, level_maps=maps, prim_f32=prim.float().cpu().numpy()), prim


def _snapshot(case, seed):
    arrays, prim = _arrays(case["grid"], case["levels"], seed)
    if case["precision"] == "fp64":
        arrays["prim_f64"] = prim.cpu().numpy()
    del prim
    return P.Snapshot.from_arrays(**arrays)


# ---- what a program has in hand -----------------------------------------------------------------------------------


def _frequencies(f0, n):
    """n frequencies from f0 to 4 f0, logarithmically spaced."""
    return [f0 * 4.0 ** (k / max(1, n - 1)) for k in range(n)]


def _params(rng, W, H, nfreqs, precision, incl, freq, m_unit):
    return P.make_params(img_width=W, img_height=H, precision=precision, frequencies=_frequencies(freq, nfreqs),
                         inclination=float(np.clip(incl + rng.uniform(-1.0, 1.0), 1.0, 179.0)),
                         phi=float(rng.uniform(0.0, 360.0)), m_unit=float(m_unit * np.exp(rng.uniform(-0.05, 0.05))))


def _survey(rng, n, precision, sizes, maxfreqs):
    """n render requests: sizes, cameras, frequencies and accretion rates of a parameter survey."""
    return [_params(rng, int(rng.choice(sizes)), int(rng.choice(sizes)), int(rng.integers(1, maxfreqs + 1)), precision,
                    rng.uniform(5.0, 175.0), math.exp(rng.uniform(math.log(86e9), math.log(345e9))),
                    math.exp(rng.uniform(math.log(1e17), math.log(1e19)))) for _ in range(n)]


def _requests(case):
    """The requests of a batch or server case by size and frequency count (the same for every seed)."""
    return np.random.default_rng(1000 * case["n"] + case["grid"])


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    st = dict(case=case)
    kind = case["kind"]
    if kind in ("image", "device"):
        st["snap"] = _snapshot(case, seed)
        p = _params(rng, case["W"], case["H"], case["nfreqs"], case["precision"], case["incl"], case["freq"],
                    case["m_unit"])
        st["params"] = p
        if kind == "device":
            jobs = P.schedule_tiles(p.img_width, p.img_height, P.default_pixel_order(p))
            st["jobs"] = torch.from_numpy(jobs).cuda()
            st["res"] = torch.zeros(p.img_width, p.img_height, p.nfreqs, 6, dtype=torch.float64, device="cuda")
            st["counters"] = torch.zeros(P.NUM_COUNTERS, dtype=torch.int64, device="cuda")
    elif kind in ("batch", "serve"):
        st["snap"] = _snapshot(case, seed)
        sizes = (48, 64, 96, 128, 160, 192, 256)
        shape = _requests(case)
        ps = _survey(shape, case["n"], case["precision"], sizes, 1 if kind == "batch" else 4)
        for p in ps:
            p.phi = float(rng.uniform(0.0, 360.0))
            p.m_unit = float(p.m_unit * np.exp(rng.uniform(-0.05, 0.05)))
        st["params"] = ps
        if kind == "batch":
            st["batch"] = P.Batch([(st["snap"], p) for p in ps])
        else:
            st["server"] = P.Server([st["snap"]], case["precision"], memory_budget=4 << 30)
    elif kind == "spectrum":
        p = P.make_params(img_width=case["W"], img_height=case["H"], frequencies=_frequencies(86e9, case["nfreqs"]))
        st["params"] = p
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        # Stokes intensities and optical depths fall off by decades from the ring outward
        shape = (case["W"], case["H"], case["nfreqs"], 6)
        mag = torch.exp(2.5 * torch.randn(shape[:3] + (1,), generator=g, device="cuda", dtype=torch.float64))
        st["res"] = mag * torch.randn(shape, generator=g, device="cuda", dtype=torch.float64).abs()
        st["res"][..., 1:4] *= torch.tensor([0.1, -0.05, 0.01], dtype=torch.float64, device="cuda")
        st["spec"] = torch.zeros(case["nfreqs"], 8, dtype=torch.float64, device="cuda")
    else:
        tmp = tempfile.TemporaryDirectory(prefix="phx_case_")
        g = case["grid"]
        subprocess.check_call([GEN, "--out", tmp.name, "--seed", str(seed), "--base", str(g), str(g // 2), str(g // 2),
                               "--nlevels", str(case["levels"]), "--nws", "0", "--sfc", "0"],
                              stdout=subprocess.DEVNULL)
        st["tmp"], st["dump"], st["grid"] = tmp, os.path.join(tmp.name, "dump.dat"), os.path.join(tmp.name, "grid.in")
    return st


def _image(res, precision):
    """One image's records: Stokes vector, absorption and Faraday depth."""
    if precision != "fp64":
        res = res.float() if isinstance(res, torch.Tensor) else res.astype(np.float32)
    return dict(stokes=res[..., :4], tau=res[..., 4], tauF=res[..., 5])


def _images(results, precision):
    """Several images' records one after the other (pixel, frequency by frequency)."""
    return _image(np.concatenate([r.reshape(-1, 6) for r in results]), precision)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "image":
        res, _ = state["snap"].render(state["params"])
        return _image(res, case["precision"])
    if kind == "device":
        stream = torch.cuda.current_stream().cuda_stream
        state["counters"].zero_()
        state["snap"].render_async(state["params"], state["jobs"].data_ptr(), state["jobs"].numel(),
                                   state["res"].data_ptr(), state["counters"].data_ptr(), stream=stream)
        return _image(state["res"], case["precision"])
    if kind == "batch":
        state["batch"].run()
        return _images([state["batch"].result(i)[0] for i in range(case["n"])], case["precision"])
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(0, p) for p in state["params"]]
        for i in ids:
            srv.wait(i, 100.0)
        return _images([srv.result(i)[0] for i in ids], case["precision"])
    if kind == "spectrum":
        P.device_spectrum(state["params"], state["res"].data_ptr(), state["spec"].data_ptr(),
                          torch.cuda.current_stream().cuda_stream)
        counts = state["spec"][:, 6:].view(torch.int64)
        return dict(totals=state["spec"][:, :6], pixels=counts)
    with P.Snapshot.load(state["dump"], state["grid"], nlevels=case["levels"], sfc=False, gpu_decode=True) as snap:
        return snap.download()


# ---- what a pass cannot do without --------------------------------------------------------------------------------


def _cells(grid, levels):
    return len(_leaves(grid, levels)[2]) * BLOCK**3


def _rays(rays, nfreqs):
    return rays * STEPS_PER_RAY * (FLOPS_STEP + EMITTING * (FLOPS_SAMPLE + FLOPS_FREQ * nfreqs))


def work(case):
    kind = case["kind"]
    if kind in ("image", "device"):
        rays = case["W"] * case["H"]
        prim = 64 if case["precision"] == "fp64" else 32
        return dict(bytes=float(_cells(case["grid"], case["levels"]) * prim + rays * case["nfreqs"] * 48),
                    flops=_rays(rays, case["nfreqs"]))
    if kind in ("batch", "serve"):
        ps = _survey(_requests(case), case["n"], case["precision"], (48, 64, 96, 128, 160, 192, 256),
                     1 if kind == "batch" else 4)
        return dict(bytes=float(_cells(case["grid"], case["levels"]) * 32 +
                                sum(p.img_width * p.img_height * p.nfreqs * 48 for p in ps)),
                    flops=sum(_rays(p.img_width * p.img_height, p.nfreqs) for p in ps))
    if kind == "spectrum":
        n = case["W"] * case["H"] * case["nfreqs"]
        return dict(bytes=n * 48.0 + case["nfreqs"] * 64.0, flops=n * 8.0)
    cells = _gen_leaves(case["grid"], case["levels"])[0].shape[0] * BLOCK**3
    # a dump holds 11 doubles a cell; the decode evaluates the metric at 28 points of a cell
    return dict(bytes=cells * (88.0 + 32.0), flops=cells * 28.0 * 60.0)


# ---- 64-bit values ------------------------------------------------------------------------------------------------


def _gen_leaves(grid, levels):
    """Block origins and cell sizes of a generated dump's leaves in file order (base blocks with the first index
    fastest, children of a refined block depth first, first index fastest)."""
    ng = [grid // BLOCK, grid // 2 // BLOCK, grid // 2 // BLOCK]
    width = [(X_HI[d] - X_LO[d]) / ng[d] for d in range(3)]
    lb, dx = [], []

    def walk(L, ijk):
        w = [v / 2**L for v in width]
        r = math.exp(X_LO[0] + (ijk[0] + 0.5) * w[0])
        x2 = X_LO[1] + (ijk[1] + 0.5) * w[1]
        th = x2 + 0.5 * HSLOPE * math.sin(2.0 * x2)
        if L + 1 < levels and 4.0 <= r <= 20.0 and abs(th - 0.5 * math.pi) < 0.5:
            for ch in range(8):
                walk(L + 1, [2 * ijk[d] + ((ch >> d) & 1) for d in range(3)])
        else:
            lb.append([X_LO[d] + ijk[d] * w[d] for d in range(3)])
            dx.append([v / BLOCK for v in w])

    for k in range(ng[2]):
        for j in range(ng[1]):
            for i in range(ng[0]):
                walk(0, [i, j, k])
    return np.array(lb), np.array(dx)


def _exact_load(case, seed):
    """The dump's conserved variables turned into primitives (metric at the cell's Simpson centroid)."""
    st = prepare(case, seed)
    lb, dx = _gen_leaves(case["grid"], case["levels"])
    n, cells = len(lb), BLOCK**3
    cons = torch.from_numpy(np.fromfile(st["dump"], dtype=np.float64, count=n * 11 * cells)).cuda()
    cons = cons.reshape(n, 11, BLOCK, BLOCK, BLOCK)
    c = torch.arange(BLOCK, device="cuda", dtype=torch.float64) + 0.5
    lb, dx = torch.from_numpy(lb).cuda(), torch.from_numpy(dx).cuda()
    ctr = [lb[:, d, None] + c * dx[:, d, None] for d in range(3)]
    X1 = ctr[0][:, None, None, :].expand(n, BLOCK, BLOCK, BLOCK)
    X2 = ctr[1][:, None, :, None].expand(n, BLOCK, BLOCK, BLOCK)
    d1, d2 = dx[:, 0, None, None, None], dx[:, 1, None, None, None]
    norm, s1, s2 = 0.0, 0.0, 0.0
    for j in range(3):
        for i in range(3):
            a, b = X1 + 0.5 * d1 * (i - 1), X2 + 0.5 * d2 * (j - 1)
            m = _metric(a, b)
            w = (1.0, 4.0, 1.0)[i] * (1.0, 4.0, 1.0)[j] * torch.sqrt(m["x22"] * (m["x11"] * m["x33"] - m["x13"] ** 2))
            norm, s1, s2 = norm + w, s1 + w * a, s2 + w * b
    a, b = s1 / norm, s2 / norm
    m = _metric(a, b)
    det = m["x11"] * m["x33"] - m["x13"] ** 2
    D, S, B = cons[:, 0], cons[:, 1:4], cons[:, 5:8]
    Bd = [m["x11"] * B[:, 0] + m["x13"] * B[:, 2], m["x22"] * B[:, 1], m["x13"] * B[:, 0] + m["x33"] * B[:, 2]]
    Su = [(m["x33"] * S[:, 0] - m["x13"] * S[:, 2]) / det, S[:, 1] / m["x22"],
          (m["x11"] * S[:, 2] - m["x13"] * S[:, 0]) / det]
    Bsq = sum(Bd[d] * B[:, d] for d in range(3))
    BS = sum(S[:, d] * B[:, d] for d in range(3))
    lfac, xi = cons[:, 9], cons[:, 10]
    rho = D / lfac
    uu = (xi / lfac**2 - rho) / GAM
    entropy = cons[:, 8] / D * rho ** (GAM - 1.0) / (GAM - 1.0)
    uu = torch.where(uu < 0.0, torch.where(entropy < 0.0, torch.full_like(uu, 1e-14), entropy), uu)
    out = torch.stack([rho, uu] + [(Su[d] / (xi + Bsq) + B[:, d] * BS / (xi * (xi + Bsq))) * lfac for d in range(3)] +
                      [B[:, d] for d in range(3)], dim=-1)
    out = torch.where((torch.exp(X1) > 1.0)[..., None], out, torch.zeros_like(out))
    return out.reshape(n, cells, 8).cpu().numpy()


def exact(case, seed):
    """Spectra and decoded primitives in 64 bits.  An image has none here: about 10^4 sequential passes of some 10^3
    tensor operations take minutes."""
    if case["kind"] == "spectrum":
        st = prepare(case, seed)
        p, res = st["params"], st["res"].reshape(-1, case["nfreqs"], 6)
        length = 6.674e-8 * p.mass * 1.989e33 / 2.99792458e10**2
        dist = p.distance * 3.086e21
        omega = (p.fov_x / p.img_width * length / dist) * (p.fov_y / p.img_height * length / dist)
        totals = torch.cat([res[..., :4].sum(0) * (omega * 1e23), res[..., 4:].mean(0)], dim=1)
        return dict(totals=totals, pixels=None)
    if case["kind"] == "load":
        return _exact_load(case, seed)
    return None
