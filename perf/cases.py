"""What is timed of this library, as a user's program calls it.

Each case is one pass through public entry points on inputs made from a seed:
scans of random ellipsoids whose line integrals are computed analytically,
with Poisson counts, and phase-contrast scans of random spheres. Sizes are
those of the repository's workloads and tests, or lie in the ranges the entry
points take: detectors of 32 to 256 columns, 4 to 64 rows, tens of views to a
thousand, one frame or several.

kind            a pass
icd             Session: start from zero or FBP, k ICD iterations with their costs (as many as near
                convergence: before it, the order in which super-voxels meet shows), the image back
reconstruct     the drop-in reconstruct(): every multi-resolution stage from host arrays
batch           Batch.run() over independent uneven problems, every image back
project         forward_project() and back_project() of host arrays
fbp             set_object_fbp(): filtered back-projection and its error sinogram
warm_start      warm_start(): FBP, the network on every frame, the error sinogram
unet            UNet.forward() of one volume on the device
train           UNet.gradients(): loss and gradient of every weight for one pair
admm            PcSession: start state, one phase-retrieval iteration, its state back
descent         PcSession: start state, k steepest-descent steps, their state back
"""
from __future__ import annotations

import math

import numpy as np
import torch

import phasecon_b200 as pc
from phasecon_b200 import pcmbir, phantoms, warmstart

DEV = "cuda"


def listed():
    return [
        # the smallest scan anyone reconstructs (a test slab): launches and latency
        dict(name="icd_small", kind="icd", n=64, nz=8, views=90, frames=1, p=1.1, huber=False, start="zero", iters=10),
        # the 4-D time-interlaced workload: 8 frames of 256 x 256 x 32 from 1,024 views
        dict(name="icd_4d", kind="icd", n=256, nz=32, views=1024, frames=8, p=1.2, huber=False, start="zero", iters=12),
        # zinger-robust data term on a slab taller than 32 rows, with sizes no tile divides
        dict(name="icd_huber_tall", kind="icd", n=100, nz=38, views=150, frames=2, p=1.2, huber=True, start="fbp", iters=6),
        # the 3-D Shepp-Logan workload through the drop-in call
        dict(name="reconstruct_3d", kind="reconstruct", n=128, nz=16, views=180, frames=1, p=1.1, iters=10),
        # uneven problems in one batched launch
        dict(name="batch_uneven", kind="batch", problems=12, pick=1, iters=16),
        # both projections of a caller that drives its own algorithm
        dict(name="project_odd", kind="project", n=180, nz=18, views=141, frames=1),
        # the classical start of the 4-D workload
        dict(name="fbp_4d", kind="fbp", n=256, nz=32, views=1024, frames=8),
        # the learned start of the 4-D workload
        dict(name="warm_start_4d", kind="warm_start", n=256, nz=32, views=1024, frames=8, c=16),
        # the network alone on a small volume
        dict(name="unet_small", kind="unet", d=16, h=72, w=40, c=16),
        # one training pair of the 4-D workload's frames
        dict(name="unet_train", kind="train", d=32, h=256, w=256, c=16),
        # the phase-contrast workload: 180 views of 256 x 256, one iteration of its ADMM
        dict(name="admm_256", kind="admm", rows=256, cols=256, views=180),
        # phase retrieval on a detector that is not square
        dict(name="descent_64x512", kind="descent", rows=64, cols=512, views=21, iters=4),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: any kind, sizes over the whole range (columns and rows even, as the entry points ask)."""
    kind = rng.choice(["icd", "icd", "icd", "reconstruct", "batch", "project", "project", "fbp", "warm_start", "unet",
                       "unet", "train", "train", "admm", "admm", "descent", "descent"])
    if kind in ("icd", "reconstruct", "project", "fbp"):
        n = 2 * int(_log(rng, 16, 128.99))
        nz = 2 * int(_log(rng, 2, 32.99))
        frames = rng.choice([1, 1, 2, 3, 5, 8])
        views = int(_log(rng, 24, 128)) * frames + rng.randrange(frames)
        if frames * views * n * n * nz > 8 * 1024 * 256 * 256 * 32 // 2:
            frames, views = 1, min(views, 128)
        case = dict(kind=kind, n=n, nz=nz, views=views, frames=frames)
        if kind in ("icd", "reconstruct"):
            case.update(p=rng.choice([1.1, 1.2, 1.3]), iters=rng.choice([10, 11, 12]))
        if kind == "icd":
            case.update(huber=rng.random() < 0.3, start="fbp", iters=rng.choice([6, 7, 8]))
            if not case["huber"] and rng.random() < 0.5:
                case.update(start="zero", iters=rng.choice([12, 13, 14]))
        if kind == "reconstruct":
            case["nz"] = max(4, min(nz, 32))
        return case
    if kind == "batch":
        return dict(kind=kind, problems=rng.randrange(3, 13), pick=rng.randrange(2, 10**6), iters=rng.choice([14, 16, 18]))
    if kind == "warm_start":
        frames = rng.choice([1, 2, 3, 4])
        return dict(kind=kind, n=8 * rng.randrange(6, 33), nz=rng.choice([8, 16, 32]), frames=frames,
                    views=rng.randrange(40, 129) * frames, c=16)
    if kind in ("unet", "train"):
        return dict(kind=kind, d=8 * rng.randrange(1, 5), h=8 * int(_log(rng, 1, 32.99)), w=8 * int(_log(rng, 1, 32.99)),
                    c=rng.choice([16, 16, 16, 8]))
    size = lambda: 2 ** rng.randrange(5, 9)  # noqa: E731
    case = dict(kind=kind, rows=size(), cols=2 * size() if kind == "descent" else size(), views=int(_log(rng, 2, 90)))
    if kind == "descent":
        case.update(iters=rng.choice([2, 3, 4]))
    return case


# ------------------------------------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(gen, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64)


def _ellipsoids(gen, n, nz, count=24):
    """[count][9]: centre x, y, z, semi-axes a, b, c, in-plane angle, attenuation (per mm), growth over the scan.
    The first is the sample's body (a cylinder of the low phase), the others inclusions of the high phase."""
    e = torch.empty(count, 9, device=DEV, dtype=torch.float64)
    rad, ang = 0.36 * n * _uniform(gen, 0, 1, count).sqrt(), _uniform(gen, 0, 2 * math.pi, count)
    e[:, 0], e[:, 1] = rad * ang.cos(), rad * ang.sin()
    e[:, 2] = _uniform(gen, -0.5 * nz, 0.5 * nz, count)
    e[:, 3], e[:, 4] = _uniform(gen, 0.02 * n, 0.11 * n, count), _uniform(gen, 0.02 * n, 0.11 * n, count)
    e[:, 5] = _uniform(gen, 0.3 * nz, 1.5 * nz, count)
    e[:, 6] = _uniform(gen, 0, math.pi, count)
    e[:, 7] = _uniform(gen, 0.004, 0.015, count)
    e[:, 8] = _uniform(gen, -0.3, 0.3, count)
    e[0] = torch.tensor([0, 0, 0, 0.46 * n, 0.44 * n, 1e3 * nz, 0, 0.005, 0], dtype=torch.float64)
    return e


def _line_integrals(e, n, nz, angles, growth):
    """[view][row][column] of the ellipsoids; growth in [0, 1]: the time of each view."""
    r = torch.arange(n, device=DEV, dtype=torch.float64) + 0.5 - n / 2
    z = torch.arange(nz, device=DEV, dtype=torch.float64) + 0.5 - nz / 2
    th = torch.as_tensor(np.asarray(angles, np.float64), device=DEV)
    tm = torch.as_tensor(np.asarray(growth, np.float64), device=DEV)
    out = torch.zeros(len(th), nz, n, device=DEV)
    for x0, y0, z0, a, b, c, phi, mu, gr in e.tolist():
        s2 = (1 - ((z - z0) / c) ** 2).clamp(min=0)[None, :] * ((1 + gr * tm) ** 2)[:, None]
        m2 = s2 * ((a * torch.cos(th + phi)) ** 2 + (b * torch.sin(th + phi)) ** 2)[:, None]
        d = r[None, :] - (x0 * th.cos() - y0 * th.sin())[:, None]
        chord = (m2[:, :, None] - (d * d)[:, None, :]).clamp(min=0).sqrt()
        out += (mu * 2 * a * b * (s2 / m2.clamp(min=1e-12))[:, :, None] * chord).float()
    return out


def _volume(e, d, h, w):
    """[d][h][w]: the ellipsoids as an image."""
    ax = lambda k: torch.arange(k, device=DEV, dtype=torch.float64) + 0.5 - k / 2  # noqa: E731
    z, y, x = ax(d)[:, None, None], ax(h)[None, :, None], ax(w)[None, None, :]
    out = torch.zeros(d, h, w, device=DEV)
    for x0, y0, z0, a, b, c, phi, mu, _ in e.tolist():
        u = (x - x0) * math.cos(phi) + (y - y0) * math.sin(phi)
        v = -(x - x0) * math.sin(phi) + (y - y0) * math.cos(phi)
        out += mu * ((u / a) ** 2 + (v / b) ** 2 + ((z - z0) / c) ** 2 <= 1)
    return out


def _scan(case, seed):
    """A Problem: counts I0 e^{-Ax}, y = -log(N / I0), w = N."""
    n, nz, views, frames = case["n"], case["nz"], case["views"], case["frames"]
    gen = _gen(seed)
    if frames > 1:  # interlaced over repeated rotations, as a time-resolved scan is taken
        angles, _ = phantoms.interlaced_views(8, 256, views)
    else:
        angles, _, _ = phantoms.uniform_views(views)
    times = np.arange(views, dtype=np.float32)
    edges = np.linspace(0, views, frames + 1).astype(np.float32)
    ax = _line_integrals(_ellipsoids(gen, n, nz), n, nz, angles, times / views)
    counts = torch.poisson(2e4 * torch.exp(-ax), generator=gen).clamp(min=1)
    y = -torch.log(counts / 2e4)
    if case.get("huber"):  # zingers: a few detector pixels far off
        y = y + 3.0 * (torch.rand(y.shape, generator=gen, device=DEV) < 1e-3)
    return pc.Problem(y.cpu().numpy(), counts.cpu().numpy(), angles, times, edges, nz, n, views, frames, vox_wid=1.0,
                      rot_center=n / 2, sig_s=0.01, sig_t=0.01, c_s=1.0, c_t=1.0, convg_thresh=0.0,
                      quad_convex=0 if case.get("huber") else 1)


def _options(case):
    o = pc.default_options()
    o.mrf_p = case.get("p", 1.2)
    return o


def _pinned(*shape):
    return torch.empty(*shape, dtype=torch.float32, pin_memory=True)


def _session(case, seed):
    stream = torch.cuda.Stream()
    pb = _scan(case, seed)
    s = pc.Session(pb, options=_options(case), stream=stream.cuda_stream)
    return dict(case=case, stream=stream, pb=pb, s=s, out=_pinned(*s.shape).numpy())


def _batch_sizes(case):
    rng = np.random.default_rng(case["pick"])
    return [dict(n=int(rng.choice([64, 96, 128, 192, 256])), nz=2 * int(rng.integers(4, 17)),
                 views=int(rng.integers(90, 361)), frames=1) for _ in range(case["problems"])]


def _channels(c):
    C = [c, 2 * c, 4 * c, 8 * c]
    convs = []
    for l in range(4):
        convs += [(1 if l == 0 else C[l - 1], C[l]), (C[l], C[l])]
    for l in (2, 1, 0):
        convs += [(C[l + 1], C[l]), (2 * C[l], C[l]), (C[l], C[l])]
    return convs


def _net_params(case, seed):
    """Flat weights as the library lays them out: per convolution w[27][cin][cout], b[cout]; the head's w[c], b."""
    rng = np.random.default_rng(seed)
    parts = []
    for cin, cout in _channels(case["c"]):
        parts += [rng.normal(0, math.sqrt(2 / (27 * cin)), 27 * cin * cout), rng.normal(0, 0.02, cout)]
    parts += [rng.normal(0, 0.05, case["c"]), [0.005]]
    return np.concatenate(parts).astype(np.float32)


SCALE = 50.0  # images of up to 0.02 per mm: the network sees values of order one


def _net(case, seed):
    net = warmstart.UNet(case["c"])
    net.set_params(_net_params(case, seed))
    net.input_scale = SCALE
    return net


def _pair(case, seed):
    """A noisy image, as filtered back-projection gives it, and the clean one."""
    gen = _gen(seed)
    t = _volume(_ellipsoids(gen, min(case["h"], case["w"]), case["d"]), case["d"], case["h"], case["w"])
    return t + 0.002 * torch.randn(t.shape, generator=gen, device=DEV), t


WAVELENGTH = 4.135668e-19 * 299792458e6 / 20.0  # um at 20 keV
DISTANCE = 5e4                                   # um
DELTA_BETA = 100.0


def _freq2(rows, cols):
    u = torch.fft.fftfreq(cols, dtype=torch.float64, device=DEV)[:, None]
    v = torch.fft.fftfreq(rows, dtype=torch.float64, device=DEV)[None, :]
    return u * u + v * v


def _pc_scan(case, seed):
    """(intensities [view][row][col], z start (zr, zi) [view][col][row]): random spheres of complex refractive
    index, Fresnel propagation, Gaussian noise at SNR 100; the start is single-material retrieval's."""
    V, R, C = case["views"], case["cols"], case["rows"]
    gen = _gen(seed)
    k = 2 * math.pi / WAVELENGTH
    n = min(R, C)
    rad = _uniform(gen, 0.02 * n, 0.15 * n, 40)
    ctr = _uniform(gen, -0.34, 0.34, 40, 3) * torch.tensor([n, R, C], device=DEV, dtype=torch.float64)
    beta = _uniform(gen, 1e-9, 5e-9, 40)
    th = torch.arange(V, device=DEV, dtype=torch.float64) * math.pi / V
    a = torch.arange(R, device=DEV, dtype=torch.float64) + 0.5 - R / 2
    b = torch.arange(C, device=DEV, dtype=torch.float64) + 0.5 - C / 2
    zr = torch.zeros(V, R, C, device=DEV, dtype=torch.float64)
    for s, (cx, cy, cz) in enumerate(ctr.tolist()):
        d2 = (a[None, :] - (cy * th.cos() - cx * th.sin())[:, None]).square()[:, :, None] + (b - cz).square()[None, None, :]
        zr += k * beta[s] * 2 * (rad[s] ** 2 - d2).clamp(min=0).sqrt()
    q = _freq2(C, R)
    w = torch.polar(torch.exp(-zr), -DELTA_BETA * zr)
    inten = torch.fft.ifft2(torch.fft.fft2(w) * torch.polar(torch.ones_like(q), -math.pi * WAVELENGTH * DISTANCE * q)).abs() ** 2
    inten = (inten * (1 + 0.01 * torch.randn(inten.shape, generator=gen, device=DEV, dtype=torch.float64))).clamp(min=1e-6) * 1e4
    meas = inten.float()
    low = 1 + DISTANCE * DELTA_BETA / (2 * k) * 4 * math.pi ** 2 * q
    zs = -0.5 * torch.log(torch.fft.ifft2(torch.fft.fft2(meas.double() / 1e4) / low).real.abs())
    return meas.transpose(1, 2).contiguous(), zs.float(), (DELTA_BETA * zs).float()


def _pc_state(case, seed):
    meas, zr, zi = _pc_scan(case, seed)
    V, C, R = meas.shape
    pb = pcmbir.PcProblem(measurements=meas.cpu().numpy(), brights=np.full((C, R), 1e4, np.float32), vox_wid=1.0,
                          mag_sig_s=0.05, mag_c_s=1.0, phase_sig_s=0.05, phase_c_s=1.0, obj2det_dist=DISTANCE,
                          light_energy=20.0, pag_regparam=DELTA_BETA)
    stream = torch.cuda.Stream()
    s = pcmbir.PcSession(pb, pcmbir.default_options(pret_max_iter=1), stream=stream.cuda_stream)
    st = dict(case=case, stream=stream, s=s)
    for name, v in (("zr0", zr), ("zi0", zi)):
        st[name] = _pinned(V, R, C)
        st[name].copy_(v)
    st.update(zr=_pinned(V, R, C), zi=_pinned(V, R, C), w=_pinned(V, R, C, 2), omega=_pinned(V, R, C, 2))
    return st


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("icd", "fbp"):
        return _session(case, seed)
    if kind == "reconstruct":
        return dict(case=case, pb=_scan(case, seed))
    if kind == "batch":
        o = _options(case)
        o.sv_size, o.cta_warps, o.sv_colors = 8, 4, 2  # a schedule that does not depend on timing
        stream = torch.cuda.Stream()
        pbs = [_scan(c, seed * 100 + i) for i, c in enumerate(_batch_sizes(case))]
        return dict(case=case, stream=stream, b=pc.Batch(pbs, options=o, stream=stream.cuda_stream))
    if kind == "project":
        st = _session(case, seed)
        gen = _gen(seed + 1)
        x = _volume(_ellipsoids(gen, case["n"], case["nz"]), case["nz"], case["n"], case["n"])
        st["x"] = x.cpu().numpy()[None].repeat(case["frames"], 0)
        st["sino"] = np.ascontiguousarray(st["pb"].projections.transpose(0, 2, 1))
        return st
    if kind == "warm_start":
        return dict(_session(case, seed), net=_net(case, seed))
    if kind in ("unet", "train"):
        x, t = _pair(case, seed)
        return dict(case=case, net=_net(case, seed), x=x, t=t)
    return _pc_state(case, seed)


# ------------------------------------------------------------------------------------------------ one pass

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "icd":
        s = st["s"]
        if case["start"] == "zero":
            s.set_object_zero()
        else:
            s.set_object_fbp()
        costs, _ = s.run(case["iters"])
        return dict(object=s.get_object(st["out"]), cost=float(costs[-1]))
    if kind == "reconstruct":
        pb = st["pb"]
        pc.set_options(mrf_p=case["p"], write_files=0, max_iterations=case["iters"])
        return pc.reconstruct(pb.projections, pb.weights, pb.proj_angles, pb.proj_times, pb.recon_times, pb.proj_rows,
                              pb.proj_cols, pb.proj_num, pb.recon_num, pb.vox_wid, pb.rot_center, pb.sig_s, pb.sig_t,
                              pb.c_s, pb.c_t, pb.convg_thresh)
    if kind == "batch":
        st["b"].run(case["iters"])
        return [st["b"].get_object(i) for i in range(case["problems"])]
    if kind == "project":
        return dict(sino=st["s"].forward_project(st["x"]), image=st["s"].back_project(st["sino"]))
    if kind == "fbp":
        st["s"].set_object_fbp()
        return dict(object=st["s"].get_object(st["out"]), cost=list(st["s"].cost()))
    if kind == "warm_start":
        warmstart.warm_start(st["s"], st["net"])
        return dict(object=st["s"].get_object(st["out"]), cost=list(st["s"].cost()))
    if kind == "unet":
        return st["net"].forward(st["x"])
    if kind == "train":
        loss, grads = st["net"].gradients(st["x"], st["t"])
        return dict(loss=loss, grads=grads)
    s, ptr = st["s"], lambda k: st[k].data_ptr()  # noqa: E731
    s.set_z(st["zr0"].numpy(), st["zi0"].numpy())
    s.init_admm()
    if kind == "admm":
        s.run()
        pcmbir.lib().mbirgpu_pc_get_state(s.h, ptr("zr"), ptr("zi"), ptr("w"), None, None)
        return dict(zr=st["zr"], zi=st["zi"], w=st["w"])
    for _ in range(case["iters"]):
        s.sd_step()
    pcmbir.lib().mbirgpu_pc_get_state(s.h, None, None, ptr("w"), None, ptr("omega"))
    return dict(w=st["w"], omega=st["omega"])


# ------------------------------------------------------------------------------------------------ what a pass needs

def _tomo_work(case, iters):
    """One visit of every A entry (2.27 per column and view inside the circle) and slice each iteration: theta and the
    update, the 28 prior terms of every voxel; the entries, e, w and x move once an iteration."""
    n, nz, views, frames = case["n"], case["nz"], case["views"], case["frames"]
    cols = 0.785 * n * n
    nnz = 2.27 * views * cols
    sino, vox = views * n * nz, frames * cols * nz
    return dict(bytes=iters * (4 * nnz + 12 * sino + 8 * vox) + 8 * sino, flops=iters * (nnz * nz * 8 + vox * 28 * 10))


def _net_flops(case, voxels):
    v, total = float(voxels), 0.0
    level = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 2, 1, 1, 1, 0, 0, 0]
    for (cin, cout), l in zip(_channels(case["c"]), level):
        total += 2 * 27 * cin * cout * v / 8 ** l
    return total


def work(case):
    kind = case["kind"]
    if kind == "icd":
        # from the second iteration the non-homogeneous passes visit about as many columns again
        return _tomo_work(case, 2 * case["iters"] - 1)
    if kind == "reconstruct":
        return _tomo_work(case, 2 * case["iters"] - 1)
    if kind == "batch":
        parts = [_tomo_work(c, case["iters"]) for c in _batch_sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind in ("project", "fbp", "warm_start"):
        n, nz, views, frames = case["n"], case["nz"], case["views"], case["frames"]
        nnz, sino, vox = 2.27 * views * n * n, views * n * nz, frames * n * n * nz
        w = dict(bytes=2 * 4 * nnz + 4 * 4 * sino + 4 * 4 * vox, flops=2 * 2 * nnz * nz)
        if kind == "warm_start":
            w["flops"] += _net_flops(case, vox)
        return w
    if kind in ("unet", "train"):
        vox = case["d"] * case["h"] * case["w"]
        f = _net_flops(case, vox)
        if kind == "unet":
            return dict(bytes=8 * vox + 2 * 90 * case["c"] ** 2 * 27, flops=f)
        return dict(bytes=8 * vox + 6 * 90 * case["c"] ** 2 * 27, flops=3 * f)
    px = case["views"] * case["rows"] * case["cols"]
    fft = 2 * 5 * math.log2(case["rows"] * case["cols"])  # forward and inverse, per pixel
    if kind == "descent":
        # five transforms a step; z in, w and omega out
        return dict(bytes=px * (8 + 16 + case["iters"] * 5 * 16), flops=px * case["iters"] * 5 * fft)
    # a search of about 20 iterations of two costs of eight neighbours each, and about 8 descent steps
    return dict(bytes=px * (8 + 16 + 8 * 5 * 16), flops=px * (20 * 2 * 8 * 25 + 8 * 5 * fft))


# ------------------------------------------------------------------------------------------------ in 64 bits

def _response(angle):
    """The detector's response to a voxel of unit width (64 bins): its trapezoidal profile at this angle, seen through
    a Hamming beam of one detector pixel."""
    off = (1 / math.sqrt(2) + 0.5) / 64
    a = angle
    while a > math.pi / 2:
        a -= math.pi / 2
    while a < 0:
        a += math.pi / 2
    peak = 1 / math.cos(a) if a <= math.pi / 4 else 1 / math.cos(math.pi / 2 - a)
    d1 = math.cos(math.pi / 4) * math.cos(math.pi / 4 - a)
    d2 = math.cos(math.pi / 4) * abs(math.cos(math.pi / 4 + a))
    t = 2.0 * np.arange(1536) / 1536
    with np.errstate(divide="ignore", invalid="ignore"):
        prof = np.where(t > 1 + d2, peak * (1 + d1 - t) / (d1 - d2), np.where(t >= 1 - d2, peak, peak * (t - 1 + d1) / (d1 - d2)))
    prof[(t <= 1 - d1) | (t >= 1 + d1)] = 0
    beam = 0.54 - 0.46 * np.cos(2 * math.pi / 512 * np.arange(512))
    beam /= beam.sum()
    r = -0.5 + np.arange(512) / 512
    idx = np.floor((r[None, :] - (np.arange(64)[:, None] * off - 1)) * (1536 / 2)).astype(int)
    ok = (idx >= 0) & (idx < 1536)
    return np.append((np.where(ok, prof[idx.clip(0, 1535)], 0) * beam).sum(1), 0.0), off


def _columns(case, angle):
    """Detector channels [3][n n] and A values of every voxel column at one view."""
    n = case["n"]
    h, off = _response(float(angle))
    h = torch.as_tensor(h, device=DEV)
    c = torch.arange(n, device=DEV, dtype=torch.float64) + 0.5 - n / 2
    r = (c[None, :] * math.cos(float(angle)) - c[:, None] * math.sin(float(angle))).reshape(-1)
    j = torch.floor(r - 1 + n / 2)[None, :] + torch.arange(3, device=DEV, dtype=torch.float64)[:, None]
    d = (r[None, :] - (j + 0.5 - n / 2)).abs()
    b = torch.floor(d / off)
    ok = (b < 64) & (j >= 0) & (j < n)
    w1 = d - b * off
    b = b.clamp(0, 63).long()
    a = ((off - w1) * h[b] + w1 * h[b + 1]) / off
    return torch.where(ok, j, 0).long(), torch.where(ok, a, 0)


def _frame_views(pb):
    return [[i for i in range(pb.proj_num) if pb.recon_times[f] <= pb.proj_times[i] < pb.recon_times[f + 1]]
            for f in range(pb.recon_num)]


def _forward64(case, pb, x):
    """[view][column][row] of images x [frame][z][y][x]."""
    n, nz = case["n"], case["nz"]
    out = torch.zeros(pb.proj_num, n, nz, device=DEV, dtype=torch.float64)
    for f, views in enumerate(_frame_views(pb)):
        cols = x[f].reshape(nz, n * n).t().contiguous()
        for v in views:
            j, a = _columns(case, pb.proj_angles[v])
            for q in range(3):
                out[v].index_add_(0, j[q], a[q][:, None] * cols)
    return out


def _back64(case, pb, sino):
    """[frame][z][y][x] of a sinogram [view][column][row]."""
    n, nz = case["n"], case["nz"]
    out = torch.zeros(pb.recon_num, n * n, nz, device=DEV, dtype=torch.float64)
    for f, views in enumerate(_frame_views(pb)):
        for v in views:
            j, a = _columns(case, pb.proj_angles[v])
            for q in range(3):
                out[f] += a[q][:, None] * sino[v][j[q]]
    return out.transpose(1, 2).reshape(pb.recon_num, nz, n, n)


def _fbp64(case, pb):
    n = case["n"]
    y = torch.as_tensor(pb.projections, device=DEV).double().transpose(1, 2)  # [view][column][row]
    k = torch.arange(n, device=DEV)
    d = k[:, None] - k[None, :]
    h = torch.where(d == 0, 0.25, torch.where(d % 2 != 0, -1 / (math.pi * d.double().abs().clamp(min=1)) ** 2, 0.0))
    x = _back64(case, pb, h @ y)
    views = torch.tensor([len(v) for v in _frame_views(pb)], device=DEV, dtype=torch.float64)
    return x * (math.pi / views)[:, None, None, None]


def _circle(case):
    c = torch.arange(case["n"], device=DEV, dtype=torch.float64) + 0.5 - case["n"] / 2
    return c[:, None] ** 2 + c[None, :] ** 2 < (case["n"] / 2) ** 2


def _conv64(x, w, b):
    """3x3x3 convolution of x [d][h][w][cin] with zero padding, and ReLU."""
    D, H, W, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    out = b.expand(D, H, W, -1)
    for t in range(27):
        z, y, k = t // 9, t // 3 % 3, t % 3
        out = out + p[z:z + D, y:y + H, k:k + W] @ w[t]
    return out.relu()


def _net64(case, flat, x):
    """The network on x [d][h][w]; flat: its weights, 64-bit."""
    from torch.utils.checkpoint import checkpoint
    layers, o = [], 0
    for cin, cout in _channels(case["c"]):
        w = flat[o:o + 27 * cin * cout].reshape(27, cin, cout)
        o += 27 * cin * cout
        layers.append((w, flat[o:o + cout]))
        o += cout
    it = iter(layers)
    conv = (lambda v: checkpoint(_conv64, v, *next(it), use_reentrant=False)) if flat.requires_grad else (lambda v: _conv64(v, *next(it)))
    y, skips = (SCALE * x)[..., None], []
    for l in range(4):
        y = conv(conv(y))
        if l < 3:
            skips.append(y)
            D, H, W, C = y.shape
            y = y.reshape(D // 2, 2, H // 2, 2, W // 2, 2, C).amax(dim=(1, 3, 5))
    for l in (2, 1, 0):
        y = y.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)
        y = conv(conv(torch.cat([conv(y), skips[l]], -1)))
    return x + (y @ flat[o:o + case["c"]] + flat[o + case["c"]]) / SCALE


def _descent64(case, seed):
    meas, zr, zi = _pc_scan(case, seed)
    V, C, R = meas.shape
    y = (meas.double() / 1e4).sqrt().transpose(1, 2)
    q = _freq2(C, R)
    sigma2 = 4.0 / (WAVELENGTH * DISTANCE)
    fwd = torch.polar(torch.exp(-q / (2 * sigma2)), -math.pi * WAVELENGTH * DISTANCE * q)
    adj = torch.polar(torch.ones_like(q), math.pi * WAVELENGTH * DISTANCE * q)
    H = lambda v: torch.fft.ifft2(torch.fft.fft2(v) * fwd)  # noqa: E731
    Ha = lambda v: torch.fft.ifft2(torch.fft.fft2(v) * adj)  # noqa: E731
    total = lambda v: v.sum(dim=(1, 2))  # noqa: E731
    w = torch.polar(torch.exp(-zr.double()), -zi.double())
    buf, nu = w, 0.5
    phase = lambda v: v.conj() / v.abs()  # noqa: E731
    om = phase(H(w))
    for _ in range(case["iters"]):
        g = Ha(om.conj() * (om * H(w) - y)) + nu * (w - buf)
        gg = total(g.abs() ** 2)
        alpha = gg / (total((g.conj() * Ha(om.conj() * om * H(g))).real) + nu * gg)
        w = w - alpha[:, None, None] * g
        om = phase(H(w))
    return dict(w=torch.view_as_real(w), omega=torch.view_as_real(om))


def exact(case, seed):
    kind = case["kind"]
    if kind == "project":
        pb = _scan(case, seed)
        x = _volume(_ellipsoids(_gen(seed + 1), case["n"], case["nz"]), case["nz"], case["n"], case["n"]).double()
        sino = torch.as_tensor(pb.projections, device=DEV).double().transpose(1, 2)
        return dict(sino=_forward64(case, pb, x[None].expand(case["frames"], -1, -1, -1)), image=_back64(case, pb, sino))
    if kind in ("fbp", "warm_start"):
        pb = _scan(case, seed)
        x = _fbp64(case, pb)
        if kind == "warm_start":
            flat = torch.as_tensor(_net_params(case, seed), device=DEV).double()
            x = torch.stack([_net64(case, flat, f) for f in x])
        return dict(object=x * _circle(case), cost=None)
    if kind in ("unet", "train"):
        x, t = _pair(case, seed)
        flat = torch.as_tensor(_net_params(case, seed), device=DEV).double().requires_grad_(kind == "train")
        out = _net64(case, flat, x.double())
        if kind == "unet":
            return out
        loss = (out - t.double()).square().mean()
        loss.backward()
        return dict(loss=loss.detach(), grads=flat.grad)
    if kind == "descent":
        return _descent64(case, seed)
    # ICD images depend on the order of the updates, and the proximal search on where it stops: no value of their own
    return None
