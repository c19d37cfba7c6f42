"""The work that users of this package have it do, at the sizes they do it: the global
orientation search in each of its forms, the local forms, refinement, reconstruction and
the proposer's training, each through the entry point of cryoim_gb300.Context that a
program calls.

A case is a dict of plain values.  `kind` names the entry point:
  search   globesearch (form "fp32") or contract_search ("bf16", "fp8", "coarse", "learned")
  local    contract_search with a local grid around each sub-particle's orientation
  refine   the descent of icosprocess mode 5
  rec      rec_begin, rec_insert, rec_finish: the symmetrised reconstruction of mode 1
  train    learn_train
Boxes, bands, grids and noise follow the repository's workloads: box 64 (its small tests),
box 128 at 2.0 A/px (band 1/60-1/10 A^-1) and box 256 at 1.5 A/px (1/50-1/6 A^-1), with the
odd sizes between them.  Inputs are made on the GPU with torch from the seed alone: a
phantom of icosahedrally placed blobs and a shell, Fourier-slice projections, CTF, origin
shift and white noise.
"""
from __future__ import annotations

import math
import os
import struct
import tempfile

import numpy as np
import torch

import cryoim_gb300 as ci

VOLT, CS, AMPWG = 300.0, 2.7, 0.07


def listed():
    return [
        # one particle of a small box against a few templates: what a script's first call costs
        dict(name="search_fp32_box64_one", kind="search", form="fp32", box=64, apix=4.0, min_r=4, max_r=22,
             step=4.0, templates=4, particles=1, snr=0.2, omax=2.0, host=True, rows=True),
        # the drop-in search at production size (it scores every view, omega and template)
        dict(name="search_fp32_box256", kind="search", form="fp32", box=256, apix=1.5, min_r=7, max_r=64, step=1.0,
             templates=20, particles=8, snr=0.1, omax=6.0, host=False),
        # the headline: learned proposals, whole batches of particles resident on the GPU
        dict(name="search_learned_box256", kind="search", form="learned", box=256, apix=1.5, min_r=7, max_r=64,
             step=1.0, templates=20, particles=512, snr=0.1, omax=6.0, host=False),
        # the judge of the proposal forms: every orientation correlated on the tensor cores
        dict(name="search_bf16_box256", kind="search", form="bf16", box=256, apix=1.5, min_r=7, max_r=64, step=1.0,
             templates=20, particles=16, snr=0.1, omax=6.0, host=False),
        # the precision form, a ragged number of particles of an intermediate box
        dict(name="search_fp8_box192", kind="search", form="fp8", box=192, apix=1.8, min_r=6, max_r=48, step=1.0,
             templates=15, particles=21, snr=0.15, omax=4.0, host=False),
        # coarse-to-fine without a trained proposer, an odd box, images on the host
        dict(name="search_coarse_box150", kind="search", form="coarse", box=150, apix=2.2, min_r=5, max_r=38,
             step=1.5, templates=12, particles=50, snr=0.2, omax=4.0, host=True),
        # localized search of vertex sub-particles around their own orientations and origins
        dict(name="local_box128", kind="local", box=128, apix=1.0, min_r=3, max_r=32, range=3.0, step=0.25,
             particles=24, snr=0.1, omax=4.0, host=False),
        # refinement of a batch after the global search
        dict(name="refine_box256", kind="refine", box=256, apix=1.5, min_r=7, max_r=64, templates=20, particles=64,
             snr=0.1, omax=6.0, host=False),
        # refinement of a handful of particles read from a file
        dict(name="refine_box100_few", kind="refine", box=100, apix=2.5, min_r=4, max_r=24, templates=7,
             particles=3, snr=0.2, omax=3.0, host=True),
        # one reconstruction from resident particles
        dict(name="rec_box256", kind="rec", box=256, apix=1.5, max_r=64, particles=512, snr=0.1, omax=6.0,
             host=False),
        # a quick map from a few particles on the host
        dict(name="rec_box90_few", kind="rec", box=90, apix=3.0, max_r=26, particles=20, snr=0.5, omax=2.0,
             host=True),
        # the proposer's training on renders of the map (forward, backward, Adam)
        dict(name="train_box128", kind="train", box=128, apix=2.0, min_r=4, max_r=26, step=1.0, samples=2048,
             batch=256, snr=0.1, omax=3.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: any kind, sizes spread over its range (odd boxes, ragged counts, steps
    that do and do not divide a turn into an even number of omegas)."""
    kind = rng.choice(["fp32", "bf16", "fp8", "coarse", "learned", "local", "refine", "refine", "rec", "rec"])
    box = 2 * round(_log(rng, 32, 128))
    apix = round(384.0 / box, 3)
    max_r = 2 * max(6, round(box * rng.uniform(0.19, 0.25) / 2))
    min_r = max(2, max_r // 9 + rng.randint(0, 2))
    c = dict(box=box, apix=apix, max_r=max_r, snr=round(_log(rng, 0.1, 0.5), 3),
             omax=float(rng.choice([2.0, 3.0, 4.0, 6.0]) if box >= 128 else 2.0), host=rng.random() < 0.4)
    if kind != "rec":
        c["min_r"] = min_r
    if kind in ("fp32", "bf16", "fp8", "coarse", "learned"):
        # 1.6: 225 omegas; the others give an even number
        c.update(kind="search", form=kind, step=rng.choice([1.0, 1.25, 1.5, 1.6, 2.0]),
                 templates=rng.randint(8, 20))
        if kind == "fp32":
            most = 8 * (64.0 / max_r) * (20.0 / c["templates"]) * c["step"] ** 3
            c["particles"] = max(1, min(96, round(_log(rng, 1, most))))
        elif kind in ("bf16", "fp8"):
            c["particles"] = max(1, min(48, round(_log(rng, 1, 16 * (64.0 / max_r) * c["step"]))))
        else:
            c["particles"] = round(_log(rng, 1, 400))
    elif kind == "local":
        c.update(kind="local", range=rng.choice([1.0, 2.0, 3.0]), step=rng.choice([0.25, 0.5]),
                 particles=round(_log(rng, 1, 16)), omax=float(rng.choice([2.0, 3.0, 4.0])), apix=1.0,
                 box=2 * round(_log(rng, 24, 64)))
        c["max_r"] = 2 * round(c["box"] / 8)
        c["min_r"] = max(2, c["max_r"] // 10)
    elif kind == "refine":
        c.update(kind="refine", templates=rng.randint(4, 20), particles=round(_log(rng, 1, 64)))
    else:
        c.update(kind="rec", particles=round(_log(rng, 1, 400)))
    return c


# ---- inputs ---------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)


def _rotations_np():
    """The 60 rotations of the icosahedral group with 2-folds on the axes and a vertex
    along (golden ratio, 1, 0), FP64."""
    g = (1 + 5 ** 0.5) / 2
    u = np.array([g, 1.0, 0.0]) / math.sqrt(g * g + 1)
    K = np.array([[0, -u[2], u[1]], [u[2], 0, -u[0]], [-u[1], u[0], 0]])
    a = 2 * math.pi / 5
    five = np.eye(3) + math.sin(a) * K + (1 - math.cos(a)) * K @ K
    gens = [five, np.diag([-1.0, -1.0, 1.0]), np.array([[0, 0, 1.0], [1, 0, 0], [0, 1, 0]])]
    ops = [np.eye(3)]
    for m in ops:
        for s in gens:
            r = s @ m
            if all(np.abs(r - o).max() > 1e-6 for o in ops):
                ops.append(r)
    return np.array(ops)


def _euler(e):
    """(..., 3) ZYZ Euler angles in degrees -> (..., 3, 3) rotations, FP64."""
    t, p, o = torch.deg2rad(e.double()).unbind(-1)
    c1, c2, c3, s1, s2, s3 = p.cos(), t.cos(), o.cos(), p.sin(), t.sin(), o.sin()
    rows = [c1 * c2 * c3 - s1 * s3, -c1 * c2 * s3 - c3 * s1, c1 * s2,
            c2 * c3 * s1 + c1 * s3, -c2 * s1 * s3 + c1 * c3, s1 * s2, -c3 * s2, s2 * s3, c2]
    return torch.stack(rows, -1).reshape(e.shape[:-1] + (3, 3))


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _random_eulers(g, n):
    """Haar-uniform orientations."""
    th = torch.rad2deg(torch.acos(_uniform(g, n, -1.0, 1.0)))
    return torch.stack([th, _uniform(g, n, -180.0, 180.0), _uniform(g, n, 0.0, 360.0)], -1)


def _blobs(n, centres, amps, sigma):
    x = torch.arange(n, device="cuda", dtype=torch.float32) - n // 2
    e = torch.exp(-(x[None, None, :] - centres.float()[:, :, None]) ** 2 / (2 * sigma * sigma))
    vol = torch.zeros(n, n, n, device="cuda")
    for i in range(0, len(centres), 60):
        ex, ey, ez = e[i:i + 60, 0], e[i:i + 60, 1], e[i:i + 60, 2] * amps.float()[i:i + 60, None]
        vol += torch.einsum("bz,by,bx->zyx", ez, ey, ex)
    return vol


def _phantom(g, n):
    """Four blobs in an asymmetric unit times the 60 rotations, and a shell."""
    s = n / 128.0
    u = torch.randn(4, 3, generator=g, device="cuda", dtype=torch.float64)
    pos = u / u.norm(dim=1, keepdim=True) * _uniform(g, 4, 40 * s, 52 * s)[:, None]
    amp = _uniform(g, 4, 0.5, 1.5)
    ops = torch.from_numpy(_rotations_np()).cuda()
    centres = torch.einsum("kij,bj->bki", ops, pos).reshape(-1, 3)
    vol = _blobs(n, centres, amp[:, None].expand(4, 60).reshape(-1), 2.5 * s)
    x = torch.arange(n, device="cuda", dtype=torch.float32) - n // 2
    r = (x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2).sqrt()
    return vol + 0.3 * ((r >= 30 * s) & (r <= 34 * s))


def _local_map(g, n):
    """A compact map without symmetry: blobs inside a sphere of 0.32 n."""
    u = torch.randn(40, 3, generator=g, device="cuda", dtype=torch.float64)
    rad = 0.32 * n * _uniform(g, 40, 0.0, 1.0) ** (1 / 3)
    return _blobs(n, u / u.norm(dim=1, keepdim=True) * rad[:, None], _uniform(g, 40, 0.5, 1.5), 0.018 * n)


def _freq(n):
    k = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
    return k[None, :].expand(n, n), k[:, None].expand(n, n)  # hx, ky


def _ctf(n, apix, df1, df2, ang):
    """Contrast transfer functions on the centred grid (defocus in um), FP64."""
    lam = 0.387818 / math.sqrt(VOLT * (1 + 0.978459e-3 * VOLT))
    hx, ky = _freq(n)
    phi = torch.atan2(ky, hx)[None] - torch.deg2rad(ang)[:, None, None]
    df = 1e4 * (df1[:, None, None] * phi.cos() ** 2 + df2[:, None, None] * phi.sin() ** 2)
    r2 = ((hx ** 2 + ky ** 2) / (n * apix) ** 2)[None]
    ph = 2 * math.pi * (-CS * 1e7 * lam ** 3 * r2 * r2 / 4 + df * lam * r2 / 2)
    return -(math.sqrt(1 - AMPWG ** 2) * ph.sin() + AMPWG * ph.cos())


class _Slicer:
    """Central sections of a map's transform, twice oversampled."""

    def __init__(self, vol):
        n = self.n = vol.shape[0]
        pad = torch.zeros(2 * n, 2 * n, 2 * n, device="cuda")
        pad[n // 2:n // 2 + n, n // 2:n // 2 + n, n // 2:n // 2 + n] = vol
        sh = (n // 2 + n // 2,) * 3  # the map's centre to index 0
        f = torch.fft.fftshift(torch.fft.fftn(torch.roll(pad, tuple(-x for x in sh), (0, 1, 2))))
        self.f = torch.view_as_real(f).permute(3, 0, 1, 2).contiguous()[None]

    def __call__(self, eulers):
        """(P, n, n) centred transforms of the projections (zero outside the Nyquist disc)."""
        n = self.n
        hx, ky = _freq(n)
        out = torch.empty(len(eulers), n, n, dtype=torch.complex64, device="cuda")
        R = _euler(eulers)
        disc = (hx ** 2 + ky ** 2) <= (n // 2 - 1) ** 2
        for i in range(0, len(eulers), 64):
            r = R[i:i + 64]
            p = r[:, None, None, :, 0] * hx[None, :, :, None] + r[:, None, None, :, 1] * ky[None, :, :, None]
            grid = ((2 * p + n) / (2 * n - 1) * 2 - 1).float()  # voxel 2 h + n of 2 n, corners aligned
            v = torch.nn.functional.grid_sample(self.f, grid[None], align_corners=True)[0]
            out[i:i + 64] = torch.complex(v[0], v[1]) * disc
        return out


def _image(F):
    return torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(F, dim=(-2, -1))), dim=(-2, -1)).real.float()


def _particles(g, sl, eulers, case, astig=0.1, origin=None):
    """CTF-modulated, shifted, noisy projections and their records (at the true origin)."""
    n, P = sl.n, len(eulers)
    df1 = _uniform(g, P, 0.8, 3.5)
    df2 = df1 + _uniform(g, P, 0.0, astig)
    ang = _uniform(g, P, 0.0, 180.0)
    om = case["omax"] if origin is None else origin
    x, y = _uniform(g, P, -om, om), _uniform(g, P, -om, om)
    hx, ky = _freq(n)
    inside = (hx ** 2 + ky ** 2) <= (0.4 * n) ** 2
    imgs = torch.empty(P, n, n, device="cuda")
    for i in range(0, P, 64):
        s = slice(i, i + 64)
        ph = -2 * math.pi / n * (hx[None] * x[s, None, None] + ky[None] * y[s, None, None])
        F = sl(eulers[s]) * torch.polar(_ctf(n, case["apix"], df1[s], df2[s], ang[s]), ph).to(torch.complex64)
        v = _image(F)
        sd = (v[:, inside].var(dim=1) / case["snr"]).sqrt()
        imgs[s] = v + sd[:, None, None] * torch.randn(v.shape, generator=g, device="cuda")
    rec = ci.particles(P)
    k = np.arange(1, P + 1)
    rec["particle_id"], rec["img_id"], rec["img_particle_id"] = k, k, k
    e = eulers.cpu().numpy()
    for f, a in (("df1", df1), ("df2", df2), ("astigang", ang), ("x", x), ("y", y)):
        rec[f] = a.cpu().numpy()
    rec["theta"], rec["phi"], rec["omega"] = e[:, 0], e[:, 1], e[:, 2]
    return imgs, rec


def _params(case):
    n, a = case["box"], case["apix"]
    return ci.default_params(n, apix=a, minRes=a * n / (case.get("min_r", 2) + 0.01),
                             maxRes=a * n / (case["max_r"] + 0.01), searchstep=case.get("step", 1.0), ampwg=AMPWG,
                             imgmask=(n // 2 - 2) * a)


def _templates(g, ctx, sl, count):
    """Templates at orientations of the searched region, noise-free, without CTF."""
    e = torch.stack([_uniform(g, count, 70.0, 90.0), _uniform(g, count, -25.0, 25.0),
                     _uniform(g, count, 0.0, 360.0)], -1)
    t = ci.templates(count)
    t["particle_id"] = np.arange(1, count + 1)
    t["theta"], t["phi"], t["omega"] = e.cpu().numpy().T
    ctx.load_templates(_image(sl(e)).cpu().numpy(), t)


def _proposer(ctx, sl, case, g):
    """Weights for the proposer that do not depend on a training run: the convolutions carry
    the polar power spectrum's positive and negative parts through, the mix takes their
    difference per radius band, and a view's template is the mean spectrum of noisy
    projections around it (so each radius weighs by what the noise leaves of it)."""
    views = ctx.learn_views()
    e0 = torch.zeros(len(views) + 1, 3, dtype=torch.float64, device="cuda")
    e0[:-1, :2] = torch.from_numpy(views).cuda()
    e0[-1] = e0[0] + torch.tensor([0.0, 0.0, 30.0], dtype=torch.float64, device="cuda")
    feat, draws = 0.0, 16
    for _ in range(draws):
        e = e0.clone()
        e[:, :2] += _uniform(g, 2 * len(e), -0.5, 0.5).reshape(-1, 2) * case["step"]
        imgs, rec = _particles(g, sl, e, case, origin=0.0)
        feat = feat + ctx.learn_features(imgs.cpu().numpy(), rec) / draws
    bands = feat.reshape(len(e), 8, 8, 128).mean(2)  # radius bands x angle
    c = [float((bands[-1] * np.roll(bands[0], sgn * round(30 * 128 / 180), axis=-1)).sum()) for sgn in (1, -1)]
    cin, cout = (1, 16, 32, 32), (16, 32, 32, 32)
    flat = []
    for i, o in zip(cin, cout):
        W = np.zeros((o, i, 3, 3), np.float32)
        W[0, 0, 1, 1] = 1.0
        W[1, min(1, i - 1), 1, 1] = -1.0 if i == 1 else 1.0
        flat += [W.ravel(), np.zeros(o, np.float32)]
    mix = np.zeros((16, 32, 8), np.float32)
    for r in range(8):
        mix[r, 0, r], mix[r, 1, r] = 1.0, -1.0
    T = np.zeros((len(views), 16, 128), np.float32)
    T[:, :8] = bands[:-1]
    T /= np.sqrt((T ** 2).sum((1, 2), keepdims=True))
    w = np.concatenate(flat + [mix.ravel(), np.zeros(16, np.float32), T.ravel()]).astype(np.float32)
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "proposer.bin")
        with open(path, "wb") as f:
            f.write(b"CRYOIMLP" + struct.pack("<iiifq", 1, len(views), 1 if c[0] >= c[1] else -1, case["step"],
                                              w.size) + w.tobytes())
        ctx.learn_load(path)


class _State:
    pass


def prepare(case, seed):
    """A context with its templates, reference map and proposer, and the particles."""
    torch.cuda.synchronize()
    s, g, n = _State(), _gen(seed), case["box"]
    s.case = case
    kind = case["kind"]
    P = case.get("particles", 0)
    s.ctx = ci.Context(0, _params(case))
    vol = _local_map(g, n) if kind == "local" else _phantom(g, n)
    if kind == "train":
        s.vol = vol.cpu().numpy()
        s.seed = int(seed) % 100003
        return s
    sl = _Slicer(vol)
    e = _random_eulers(g, P)
    s.imgs, s.parts = _particles(g, sl, e, case)
    if kind in ("search", "refine"):
        _templates(g, s.ctx, sl, case["templates"])
    if kind == "search" and case["form"] != "fp32":
        s.ctx.set_reference_map(vol.cpu().numpy())
        if case["form"] == "learned":
            _proposer(s.ctx, sl, case, g)
    if kind == "local":
        s.ctx.set_interpolation("oversampled")
        s.ctx.set_reference_map(vol.cpu().numpy())
    rng = np.random.default_rng(int(seed) & 0xFFFFFFFF)
    if kind in ("local", "refine"):  # where a search before it left them
        for f in ("theta", "phi", "omega"):
            s.parts[f] += rng.uniform(-1.0, 1.0, P)
        for f in ("x", "y"):
            s.parts[f] += rng.uniform(-0.7, 0.7, P)
        s.parts["pr"] = 60.0
    s.arg = s.imgs.cpu().numpy() if case["host"] else s.imgs.data_ptr()
    torch.cuda.synchronize()
    return s


def _records(q):
    return {f: q[f].copy() for f in ("theta", "phi", "omega", "x", "y", "pr")}


def run(s):
    case, ctx = s.case, s.ctx
    kind = case["kind"]
    if kind == "train":
        ctx.learn_train(s.vol, samples=case["samples"], batch=case["batch"], lr=2e-3, seed=s.seed, snr=case["snr"],
                        df_min=0.8, df_max=3.5, astig_max=0.1, origin_max=case["omax"])
        return ctx.learn_params()
    q = s.parts.copy()
    if kind == "rec":
        ctx.rec_begin()
        used = ctx.rec_insert(s.arg, q)
        return {"map": ctx.rec_finish(), "used": used}
    if kind == "refine":
        ctx.refine(s.arg, q)
    elif kind == "local":
        ctx.contract_search(s.arg, q, origin_max=case["omax"], origin_step=0.5, topk=16, pick=1,
                            local_range=case["range"], local_step=case["step"], centred_origins=True)
    elif case["form"] == "fp32":
        pr = ctx.globesearch(s.arg, q, want_pr_array=bool(case.get("rows")))  # rows: every score too
        return _records(q) if pr is None else dict(_records(q), rows=pr)
    else:
        opts = {"bf16": {}, "fp8": dict(precision="fp8"), "coarse": dict(coarse=16, nbr_best=4),
                "learned": dict(learned=24, nbr_best=4, proposal_nbr=1)}[case["form"]]
        ctx.contract_search(s.arg, q, origin_max=case["omax"], origin_step=0.5, topk=16, **opts)
    return _records(q)


# ---- what a pass cannot do without ------------------------------------------------------


def _views(step):
    return 664.0 / step ** 2  # directions of the asymmetric unit at this step


def work(case):
    n, kind, P = case["box"], case["kind"], case.get("particles", 0)
    R = case["max_r"]
    nr = R - case.get("min_r", 0) + 1
    img = 4.0 * n * n * P
    if kind == "train":
        # three passes (forward, data and weight gradients) of 0.4 GFLOP a projection
        return {"bytes": 4.0 * n ** 3 + 4.0 * 4e5, "flops": 1.2e9 * case["samples"]}
    if kind == "rec":
        # 60 x 8 taps of three sums for each half-plane sample
        return {"bytes": img + 4.0 * n ** 3, "flops": 6.0 * 60 * 8 * math.pi * R * R / 2 * P}
    terms = 60.0 * nr * case.get("templates", 0)  # phase-residual terms of one orientation
    if kind == "refine":
        return {"bytes": img + 96.0 * P, "flops": 30.0 * terms * 11 * 6 * P}
    S = math.pi * (R * R - case["min_r"] ** 2) / 2  # half-plane samples
    # a correlation is band-limited over the origins: its independent values lie n / 2R px
    # apart; a section turned by 180 degrees is the complex conjugate of the section
    O = (2 * case["omax"] * 2 * R / n + 1) ** 2
    if kind == "local":
        N = (2 * round(case["range"] / case["step"]) + 1) ** 3
        return {"bytes": img + 96.0 * P, "flops": 2.0 * 2 * S * O * N * P}
    N = _views(case["step"]) * int(360 / case["step"])
    if case["form"] == "fp32":
        return {"bytes": img + 96.0 * P, "flops": 30.0 * terms * N * P}
    # correlated orientations of a particle, and orientations scored by phase residual
    rows, scored = {"bf16": (N, 300), "fp8": (N, 300), "coarse": (N / 30 + 1500, 90), "learned": (900, 90)}[case["form"]]
    return {"bytes": img + 96.0 * P, "flops": (2.0 * S * O * rows + 30.0 * terms * scored) * P}


# ---- the same in 64 bits ------------------------------------------------------------------


def exact(case, seed):
    """The reconstruction in FP64.  The searches and descents return the grid point (or the
    end of a descent) of least phase residual: a term of that score counts only where both
    amplitudes reach cuts fitted to the same data, which FP32 rounding decides, so it has no
    value in 64 bits; neither has the training, whose renders add the library's own noise."""
    if case["kind"] != "rec":
        return None
    n, R, apix = case["box"], case["max_r"], case["apix"]
    g = _gen(seed)
    sl = _Slicer(_phantom(g, n))
    e = _random_eulers(g, case["particles"])
    imgs, rec = _particles(g, sl, e, case)
    del sl
    h = n // 2
    col = {f: torch.from_numpy(rec[f].astype(np.float64)).cuda() for f in
           ("x", "y", "df1", "df2", "astigang", "theta", "phi", "omega")}
    rot = _euler(torch.stack([col["theta"], col["phi"], col["omega"]], -1))
    use = (col["x"].abs() <= h - 2) & (col["y"].abs() <= h - 2)
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    # the mask sits at the first particle's origin for every image
    ra = ((k[None, :] - col["x"][0] - h) ** 2 + (k[:, None] - col["y"][0] - h) ** 2).sqrt()
    R1, R2 = max(0.0, h - 2 - 3.0), min(h - 2 + 3.0, float(h))
    ring, out = (ra > R1) & (ra <= R2), ra > R2
    edge = (1 + torch.cos(math.pi * (ra - R1) / 6)) / 2
    sign = 1.0 - 2.0 * ((k[None, :] + k[:, None]) % 2)
    hx = torch.arange(0, R + 1, device="cuda", dtype=torch.float64)[None, :].expand(2 * R + 1, R + 1)
    ky = torch.arange(-R, R + 1, device="cuda", dtype=torch.float64)[:, None].expand(2 * R + 1, R + 1)
    keep = (hx ** 2 + ky ** 2) <= R * R
    hx, ky = hx[keep], ky[keep]
    at = ((ky + h) * n + hx + h).long()
    ops = torch.from_numpy(_rotations_np()).cuda()
    D = 2 * R + 4
    acc = torch.zeros(3, D * D * D, device="cuda", dtype=torch.float64)
    for i in range(0, len(imgs), 8):
        s = slice(i, i + 8)
        v = imgs[s].double()
        v = (v - v.mean((1, 2), keepdim=True)) / v.var((1, 2), unbiased=False, keepdim=True).sqrt()
        m = v[:, ring].mean(1)[:, None, None]
        v = torch.where(ring, v * edge + (1 - edge) * m, v)
        v = torch.where(out, m.expand_as(v), v)
        f = (torch.fft.fft2(v * sign) / (n * n)).flatten(1)[:, at]
        ph = 2 * math.pi / n * ((col["x"][s, None] + h) * hx + (col["y"][s, None] + h) * ky)
        a, b = f.real, -f.imag
        a, b = a * ph.cos() + b * ph.sin(), -a * ph.sin() + b * ph.cos()
        c = _ctf(n, apix, col["df1"][s], col["df2"][s], col["astigang"][s]).flatten(1)[:, at]
        c = c * use[s, None]
        x = torch.einsum("kij,pjl,lq->pkiq", ops, rot[s][:, :, :2], torch.stack([hx, ky]))
        sg = torch.where(x[:, :, 2] < 0, -1.0, 1.0)
        x = x * sg[:, :, None]
        lo = x.floor()
        fr, lo = x - lo, (lo + R + 1).long()
        val = torch.stack([(a * c)[:, None].expand_as(sg), (b * c)[:, None] * sg, (c * c)[:, None].expand_as(sg)])
        for j in range(8):
            d = (j & 1, j >> 1 & 1, j >> 2)
            w, q = 1.0, 0
            for axis in (2, 1, 0):
                w = w * (fr[:, :, axis] if d[axis] else 1 - fr[:, :, axis])
                q = q * D + lo[:, :, axis] + d[axis]
            for u in range(3):
                acc[u].index_add_(0, q.flatten(), (val[u] * w).flatten())
    acc = acc.reshape(3, D, D, D)[:, 1:2 * R + 2, 1:2 * R + 2, 1:2 * R + 2]  # z, y, x = -R .. R
    fa, fb, wg = acc[0], acc[1], acc[2] + 0.01
    z = torch.arange(-R, R + 1, device="cuda", dtype=torch.float64)
    d2 = z[:, None, None] ** 2 + z[None, :, None] ** 2 + z[None, None, :] ** 2
    par = 1.0 - 2.0 * ((z[:, None, None] + z[None, :, None] + z[None, None, :]).abs() % 2)
    up = torch.complex(fa / wg, -fb / wg)[R + 1:]
    full = torch.zeros(2 * R + 1, 2 * R + 1, 2 * R + 1, dtype=torch.complex128, device="cuda")
    full[R + 1:] = up
    full[:R] = up.conj().flip(0, 1, 2)
    p0 = torch.complex(fa[R] + fa[R].flip(0, 1), -(fb[R] - fb[R].flip(0, 1))) / (wg[R] + wg[R].flip(0, 1))
    p0[R, R] = fa[R, R, R] / wg[R, R, R]
    full[R] = p0
    full = full * par * (d2 <= R * R)
    vol = torch.zeros(n, n, n, dtype=torch.complex128, device="cuda")
    vol[h - R:h + R + 1, h - R:h + R + 1, h - R:h + R + 1] = full
    m = torch.fft.ifftn(torch.fft.ifftshift(vol)).real * float(n) ** 3
    return {"map": m, "used": None}
