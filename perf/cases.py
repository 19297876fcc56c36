"""Performance cases: the calls a user of the orientation-search framework makes, over their real sizes.

``listed()`` names the cases that are timed by default, ``draw(rng)`` gives another one of the same
ranges.  ``prepare(case, seed)`` makes a case's inputs on the GPU from the seed alone, with torch and
numpy only, and the handles a user's program keeps; ``run(state)`` is one pass through the public entry
points; ``exact(case, seed)`` is what that pass returns, evaluated by torch in 64 bits; ``work(case)`` is
what the pass cannot do without.

Kinds of case:

* ``rotate``     one volume rotated, shifted and interpolated (``Interpolator``)
* ``fft``        a forward and an inverse 3-D real transform (``FourierTransformer``)
* ``spectra``    weighted particle spectra and energies of a batch (``particle_spectra``)
* ``align``      the orientation search: particles x orientations, boxes 64, 96 and 128 (``Search``)
* ``refine``     CC and pose gradient of a batch, one step of the refinement (``refine.BatchObjective``)
* ``tsearch``    template search over a tomogram (``TemplateSearch``)
* ``normalize``  local normalisation of a tomogram before that search (``local_normalize``)
* ``average``    half-set sums of a batch of windows with their wedge weights (``Average``)
* ``sf3d``       per-particle 3-D sampling weights from the tilt table (``sf3d_particles``)
"""
import math

import numpy as np
import torch

from emclarity_b200 import api, refine

# Edges with an FFT plan that tomograms, windows and tilt images are padded to (2, 3, 5, 7 and 13).
EDGES = (48, 64, 72, 80, 84, 90, 96, 108, 112, 120, 126, 128, 144, 160, 162, 168, 180, 192, 216, 224, 240, 252, 256,
         270, 288, 320, 324, 336, 360, 378, 384, 400, 416, 432, 448, 480, 486, 504, 512)


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: an interactive rotation of one 64^3 reference (mexXform3d's texture mode)
        dict(name="rotate_64", kind="rotate", n=64, interp="linear_border", store="f32", symmetry=1),
        # mexFFT on a sub-tomogram whose edges are ordinary padded sizes, both directions
        dict(name="fft_ragged", kind="fft", nx=216, ny=180, nz=168),
        # spectra of a batch of 64^3 particles with their weights, before every alignment cycle
        dict(name="spectra_64", kind="spectra", n=64, count=256, weights=True),
        # one particle against a 10 degree grid: the single-subtomogram search
        dict(name="align_plain_64", kind="align", n64=1, n96=0, n128=0, orients=540, step=10.0, store="f32", peaks=True),
        # an alignment cycle: 64^3 particles, each a local search around its prior
        dict(name="align_batch_64", kind="align", n64=64, n96=0, n128=0, orients=256, step=2.0, store="f32",
             peaks=False),
        # the same over particles of uneven boxes, 60 / 30 / 10 %
        dict(name="align_uneven", kind="align", n64=36, n96=18, n128=6, orients=256, step=2.0, store="f32",
             peaks=False),
        # 96^3 particles with the reference kept in BF16
        dict(name="align_96_bf16", kind="align", n64=0, n96=12, n128=0, orients=256, step=2.0, store="bf16",
             peaks=False),
        # one step of the gradient refinement over 100 particles of 96^3
        dict(name="refine_96", kind="refine", n=96, items=100),
        # template matching in a 512 x 512 x 256 tomogram: a dozen of the grid's orientations
        dict(name="tsearch_512", kind="tsearch", nx=512, ny=512, nz=256, t=48, orients=12),
        # the same tomogram's local normalisation, feature size 16
        dict(name="normalize_512", kind="normalize", nx=512, ny=512, nz=256, feature=16),
        # half-set averages of 512 windows of 64^3, eight tilt groups' wedge weights
        dict(name="average_64", kind="average", n=64, count=512, symmetry=1),
        # the sampling weights of 128 particle positions, 41 tilts
        dict(name="sf3d_64", kind="sf3d", n=64, count=128, tilts=41),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edges(rng, lo, hi):
    return rng.choice([e for e in EDGES if lo <= e <= hi])


def draw(rng):
    kind = rng.choice(["rotate", "fft", "spectra", "align", "align", "align", "refine", "tsearch", "normalize",
                       "average", "sf3d"])
    if kind == "rotate":
        return dict(kind=kind, n=_log_int(rng, 24, 200), interp=rng.choice(["linear", "linear_border", "cubic"]),
                    store=rng.choice(["f32", "bf16"]), symmetry=rng.choice([1, 1, 2, 4]))
    if kind == "fft":
        return dict(kind=kind, nx=_edges(rng, 48, 384), ny=_edges(rng, 48, 384), nz=_edges(rng, 48, 384))
    if kind == "spectra":
        n = _edges(rng, 48, 144)
        return dict(kind=kind, n=n, count=max(1, min(_log_int(rng, 1, 400), 1200 * 40 ** 3 // n ** 3)),
                    weights=rng.random() < 0.7)
    if kind == "align":
        mix = rng.choice(["64", "96", "128", "all"])
        few = rng.random() < 0.4  # a few particles with a wide grid, or a batch with a local one
        orients = rng.randrange(300, 700) if few else rng.randrange(60, 300)
        most = 3 if few else 20
        return dict(kind=kind, n64=rng.randrange(1, 2 * most) if mix in ("64", "all") else 0,
                    n96=rng.randrange(1, 2 + most // 2) if mix in ("96", "all") else 0,
                    n128=rng.randrange(1, 2 + most // 6) if mix in ("128", "all") else 0, orients=orients,
                    step=10.0 if few else 2.0, store=rng.choice(["f32", "f32", "bf16"]), peaks=False)
    if kind == "refine":
        return dict(kind=kind, n=rng.choice([64, 96, 128]), items=_log_int(rng, 1, 120))
    if kind == "tsearch":
        nx, ny, nz = _edges(rng, 160, 512), _edges(rng, 160, 512), _edges(rng, 96, 256)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, t=rng.randrange(20, 65), orients=rng.randrange(3, 13))
    if kind == "normalize":
        return dict(kind=kind, nx=_log_int(rng, 96, 512), ny=_log_int(rng, 96, 512), nz=_log_int(rng, 64, 256),
                    feature=rng.randrange(5, 41))
    if kind == "average":
        n = rng.randrange(32, 97)
        return dict(kind=kind, n=n, count=max(4, min(_log_int(rng, 8, 600), 512 * 64 ** 3 // n ** 3)),
                    symmetry=rng.choice([1, 1, 2, 4]))
    n = rng.randrange(32, 97)
    return dict(kind=kind, n=n, count=max(1, min(_log_int(rng, 1, 160), 128 * 64 ** 3 // n ** 3)),
                tilts=rng.randrange(21, 62))


# --------------------------------------------------------------------------- geometry
def _matrix(angles):
    """Rz(a1) Rx(a2) Rz(a3) of an angle triple in degrees (BH_defineMatrix 'inv'), 64 bits."""
    a1, a2, a3 = (math.radians(float(v)) for v in angles)

    def rz(a):
        return np.array([[math.cos(a), -math.sin(a), 0.0], [math.sin(a), math.cos(a), 0.0], [0.0, 0.0, 1.0]])

    rx = np.array([[1.0, 0.0, 0.0], [0.0, math.cos(a2), -math.sin(a2)], [0.0, math.sin(a2), math.cos(a2)]])
    return rz(a1) @ rx @ rz(a3)


def _random_angles(rng):
    return [rng.uniform(0, 360), rng.uniform(0, 180), rng.uniform(-180, 180)]


def _grid(count, step):
    """(phi, theta, psi) triples of a cone search in `step` degrees, the `count` nearest to the identity."""
    out = []
    for theta in np.arange(0.0, 4 * step + 1e-9, step):
        turns = 1 if theta == 0 else max(1, round(360.0 * math.sin(math.radians(theta)) / step))
        for k in range(turns):
            for psi in np.arange(-4 * step, 4 * step + 1e-9, step):
                out.append((360.0 * k / turns, float(theta), float(psi)))
    while len(out) < count:  # a wider request repeats the cone at half a step in psi
        out += [(p, t, s + 0.5 * step) for p, t, s in out]
    turn = [math.acos(max(-1.0, min(1.0, (np.trace(_matrix([p, t, s - p])) - 1) / 2))) for p, t, s in out]
    keep = np.sort(np.argsort(np.round(turn, 9), kind="stable")[:count])
    return np.array(out)[keep]


def _points(shape, m, shift, forward, dtype):
    """Sample points (x, y, z) of every voxel of a (nz, ny, nx) volume under matrix m (rows)."""
    nz, ny, nx = shape
    z, y, x = torch.meshgrid(*[torch.arange(n, device="cuda", dtype=dtype) - n // 2 for n in (nz, ny, nx)],
                             indexing="ij")
    u = [x, y, z]
    if forward:
        u = [a - float(t) for a, t in zip(u, shift)]
    s = [float(m[i][0]) * u[0] + float(m[i][1]) * u[1] + float(m[i][2]) * u[2] for i in range(3)]
    if not forward:
        s = [a + float(t) for a, t in zip(s, shift)]
    return [a + n // 2 for a, n in zip(s, (nx, ny, nz))]


def _sample(vol, pts, interp="linear"):
    """Trilinear ('linear': zero outside [0, n - 1]; 'linear_border': zero voxels around the volume) or
    Catmull-Rom tricubic ('cubic') value of vol (nz, ny, nx) at pts, in vol's precision."""
    nz, ny, nx = vol.shape
    dims = (nx, ny, nz)
    base = [torch.floor(p) for p in pts]
    frac = [p - b for p, b in zip(pts, base)]
    base = [b.long() for b in base]
    flat = vol.reshape(-1)
    if interp == "cubic":
        offs = (-1, 0, 1, 2)
        wts = [[0.5 * (-t ** 3 + 2 * t ** 2 - t), 0.5 * (3 * t ** 3 - 5 * t ** 2 + 2),
                0.5 * (-3 * t ** 3 + 4 * t ** 2 + t), 0.5 * (t ** 3 - t ** 2)] for t in frac]
    else:
        offs = (0, 1)
        wts = [[1 - t, t] for t in frac]
    out = torch.zeros_like(pts[0])
    for kz, oz in enumerate(offs):
        for ky, oy in enumerate(offs):
            for kx, ox in enumerate(offs):
                idx = [b + o for b, o in zip(base, (ox, oy, oz))]
                ok = torch.ones_like(idx[0], dtype=torch.bool)
                for i, n in zip(idx, dims):
                    ok &= (i >= 0) & (i < n)
                x, y, z = (i.clamp(0, n - 1) for i, n in zip(idx, dims))
                v = flat[(z * ny + y) * nx + x]
                out = out + wts[0][kx] * wts[1][ky] * wts[2][kz] * torch.where(ok, v, torch.zeros_like(v))
    if interp != "linear_border":
        ok = torch.ones_like(out, dtype=torch.bool)
        for p, n in zip(pts, dims):
            ok &= (p >= 0) & (p <= n - 1)
        out = torch.where(ok, out, torch.zeros_like(out))
    return out


# --------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _blobs(rng, n):
    """40 Gaussian blobs of sigma 2 to 4 voxels (at 64^3) inside a ball, like a density map."""
    scale = n / 64.0
    ax = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
    vol = torch.zeros((n, n, n), device="cuda", dtype=torch.float64)
    for _ in range(40):
        d = rng.standard_normal(3)
        c = 24.0 * scale * rng.uniform() ** (1 / 3) * d / np.linalg.norm(d)
        s = rng.uniform(2, 4) * scale
        gx, gy, gz = (torch.exp(-((ax - float(v)) ** 2) / (2 * s * s)) for v in c)
        vol += gz[:, None, None] * gy[None, :, None] * gx[None, None, :]
    return vol.float()


def _soft_ball(n, radius):
    """A ball with clear faces, smoothed by a nine-tap Gaussian, small values cut to zero."""
    ax = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
    r2 = ax[:, None, None] ** 2 + ax[None, :, None] ** 2 + ax[None, None, :] ** 2
    ball = (r2 <= (radius + 5) ** 2).double()
    for axis in range(3):
        ball.narrow(axis, 0, 5).zero_()
        ball.narrow(axis, n - 5, 5).zero_()
    g = torch.exp(-0.5 * ((torch.arange(9, device="cuda", dtype=torch.float64) - 4) / 2.12) ** 2)
    g = g / g.sum()
    for axis in range(3):
        lead = ball.movedim(axis, -1)
        flat = torch.nn.functional.pad(lead.reshape(-1, 1, n), (4, 4)).unfold(-1, 9, 1)
        ball = (flat * g).sum(-1).reshape(lead.shape).movedim(-1, axis)
    ball = ball / ball.max()
    return torch.where(ball > 1e-3, ball, torch.zeros_like(ball)).float().contiguous()


def _weight(n, tilt, defocus):
    """Half-spectrum weight: missing wedge of a Y tilt axis (+/- tilt degrees) times a CTF (300 kV, 2.5 A)."""
    k = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * n
    kx = torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64)
    kz, ky, kx = torch.meshgrid(k, k, kx, indexing="ij")
    keep = (torch.abs(kz) <= math.tan(math.radians(tilt)) * torch.abs(kx)) | ((kx <= 2) & (torch.abs(kz) <= 2))
    r2 = (kx ** 2 + ky ** 2 + kz ** 2) / (n * 2.5) ** 2
    lam, amp = 0.019687, math.asin(0.07)
    ctf = torch.sin(math.pi * 0.5 * 2.7e7 * lam ** 3 * r2 ** 2 - math.pi * lam * r2 * defocus - amp)
    roll = torch.exp(-((torch.sqrt(kx ** 2 + ky ** 2 + kz ** 2) / n - 0.485).clamp(min=0) * n / 1.5) ** 2 / 2)
    return (keep * ctf * roll).float().contiguous()


def _particle(ref, rng, gen, rotation, shift, weight, snr):
    """The reference rotated, shifted by whole voxels, filtered by its weight, with noise."""
    n = ref.shape[0]
    rot = _sample(ref, _points(ref.shape, rotation.T, (0, 0, 0), True, torch.float32))
    rot = torch.roll(rot, shifts=[int(v) for v in shift], dims=(2, 1, 0))
    sig = torch.fft.irfftn(torch.fft.rfftn(rot) * weight, s=(n, n, n))
    noise = torch.randn((n, n, n), device="cuda", generator=gen) * (sig.std() / math.sqrt(snr))
    return (sig + noise).contiguous()


def _align_inputs(case, seed):
    rng, gen = np.random.default_rng(seed), _generator(seed)
    refs, items = {}, []
    for n, key in ((64, "n64"), (96, "n96"), (128, "n128")):
        if not case[key]:
            continue
        refs[n] = (_blobs(rng, n), _soft_ball(n, 28 * n / 64))
        for _ in range(case[key]):
            prior = _matrix(_random_angles(rng)) if case["step"] < 5 else np.eye(3)
            truth = prior @ _matrix([rng.uniform(-6, 6), rng.uniform(0, 6), rng.uniform(-6, 6)])
            w = _weight(n, rng.uniform(50, 65), rng.uniform(15000, 40000))
            part = _particle(refs[n][0], rng, gen, truth, rng.integers(-4, 5, 3), w, 0.1)
            items.append(dict(n=n, prior=prior, weight=w, particle=part))
    order = rng.permutation(len(items))
    return refs, [items[i] for i in order], _grid(case["orients"], case["step"])


def _refine_inputs(case, seed):
    rng, gen = np.random.default_rng(seed), _generator(seed)
    n = case["n"]
    ref, mask = _blobs(rng, n), _soft_ball(n, 28 * n / 64)
    priors, poses, templates, energies = [], [], [], []
    weight = _weight(n, 60.0, 25000.0)
    for _ in range(case["items"]):
        prior = _matrix(_random_angles(rng))
        pose = np.concatenate([rng.uniform(-3, 3, 3), rng.uniform(-1.5, 1.5, 3)])
        part = _particle(ref, rng, gen, prior, rng.integers(-1, 2, 3), weight, 0.05)
        q = torch.fft.rfftn(part) * weight
        q[0, 0, 0] = 0
        herm = torch.full((n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
        herm[0] = herm[-1] = 1.0
        energies.append(float(((q.real.double() ** 2 + q.imag.double() ** 2) * herm).sum()))
        templates.append((torch.fft.irfftn(q, s=(n, n, n)) * float(n ** 3)).contiguous())
        priors.append(prior)
        poses.append(pose)
    return ref, mask, priors, np.array(poses), templates, energies


def _tsearch_inputs(case, seed):
    rng, gen = np.random.default_rng(seed), _generator(seed)
    t, shape = case["t"], (case["nz"], case["ny"], case["nx"])
    tmpl = _blobs(rng, t)
    grid = _grid(case["orients"] * 20, 12.0)[::20]
    tomo = torch.randn(shape, device="cuda", generator=gen)
    for _ in range(20):
        o = grid[rng.integers(len(grid))]
        rot = _sample(tmpl, _points(tmpl.shape, _matrix([o[0], o[1], o[2] - o[0]]).T, (0, 0, 0), True, torch.float32))
        at = [int(rng.integers(0, s - t + 1)) for s in shape]
        tomo[at[0]:at[0] + t, at[1]:at[1] + t, at[2]:at[2] + t] -= 2.0 * rot
    return tomo, tmpl, grid


def _average_inputs(case, seed):
    rng, gen = np.random.default_rng(seed), _generator(seed)
    n, count = case["n"], case["count"]
    ref, mask = _blobs(rng, n), _soft_ball(n, 28 * n / 64)
    parts = torch.randn((count, n, n, n), device="cuda", generator=gen) * 0.5
    rots, shifts = [], rng.uniform(-2, 2, (count, 3)).astype(np.float32)
    for i in range(count):
        r = _matrix(_random_angles(rng))
        if i % 4 == 0:  # a quarter of the windows hold a copy, the others are background
            parts[i] += _sample(ref, _points(ref.shape, r.T, shifts[i], True, torch.float32))
        rots.append(r)
    return dict(parts=parts, rots=np.array(rots), shifts=shifts, mask=mask,
                weights=rng.uniform(0.5, 1.0, count).astype(np.float32), halves=1 + np.arange(count) % 2,
                wedges=torch.rand((8, n, n, n), device="cuda", generator=gen), index=np.arange(count) % 8,
                sym=np.array([_matrix([0, 0, 360.0 * k / case["symmetry"]]) for k in range(case["symmetry"])]))


def _sf3d_inputs(case, seed):
    rng = np.random.default_rng(seed)
    k = case["tilts"]
    tlt = np.zeros((k, 22))
    tlt[:, 0] = rng.permutation(k) + 1
    tlt[:, 3] = np.linspace(-60, 60, k)
    tlt[:, 10] = np.linspace(0, 120, k)
    tlt[:, 11] = 4.1e-8
    tlt[:, 12] = -1.05
    tlt[:, 13] = rng.uniform(0.8, 1.2, k)
    tlt[:, 14] = -rng.uniform(2.5e-6, 3.5e-6, k)
    tlt[:, 15] = 2.17e-10
    tlt[:, 16] = 2.7e-3
    tlt[:, 17] = 1.968697e-12
    tlt[:, 18] = 0.085
    xyz = rng.uniform(1, [512, 512, 256], (case["count"], 3))
    return tlt, xyz, np.array([[512.0, 512.0, 256.0], [0.0, 1.0, -2.0]])


def _rotate_inputs(case, seed):
    rng = np.random.default_rng(seed)
    vol = torch.randn((case["n"],) * 3, device="cuda", generator=_generator(seed))
    sym = None if case["symmetry"] == 1 else [_matrix([0, 0, 360.0 * k / case["symmetry"]])
                                              for k in range(case["symmetry"])]
    return vol, _matrix(_random_angles(rng)), rng.uniform(-2, 2, 3).astype(np.float32), sym


# --------------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "rotate":
        vol, matrix, shift, sym = _rotate_inputs(case, seed)
        return dict(kind=kind, interp=api.Interpolator(vol, store=case["store"], interp=case["interp"]),
                    matrix=matrix, shift=shift, sym=sym)
    if kind == "fft":
        shape = (case["nz"], case["ny"], case["nx"])
        return dict(kind=kind, ft=api.FourierTransformer(shape),
                    vol=torch.randn(shape, device="cuda", generator=_generator(seed)))
    if kind == "spectra":
        n, b = case["n"], case["count"]
        gen = _generator(seed)
        return dict(kind=kind, parts=torch.randn((b, n, n, n), device="cuda", generator=gen),
                    weights=torch.rand((b, n, n, n // 2 + 1), device="cuda", generator=gen) if case["weights"] else None)
    if kind == "align":
        refs, items, grid = _align_inputs(case, seed)
        s = api.Search(peak_radius=7)
        ids = {n: s.add_reference(r[0], r[1], store=case["store"]) for n, r in refs.items()}
        s.set_orientations(grid)
        keep, descs = [], []
        energies = torch.empty(len(items), device="cuda", dtype=torch.float64)
        for i, it in enumerate(items):
            q, _ = api.particle_spectra(it["particle"][None], energies=energies[i:i + 1])
            keep += [q, it["weight"]]
            descs.append(s.particle(q[0], 0.0, ids[it["n"]], prior=it["prior"], orient_count=len(grid),
                                    wedge=it["weight"]))
        pairs = len(items) * len(grid)
        return dict(kind=kind, search=s, descs=descs, energies=energies, keep=keep,
                    cc=torch.empty(pairs, device="cuda"),
                    peak=torch.empty((pairs, 3), device="cuda", dtype=torch.int32) if case["peaks"] else None,
                    best=torch.empty((len(items), 5), device="cuda", dtype=torch.int32))
    if kind == "refine":
        ref, mask, priors, poses, templates, energies = _refine_inputs(case, seed)
        s = api.Search(peak_radius=6)
        rid = s.add_reference(ref, mask)
        return dict(kind=kind, search=s, poses=poses,
                    objective=refine.BatchObjective(s, [rid] * len(priors), templates, energies, priors))
    if kind == "tsearch":
        tomo, tmpl, grid = _tsearch_inputs(case, seed)
        return dict(kind=kind, search=api.TemplateSearch(tomo), template=tmpl, grid=grid,
                    peak=torch.empty_like(tomo), angle=torch.empty_like(tomo))
    if kind == "normalize":
        shape = (case["nz"], case["ny"], case["nx"])
        vol = torch.randn(shape, device="cuda", generator=_generator(seed))
        z = torch.linspace(0, 1, case["nz"], device="cuda")[:, None, None]
        return dict(kind=kind, vol=(vol * (1 + z) + 0.5 * z).contiguous(), feature=case["feature"])
    if kind == "average":
        a = _average_inputs(case, seed)
        a["sums"] = api.Average(a["mask"], symmetry=a["sym"], wedge_box=case["n"])
        return dict(a, kind=kind)
    tlt, xyz, recon = _sf3d_inputs(case, seed)
    return dict(kind=kind, size=(case["n"],) * 3, tlt=tlt, xyz=xyz, recon=recon)


# --------------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "rotate":
        return s["interp"].interp3d(s["matrix"], s["shift"], "forward", symmetry=s["sym"])
    if kind == "fft":
        spectrum = s["ft"].fwd_fft(s["vol"])
        return spectrum, s["ft"].inv_fft(spectrum)
    if kind == "spectra":
        return api.particle_spectra(s["parts"], s["weights"])
    if kind == "align":
        s["search"].run(s["descs"], cc=s["cc"], peak=s["peak"], best=s["best"], energies=s["energies"])
        # a hit is (cc, orientation, x, y, z): the float and the whole numbers of the same rows
        return dict(cc=s["cc"], peak=s["peak"], best_cc=s["best"][:, 0].view(torch.float32), best=s["best"][:, 1:])
    if kind == "refine":
        return s["objective"].cc_grad(s["poses"])
    if kind == "tsearch":
        return s["search"].run(s["template"], s["grid"], s["peak"], s["angle"])
    if kind == "normalize":
        return api.local_normalize(s["vol"], s["feature"])
    if kind == "average":
        a = s["sums"]
        a.reset()
        kept = a.add(s["parts"], s["rots"], s["halves"], shifts=s["shifts"], weights=s["weights"],
                     wedges=s["wedges"], wedge_index=s["index"])
        return kept, a.result(1), a.result(2)
    return api.sf3d_particles(s["size"], 2.0, s["tlt"], s["xyz"], s["recon"])


# --------------------------------------------------------------------------- work
def _fft_flops(*dims):
    v = 1.0
    for n in dims:
        v *= n
    return 2.5 * v * math.log2(v)


def work(case):
    kind = case["kind"]
    if kind == "rotate":
        v = case["n"] ** 3
        return dict(bytes=v * ((4 if case["store"] == "f32" else 2) + 4), flops=v * 35 * case["symmetry"])
    if kind == "fft":
        v, h = case["nx"] * case["ny"] * case["nz"], (case["nx"] // 2 + 1) * case["ny"] * case["nz"]
        return dict(bytes=2 * (4 * v + 8 * h), flops=2 * _fft_flops(case["nx"], case["ny"], case["nz"]))
    if kind == "spectra":
        n, b = case["n"], case["count"]
        h = (n // 2 + 1) * n * n
        return dict(bytes=b * (4 * n ** 3 + 8 * h + (4 * h if case["weights"] else 0)), flops=b * _fft_flops(n, n, n))
    if kind == "align":
        total, flops = 0, 0
        for n, key in ((64, "n64"), (96, "n96"), (128, "n128")):
            if case[key]:
                h = (n // 2 + 1) * n * n
                pairs = case[key] * case["orients"]
                total += case[key] * 12 * h + 8 * n ** 3 + pairs * 4
                # the rotated reference, its transform, the product, and the transform of the 15^3 window's planes
                flops += pairs * (35 * n ** 3 + _fft_flops(n, n, n) + 12 * h + 5 * h * math.log2(n) + 2 * 15 * n * n * 8)
        return dict(bytes=total, flops=flops)
    if kind == "refine":
        v = case["n"] ** 3
        return dict(bytes=8 * v + case["items"] * 4 * v, flops=case["items"] * v * 150)
    if kind == "tsearch":
        v, h = case["nx"] * case["ny"] * case["nz"], (case["nx"] // 2 + 1) * case["ny"] * case["nz"]
        return dict(bytes=8 * h + 8 * v + 4 * case["t"] ** 3,
                    flops=case["orients"] * (2 * _fft_flops(case["nx"], case["ny"], case["nz"]) + 8 * h))
    if kind == "normalize":
        v = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=8 * v, flops=v * (12 * case["feature"] + 5))
    if kind == "average":
        v = case["n"] ** 3
        return dict(bytes=4 * v * (case["count"] + 8 + 4), flops=2 * case["count"] * v * 40 * case["symmetry"])
    # sf3d: every tilt's CTF image once, and the voxels within 4 of each tilted plane
    n = case["n"]
    return dict(bytes=4 * case["count"] * n ** 3, flops=case["count"] * case["tilts"] * n * n * (60 + 8 * 20))


# --------------------------------------------------------------------------- exact
def _stored(vol, store):
    return vol.bfloat16().double() if store == "bf16" else vol.double()


def _exact_align(case, seed):
    refs, items, grid = _align_inputs(case, seed)
    held = {n: (_stored(r, case["store"]), m.double()) for n, (r, m) in refs.items()}
    cc = torch.empty((len(items), len(grid)), device="cuda", dtype=torch.float64)
    for i, it in enumerate(items):
        n = it["n"]
        ref, mask = held[n]
        w = it["weight"].double()
        q = torch.fft.rfftn(it["particle"].double())
        q[0, 0, 0] = 0
        herm = torch.full((n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
        herm[0] = herm[-1] = 1.0
        energy_p = ((q.real ** 2 + q.imag ** 2) * herm).sum()
        ax = torch.arange(-7, 8, device="cuda")
        inside = (ax[:, None, None] ** 2 + ax[None, :, None] ** 2 + ax[None, None, :] ** 2) <= 49
        at = ax % n
        for o, (phi, theta, psi) in enumerate(grid):
            m = (it["prior"] @ _matrix([phi, theta, psi - phi])).T
            r = torch.fft.rfftn(_sample(ref, _points(ref.shape, m, (0, 0, 0), True, torch.float64)) * mask) * w
            r[0, 0, 0] = 0
            energy_r = ((r.real ** 2 + r.imag ** 2) * herm).sum()
            x = torch.fft.irfftn(q * r.conj(), s=(n, n, n)) * float(n ** 3)
            win = x[at][:, at][:, :, at] / torch.sqrt(energy_r * energy_p)
            cc[i, o] = win[inside].max()
    return dict(cc=cc.reshape(-1), peak=None, best_cc=cc.max(dim=1).values, best=None)


def _exact_refine(case, seed):
    ref, mask, priors, poses, templates, energies = _refine_inputs(case, seed)
    n = case["n"]
    ref, mask = ref.double(), mask.double()
    z, y, x = torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float64) - n // 2] * 3, indexing="ij")
    ccs, grads = [], []
    for prior, pose, h, ep in zip(priors, poses, templates, energies):
        p = torch.tensor(pose, dtype=torch.float64, requires_grad=True)
        a = [p[0], p[1], p[2] - p[0]]
        c, s = [torch.cos(torch.deg2rad(v)) for v in a], [torch.sin(torch.deg2rad(v)) for v in a]
        one, zero = torch.ones((), dtype=torch.float64), torch.zeros((), dtype=torch.float64)

        def mat(rows):
            return torch.stack([torch.stack(r) for r in rows])

        d = (mat([[c[0], -s[0], zero], [s[0], c[0], zero], [zero, zero, one]])
             @ mat([[one, zero, zero], [zero, c[1], -s[1]], [zero, s[1], c[1]]])
             @ mat([[c[2], -s[2], zero], [s[2], c[2], zero], [zero, zero, one]]))
        m = (torch.tensor(prior) @ d).T.cuda()
        t = p[3:].cuda()
        u = [x - t[0], y - t[1], z - t[2]]
        pts = [m[i, 0] * u[0] + m[i, 1] * u[1] + m[i, 2] * u[2] + n // 2 for i in range(3)]
        r = _sample(ref, pts) * mask
        cc = (r * h.double()).sum() / torch.sqrt((n ** 3 * (r * r).sum() - r.sum() ** 2) * ep)
        cc.backward()
        ccs.append(float(cc))
        grads.append(p.grad.numpy())
    return np.array(ccs), np.array(grads)


def _exact_tsearch(case, seed):
    tomo, tmpl, grid = _tsearch_inputs(case, seed)
    shape, t = tuple(tomo.shape), case["t"]
    spec = torch.fft.rfftn(tomo.double())
    nz, ny, nx = shape
    for axis, n in enumerate(shape):
        k = torch.arange(spec.shape[axis], device="cuda", dtype=torch.float64)
        ramp = torch.exp(-2j * math.pi * (k - n // 2) * (n // 2 + 1) / n)
        spec *= ramp.reshape([-1 if a == axis else 1 for a in range(3)])
    low = [(n - t) // 2 + ((n - t) % 2 if t % 2 else 0) for n in shape]
    best = torch.full(shape, -math.inf, device="cuda", dtype=torch.float64)
    for phi, theta, psi in grid:
        m = _matrix([phi, theta, psi - phi]).T  # 'forward' is the transpose of 'inv'
        rot = _sample(tmpl.double(), _points(tmpl.shape, m, (1, 1, 1), True, torch.float64))
        g = torch.zeros(shape, device="cuda", dtype=torch.float64)
        g[low[0]:low[0] + t, low[1]:low[1] + t, low[2]:low[2] + t] = rot
        cc = torch.fft.irfftn(spec * torch.fft.rfftn(g).conj(), s=shape)
        best = torch.maximum(best, cc / cc.std())
        del g, cc
    return best, None


def _exact_normalize(case, seed):
    x = prepare(case, seed)["vol"].double()
    size = case["feature"]
    g = torch.exp(-0.5 * ((torch.arange(size, device="cuda", dtype=torch.float64) - (size - 1) / 2) / 3) ** 2)
    g = g / g.sum()

    def smooth(v):
        for axis in (2, 1, 0):
            n = v.shape[axis]
            out = torch.zeros_like(v)
            for t in range(size):
                q = torch.arange(n, device="cuda") + size // 2 - t
                q = torch.where(q < 0, -q - 1, q)
                q = torch.where(q >= n, 2 * n - q - 1, q)
                out += g[t] * v.index_select(axis, q.clamp(0, n - 1))
            v = out
        return v

    a = smooth(x)
    return (x - a) / torch.sqrt(smooth(x * x) - a * a)


def _exact_average(case, seed):
    a = _average_inputs(case, seed)
    n, mask = case["n"], a["mask"].double()
    inside = a["mask"] > 0.01
    sums = torch.zeros((2, n, n, n), device="cuda", dtype=torch.float64)
    wsum = torch.zeros_like(sums)

    def turned(vol, r, shift):
        out = 0
        for s in a["sym"]:
            out = out + _sample(vol, _points(vol.shape, r @ s, shift, False, torch.float64), "linear_border")
        return out / len(a["sym"])

    for i in range(case["count"]):
        h, w = int(a["halves"][i]) - 1, float(a["weights"][i])
        r = turned(a["parts"][i].double(), a["rots"][i], a["shifts"][i])
        r = r - r[inside].mean()
        sums[h] += r / torch.sqrt((r[inside] ** 2).mean()) * mask * w
        wsum[h] += turned(a["wedges"][int(a["index"][i])].double(), a["rots"][i], (0, 0, 0)) * w
    counts = [int((a["halves"] == k).sum()) for k in (1, 2)]
    return None, (sums[0] / counts[0], wsum[0], None), (sums[1] / counts[1], wsum[1], None)


def _exact_sf3d(case, seed):
    tlt, xyz, recon = _sf3d_inputs(case, seed)
    tlt = tlt[np.argsort(tlt[:, 0], kind="stable")]
    n = case["n"]
    pix, cs, lam, amp = tlt[:, 15] * 2e10, tlt[:, 16] * 1e3, tlt[:, 17] * 1e10, tlt[:, 18]
    tilt = np.radians(tlt[:, 3])
    elastic = np.exp(-75 / (np.cos(tilt) * 400))
    occ = elastic / elastic.max() * tlt[:, 13] / tlt[:, 13].mean()
    c = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
    fy, fx = torch.meshgrid(c, c, indexing="ij")
    half = 0.5 if n % 2 == 0 else 0.0
    z, y, x = torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float64)] * 3, indexing="ij")
    u, w = x - n / 2, z - n // 2
    out = []
    origin = np.ceil((recon[0] + 1) / 2)
    for p in xyz:
        v = p - origin + recon[1]
        vol = torch.zeros((n, n, n), device="cuda", dtype=torch.float64)
        for k in range(len(tlt)):
            df = -tlt[k, 14] * 1e10 - (-math.sin(tilt[k]) * v[0] + math.cos(tilt[k]) * v[2]) * pix[k]
            ddf = tlt[k, 11] * 1e10
            ast = tlt[k, 12] - math.pi * round(math.degrees(tlt[k, 12]) / 180)
            r2 = (fx ** 2 + fy ** 2) / (pix[k] * n) ** 2
            phase = (math.pi * 0.5 * cs[k] * 1e7 * lam[k] ** 3 * r2 ** 2 - math.pi * lam[k] * r2 *
                     (df + ddf * torch.cos(2 * (torch.atan2(fy, fx) - ast))) - math.atan(amp[k] / math.sqrt(1 - amp[k] ** 2)))
            img = torch.sin(phase) ** 2 * occ[k] * torch.where(fx == 0, torch.full_like(fx, 0.2), fx.abs())
            img = img * torch.exp(-0.5 * tlt[k, 10] / (0.24499 * r2 ** -0.8325 + 2.8141))
            s, co = math.sin(-tilt[k]), math.cos(-tilt[k])
            tw = -u * s + half + w * co
            tx = u * co + w * s + half + n / 2 - 0.5
            ty = (y - n // 2) + half + n / 2 - 0.5
            edge = torch.where(tw.abs() <= 4, (0.5 + 0.5 * torch.cos(tw * math.pi / 4)) * 0.25, torch.zeros_like(tw))
            vol += edge * _sample(img[None], [tx, ty, torch.zeros_like(tx)], "linear_border")
        out.append(vol - (vol.min() - 1e-4))
    return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "rotate":
        vol, matrix, shift, sym = _rotate_inputs(case, seed)
        vol = _stored(vol, case["store"])
        mats = [matrix] if sym is None else [matrix @ s for s in sym]
        return sum(_sample(vol, _points(vol.shape, m, shift, True, torch.float64), case["interp"]) for m in mats) / len(mats)
    if kind == "fft":
        vol = torch.randn((case["nz"], case["ny"], case["nx"]), device="cuda", generator=_generator(seed)).double()
        return torch.fft.rfftn(vol), vol * float(vol.numel())
    if kind == "spectra":
        s = prepare(case, seed)
        q = torch.stack([torch.fft.rfftn(p.double()) for p in s["parts"]])
        if s["weights"] is not None:
            q = q * s["weights"].double()
        q[:, 0, 0, 0] = 0
        herm = torch.full((q.shape[-1],), 2.0, device="cuda", dtype=torch.float64)
        herm[0] = 1.0
        if case["n"] % 2 == 0:
            herm[-1] = 1.0
        return q, ((q.real ** 2 + q.imag ** 2) * herm).sum(dim=(1, 2, 3))
    return {"align": _exact_align, "refine": _exact_refine, "tsearch": _exact_tsearch, "normalize": _exact_normalize,
            "average": _exact_average, "sf3d": _exact_sf3d}[kind](case, seed)
