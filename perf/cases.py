"""Performance cases of the GisSPA search: what a user of this library has it do.

Each case is one call (or the few calls of one program step) through the
public entry points of ``gisspa_b200``, on seeded synthetic data of the kind
``gisspa_b200/synth.py`` makes (Gaussian-blob projections, CTF-modulated
particles, 1/f^0.5 noise), generated here on the GPU so that it is quick.

``exact`` computes the same outputs in 64 bits with plain torch.  The discrete
decisions that the search defines in float32 (hot-pixel bounds from running
float sums, band limits, the float rotation coordinates) are taken in float32
there too; everything else is float64.
"""
import math

import numpy as np
import torch

import gisspa_b200 as G

DEV = "cuda"
PI_REF = 3.141592654  # the literal that the search's CTF and rotation angles use
ENERGY, CS, AMP = 300.0, 2.7, 0.07
HIGHRES, LOWRES, KK = 8.0, 100.0, 3.0
NOISE_A, NOISE_B, NOISE_B2 = -9.32, 2.65, 0.01908
BF, BF2, BF3 = -78.7757, -12.9121, 1.28732
CAPACITY = 16384  # picks that a program makes room for per micrograph


def listed():
    return [
        # a first look at a small crop: template set-up and one search, latency counts
        dict(name="oneshot-128", kind="oneshot", nx=512, ny=384, window=128, overlap=32, templates=6, tsize=64,
             phistep=30.0, diameter=48.0, particles=4, snr=0.3, thres=7.0, phase_flip=1, invert=0, precision=0),
        # the library's default window on a K2 micrograph with a coarse template set
        dict(name="default-320", kind="search", nx=3838, ny=3710, window=320, overlap=120, templates=24, tsize=120,
             phistep=15.0, diameter=100.0, particles=120, snr=0.08, thres=8.5, phase_flip=1, invert=0, precision=0),
        # another window, no phase flip (flipped before), inverted contrast, an odd-sided cropped micrograph
        dict(name="ragged-300", kind="search", nx=1443, ny=1190, window=300, overlap=60, templates=15, tsize=90,
             phistep=20.0, diameter=70.0, particles=30, snr=0.8, thres=11.0, phase_flip=0, invert=1, precision=0),
        # the benchmark's small workload: 1024^2, 50 templates of 128^2, 72 angles
        dict(name="small-512", kind="search", nx=1024, ny=1024, window=512, overlap=128, templates=50, tsize=128,
             phistep=5.0, diameter=90.0, particles=20, snr=0.08, thres=8.5, phase_flip=1, invert=0, precision=0),
        # an uneven batch of three detectors' micrographs sharing one template set
        dict(name="batch-512", kind="batch", nx=4096, ny=4096, window=512, overlap=200, templates=20, tsize=180,
             phistep=30.0, diameter=170.0, particles=100, snr=0.05, thres=9.0, phase_flip=1, invert=0, precision=0),
        # the full-size micrograph at window 720, a template set of 100
        dict(name="full-720", kind="search", nx=5760, ny=4092, window=720, overlap=200, templates=100, tsize=200,
             phistep=15.0, diameter=190.0, particles=200, snr=0.05, thres=10.0, phase_flip=1, invert=0, precision=0),
        # the reference's own geometry (window 768), odd template count
        dict(name="wide-768", kind="search", nx=4096, ny=4096, window=768, overlap=200, templates=41, tsize=200,
             phistep=24.0, diameter=190.0, particles=100, snr=0.05, thres=9.0, phase_flip=1, invert=0, precision=0),
        # the all-tensor-core mode that a caller chooses for speed
        dict(name="tensor-720", kind="search", nx=4096, ny=4096, window=720, overlap=200, templates=60, tsize=200,
             phistep=30.0, diameter=190.0, particles=100, snr=0.05, thres=10.0, phase_flip=1, invert=0, precision=4),
        # norm_type 1: z-scores per pixel over all templates and angles
        dict(name="norm1-512", kind="norm1", nx=1100, ny=960, window=512, overlap=100, templates=23, tsize=120,
             phistep=24.0, diameter=90.0, particles=12, snr=0.3, thres=6.0, phase_flip=1, invert=0, precision=0),
        # off-grid refinement: one evaluation of score and gradient (forward and backward) of a set of picks
        dict(name="gradient-512", kind="grad", nx=2048, ny=2048, window=512, overlap=200, templates=32, tsize=128,
             phistep=30.0, diameter=90.0, particles=64, snr=0.1, thres=9.0, phase_flip=1, invert=0, precision=0),
        # one window against a handful of templates from a caller that may not allocate
        dict(name="window-512", kind="window", window=512, templates=16, diameter=90.0),
        # duplicate merging of a session's picks
        dict(name="merge-20000", kind="merge", items=20000, groups=8),
    ]


def _smooth(n, step, prime, least):
    """The largest n - k step that has no prime factor above `prime`."""
    while n > least:
        m, f = n, 2
        while f <= prime:
            if m % f:
                f += 1
            else:
                m //= f
        if m == 1:
            break
        n -= step
    return n


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search"] * 12 + ["oneshot", "batch", "norm1", "tensor", "grad", "window", "merge"])
    if kind == "merge":
        return dict(kind="merge", items=_log_int(rng, 500, 20000), groups=rng.randint(1, 12))
    how = rng.random()
    if how < 0.5:
        window = 32 * rng.randint(4, 24)       # what the reference takes: multiples of 32
    elif how < 0.75:
        window = rng.choice([320, 512, 720, 768])
    else:
        # other windows; at l = 2 mod 4 the search's sign convention turns every peak negative
        window = _smooth(4 * rng.randint(32, 192), 4, 23, 128)
    if kind == "norm1":
        window = 32 * rng.randint(4, 16)
    if kind == "tensor":
        window = 720
    if kind == "window":
        return dict(kind="window", window=window, templates=rng.randint(1, 40), diameter=round(window * rng.uniform(0.15, 0.3), 1))
    tsize = max(50, 2 * int(window * rng.uniform(0.13, 0.25)))
    diameter = float(int(tsize * rng.uniform(0.72, 0.9)))
    big = kind in ("search", "tensor")
    nx = min(5760, max(int(1.4 * window), _log_int(rng, 600, 5760 if big else 2048)))
    ny = min(4096, max(int(1.3 * window), int(nx * rng.uniform(0.65, 1.0))))
    # cropped or binned ones may be odd; prime factors up to the detectors' (3838 = 2 19 101)
    nx, ny = _smooth(nx, 1, 127, window), _smooth(ny, 1, 127, window)
    overlap = int(window * rng.uniform(0.15, 0.4))
    step = window - overlap
    nw = (1 + math.ceil((nx - window) / step)) * (1 + math.ceil((ny - window) / step))
    # pair units x window^2 stays well below the largest listed case's, and below default-320's at
    # windows other than the common three
    most = 105600.0 * 720 * 720 * {"search": 0.5, "tensor": 0.5, "batch": 0.1}.get(kind, 0.02)
    if window not in (512, 720, 768):
        most *= 0.3
    angles = rng.choice([6, 8, 10, 12, 15, 18, 24, 36, 72])
    while angles > 6 and nw * angles * 3 * window * window > most:
        angles //= 2
    top = max(1, int(most / (float(nw) * angles * window * window)))
    templates = min(2 * _log_int(rng, 1, max(2, min(60, top))) - rng.randint(0, 1), 2 * top)
    if kind == "norm1":
        templates, angles = max(9, templates), max(10, angles)
    flip = 0 if kind == "search" and rng.random() < 0.25 else 1
    return dict(kind=("search" if kind == "tensor" else kind), nx=nx, ny=ny, window=window, overlap=overlap,
                templates=max(2, templates), tsize=tsize, phistep=360.0 / angles, diameter=diameter,
                particles=rng.randint(6, 40), snr=round((1200.0 if flip else 4000.0) / diameter ** 2, 4), thres=(5.5 if kind == "norm1" else 9.0 if flip else 11.0),
                phase_flip=flip, invert=rng.randint(0, 1),
                precision=(4 if kind == "tensor" else 0))


# --------------------------------------------------------------------------
# Seeded inputs
# --------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _views(g, n):
    alt = torch.arccos(2.0 * _rand(g, n) - 1.0)
    az = 2.0 * math.pi * _rand(g, n)
    return alt, az


def _density(g, radius, blobs=150):
    d = torch.randn(blobs, 3, generator=g, device=DEV, dtype=torch.float64)
    d = d / d.norm(dim=1, keepdim=True) * (radius * _rand(g, blobs, 1) ** (1.0 / 3.0))
    return d, 2.0 + 2.0 * _rand(g, blobs)


def _project(centers, alt, az):
    ca, sa, cz, sz = torch.cos(alt), torch.sin(alt), torch.cos(az), torch.sin(az)
    zero = torch.zeros_like(ca)
    rows = torch.stack([torch.stack([cz, sz, zero], -1), torch.stack([-ca * sz, ca * cz, sa], -1)], -2)
    return torch.einsum("nij,bj->nbi", rows, centers)


def _render(xy, amp, sig, size):
    grid = torch.arange(size, device=DEV, dtype=torch.float64) - size // 2
    s2 = 2.0 * sig[None, :, None] ** 2
    gx = torch.exp(-((grid - xy[:, :, 0:1]) ** 2) / s2) * amp[None, :, None]
    gy = torch.exp(-((grid - xy[:, :, 1:2]) ** 2) / s2)
    return torch.bmm(gy.transpose(1, 2), gx)


def _offsets(n, l, overlap):
    offs, off = [0], 0
    while off + l < n:
        off += l - overlap
        if off + l >= n:
            off = n - l
        offs.append(off)
    return offs


def _angles(step):
    out, e = [], np.float32(0.0)
    while e < np.float32(360.0):
        out.append(float(e))
        e = np.float32(e + np.float32(step))
    return out


def _lambda():
    return float(np.float32(12.2639 / math.sqrt(ENERGY * 1000.0 + 0.97845 * ENERGY * ENERGY)))


def _ctf_grid(nx, ny, ctf):
    """The search's CTF at the FFT indices of an nx x ny spectrum, and s^2, in 64 bits."""
    defocus, dfdiff, dfang = (float(np.float32(v)) for v in ctf)
    x = torch.arange(nx, device=DEV)[None, :].expand(ny, nx)
    y = torch.arange(ny, device=DEV)[:, None].expand(ny, nx)
    y1 = (y + ny // 2) % ny
    y1 = torch.where(x > nx // 2, ny - y1, y1)
    dx = torch.minimum(x, nx - x).double()
    dy = (y1 - ny // 2).double()
    ss = dx * dx / float(nx * nx) + dy * dy / float(ny * ny)
    df = -defocus + dfdiff * torch.cos(2.0 * (dfang * PI_REF / 180.0 - torch.atan2(dy, dx)))
    return _ctf_value(ss, df), ss


def _ctf_value(ss, df):
    lam, cs, amp = _lambda(), float(np.float32(CS)), float(np.float32(AMP))
    gamma = -2.0 * PI_REF * (cs * 2.5e6 * lam ** 3 * ss * ss + df * 5000.0 * lam * ss)
    return math.sqrt(1.0 - amp * amp) * torch.sin(gamma) + amp * torch.cos(gamma)


def _sizes(case):
    if case["kind"] != "batch":
        return [(case["nx"], case["ny"])]
    if min(case["nx"], case["ny"]) >= 3710:
        return [(3838, 3710), (4096, 4096), (5760, 4092)]
    return [(case["nx"], case["ny"]), (case["ny"], case["nx"] - 7), (case["nx"] - 31, case["ny"] - 2)]


def _inputs(case, seed):
    """Templates (n, t, t) float32 on the host, and per micrograph its pixels
    (float32, host), CTF line and planted particles (x, y, template, angle index)."""
    g = _gen(seed)
    t, n = case["tsize"], case["templates"]
    centers, sig = _density(g, 0.42 * case["diameter"])
    alt, az = _views(g, n)
    amp = math.sqrt(2.0 * math.pi) * sig
    xy = _project(centers, alt, az)
    templates = _render(xy, amp, sig, t).float().cpu().numpy()
    angles = _angles(case["phistep"])
    host = np.random.RandomState(int(seed) % (1 << 31))
    mics = []
    for nx, ny in _sizes(case):
        ctf = (float(np.float32(0.8 + 1.7 * host.rand())), float(np.float32(0.02 * host.rand())), float(np.float32(180.0 * host.rand())))
        spec = torch.fft.rfft2(torch.randn(ny, nx, generator=g, device=DEV))
        fy, fx = torch.fft.fftfreq(ny, device=DEV)[:, None], torch.fft.rfftfreq(nx, device=DEV)[None, :]
        f = torch.sqrt(fx * fx + fy * fy)
        f[0, 0] = 1.0
        spec = spec * f ** -0.25
        spec[0, 0] = 0.0
        img = torch.fft.irfft2(spec, s=(ny, nx)).double()
        img *= 1.2 / img.std()
        m = int(math.ceil(case["diameter"])) + 2
        box = 2 * (t // 2)
        edge = max(m, box // 2)
        clean = torch.zeros(ny, nx, device=DEV, dtype=torch.float64)
        parts, pitch = [], int(case["diameter"])
        cells = [(x, y) for y in range(edge, ny - edge, pitch) for x in range(edge, nx - edge, pitch)]
        for k in host.permutation(len(cells))[: case["particles"]]:
            parts.append((cells[k][0], cells[k][1], int(host.randint(n)), int(host.randint(len(angles)))))
        if parts:
            e = torch.tensor([math.radians(angles[p[3]]) for p in parts], device=DEV, dtype=torch.float64)
            q = xy[[p[2] for p in parts]]
            c, s = torch.cos(e)[:, None], torch.sin(e)[:, None]
            q = torch.stack([c * q[..., 0] - s * q[..., 1], s * q[..., 0] + c * q[..., 1]], -1)
            for p, r in zip(parts, _render(q, amp, sig, box)):
                clean[p[1] - box // 2: p[1] - box // 2 + box, p[0] - box // 2: p[0] - box // 2 + box] += r
            # phase_flip 0 is for micrographs whose phases were flipped before, invert 1 for dark particles
            seen = _ctf_grid(nx, ny, ctf)[0] * (-1.0 if case["invert"] else 1.0)
            if case["phase_flip"] == 0:
                seen = seen.abs() * (-1.0 if case["invert"] else 1.0)
            seen = torch.fft.ifft2(torch.fft.fft2(clean) * seen).real
            area = len(parts) * math.pi * case["diameter"] ** 2 / 4.0
            img += seen * math.sqrt(case["snr"] * 1.44 / (float(seen.square().sum()) / area))
        mics.append((img.float().cpu().numpy(), ctf, parts))
    return templates, mics


def _params(case):
    return G.default_params(apix=1.0, phi_step=case["phistep"], kk=KK, energy=ENERGY, cs=CS, highres=HIGHRES,
                            lowres=LOWRES, d_m=case["diameter"], thres=case["thres"], window_size=case["window"],
                            overlap=case["overlap"], phase_flip=case["phase_flip"], invert=case["invert"],
                            norm_type=1 if case["kind"] == "norm1" else 0, precision=case["precision"])


def _grad_picks(case, mic, seed):
    """One pick per particle, moved off the grid: its most central window, position, angle, shift and CTF."""
    img, ctf, parts = mic
    l = case["window"]
    ox, oy = _offsets(img.shape[1], l, case["overlap"]), _offsets(img.shape[0], l, case["overlap"])
    angles = _angles(case["phistep"])
    r = np.random.RandomState((int(seed) + 5) % (1 << 31))
    picks = np.zeros(len(parts), dtype=G.REFINE_PICK_DTYPE)
    for k, (x, y, J, a) in enumerate(parts):
        i = min(range(len(ox)), key=lambda q: abs(ox[q] + l // 2 - x))
        j = min(range(len(oy)), key=lambda q: abs(oy[q] + l // 2 - y))
        picks[k] = (i + j * len(ox), J, (y - oy[j]) * l + (x - ox[i]), angles[a] + r.uniform(-1.5, 1.5),
                    r.uniform(-0.4, 0.4), r.uniform(-0.4, 0.4), ctf[0] + r.uniform(-0.03, 0.03),
                    0.005 + 0.02 * r.rand(), ctf[2] + r.uniform(-5.0, 5.0))
    return picks


def _window_inputs(case, seed):
    """A window spectrum and template-pair spectra as the search builds them (FFT / l^2)."""
    g = _gen(seed)
    l, n, d = case["window"], case["templates"], case["diameter"]
    centers, sig = _density(g, 0.42 * d)
    alt, az = _views(g, n)
    amp = math.sqrt(2.0 * math.pi) * sig
    xy = _project(centers, alt, az)
    t = _render(xy, amp, sig, l)
    t = t - t.mean(dim=(1, 2), keepdim=True)
    t = t / t.square().mean(dim=(1, 2), keepdim=True).sqrt()
    win = torch.randn(l, l, generator=g, device=DEV, dtype=torch.float64)
    at = _rand(g, 2) * (l - 1.2 * d) - (l / 2.0 - 0.6 * d)
    win += 0.25 * t[0].roll((int(at[0]), int(at[1])), (0, 1))
    win -= win.mean()
    if n % 2:
        t = torch.cat([t, torch.zeros_like(t[:1])])
    W = (torch.fft.fft2(win) / (l * l)).to(torch.complex64)
    T = torch.fft.fft2(t) / (l * l)
    return W, (T[0::2] - 1j * T[1::2]).to(torch.complex64).contiguous()


def _merge_inputs(case, seed):
    r = np.random.RandomState(int(seed) % (1 << 31))
    n, groups = case["items"], case["groups"]
    it = np.zeros(n, dtype=G.MERGE_ITEM_DTYPE)
    real = max(1, n // 15)                      # about fifteen templates and angles pick the same particle
    px, py = r.uniform(100, 5600, real), r.uniform(100, 4000, real)
    pa = np.stack([r.uniform(5, 175, real), r.uniform(0, 360, real), r.uniform(0, 360, real)], 1)
    pg = r.randint(0, groups, real)
    who = r.randint(0, real, n)
    who = who[np.argsort(pg[who], kind="stable")]
    it["x"], it["y"] = px[who] + r.randint(-6, 7, n), py[who] + r.randint(-6, 7, n)
    it["alt"], it["az"], it["phi"] = (pa[who, k] + r.normal(0, 4.0, n) for k in range(3))
    it["score"], it["group"] = r.uniform(7, 14, n), pg[who]
    return it


# --------------------------------------------------------------------------
# What a program has in hand, and one pass
# --------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "merge":
        return dict(kind=kind, items=_merge_inputs(case, seed))
    if kind == "window":
        W, P = _window_inputs(case, seed)
        return dict(kind=kind, W=W, P=P, n=case["templates"], l=case["window"], d_m=case["diameter"],
                    out=torch.zeros(case["templates"], 4, dtype=torch.int32, device=DEV))
    templates, mics = _inputs(case, seed)
    params = _params(case)
    ctx = G.Context(0)
    state = dict(kind=kind, ctx=ctx, images=[m[0] for m in mics], ctfs=[m[1] for m in mics])
    if kind == "oneshot":
        state.update(params=params, templates=templates)
    else:
        ctx.set_templates(params, templates, mics[0][1])
    if kind == "grad":
        ctx.search(mics[0][0], mics[0][1])      # the picks refer to the window spectra of a search
        state["picks"] = _grad_picks(case, mics[0], seed)
    return state


def _columns(picks):
    """The pick list in a program's fixed buffers: one column per field, zeros
    behind the last pick (the count is `n`)."""
    out = dict(n=len(picks))
    for k in picks.dtype.names:
        out[k] = np.zeros(CAPACITY, dtype=picks.dtype[k])
        out[k][: len(picks)] = picks[k]
    return out


def run(state):
    kind = state["kind"]
    if kind == "merge":
        return G.merge_duplicates(state["items"], 20.0, 10.0)
    if kind == "window":
        out = state["out"]
        G.correlate_window_noalloc(state["W"].data_ptr(), state["P"].data_ptr(), state["n"], state["l"],
                                   state["d_m"], out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        f = out.view(torch.float32)
        return dict(score=f[:, 0], pos=out[:, 1], peak=f[:, 2], sigma=f[:, 3])
    ctx = state["ctx"]
    if kind == "grad":
        r = ctx.score_grad(state["picks"])
        return dict(score=r["score"].copy(), gradient=np.stack([r[k] for k in r.dtype.names[1:]], 1))
    if kind == "batch":
        return [_columns(p) for p in ctx.search_batch(state["images"], state["ctfs"])]
    if kind == "oneshot":
        ctx.set_templates(state["params"], state["templates"], state["ctfs"][0])
    return _columns(ctx.search(state["images"][0], state["ctfs"][0]))


def work(case):
    """Inputs once, outputs once; FLOPs of a real transform per (template,
    window, angle) unit (2.5 n log2 n) with product and reductions (6 n), and
    of the template spectra, micrograph and window transforms."""
    kind = case["kind"]
    if kind == "merge":
        n, per = case["items"], case["items"] / float(case["groups"])
        return dict(bytes=57.0 * n, flops=4.0 * n * per / 2.0)  # one distance test per pair of a group
    l = case["window"]
    px = float(l * l)
    unit = 2.5 * px * math.log2(px) + 6.0 * px
    if kind == "window":
        n = case["templates"]
        return dict(bytes=8.0 * px * (1 + (n + 1) // 2) + 16.0 * n, flops=n * unit)
    n, angles = case["templates"], len(_angles(case["phistep"]))
    bytes_, flops = 4.0 * n * (px if kind != "oneshot" else case["tsize"] ** 2), 0.0
    if kind == "grad":
        k = case["particles"]
        # forward: base, weighted, rotated transforms and the product; backward the same back
        return dict(bytes=k * (4.0 + 8.0) * px, flops=k * (5 * 2 * 2.5 * px * math.log2(px) + 60.0 * px))
    sweeps = 2 if kind == "norm1" else 1
    for nx, ny in _sizes(case):
        nw = len(_offsets(nx, l, case["overlap"])) * len(_offsets(ny, l, case["overlap"]))
        bytes_ += 4.0 * nx * ny
        flops += 5.0 * nx * ny * math.log2(nx * ny) + nw * 2.5 * px * math.log2(px) + sweeps * n * angles * nw * unit
    return dict(bytes=bytes_, flops=flops + sweeps * n * angles * (2.5 * px * math.log2(px) + 14.0 * px))


# --------------------------------------------------------------------------
# The same outputs in 64 bits
# --------------------------------------------------------------------------
def _f32(v):
    return float(np.float32(v))


def _shells(nx, ny):
    x = torch.arange(nx, device=DEV)[None, :]
    y = torch.arange(ny, device=DEV)[:, None]
    dx, dy = torch.minimum(x, nx - x).double(), torch.minimum(y, ny - y).double()
    rf = torch.sqrt(dx * dx + dy * dy).float().double()
    return torch.floor(rf + 0.5).long() - 1, rf


def _band(r, hp, lp, low_cut):
    r = r.double()
    keep = (r < hp) & ((r >= lp) if low_cut else (r >= 0))
    hi = ~keep & (r >= hp) & (r < hp + 8)
    lo = ~keep & ~hi & (r >= lp - 8) & (r < lp) & (r >= 0)
    out = torch.zeros_like(r)
    out = torch.where(hi, 0.5 * torch.cos(PI_REF * (r - hp) / 16.0) + 0.5, out)
    out = torch.where(lo, 0.5 * torch.cos(PI_REF * (lp - r) / 16.0) + 0.5, out)
    return torch.where(keep, torch.ones_like(out), out)


def _limits(L):
    return _f32(np.float32(L) / np.float32(HIGHRES)), _f32(np.float32(L) / np.float32(LOWRES))


def _half(l):
    r, _ = _shells(l, l)
    inside = (r >= 0) & (r < l // 2)
    return r, inside, inside & (torch.arange(l, device=DEV)[None, :] <= l // 2)


def _curves(ss, kk):
    signal = torch.exp(BF * ss * ss + BF2 * ss + BF3)
    noise = torch.exp(NOISE_A * ss * ss + NOISE_B * ss + NOISE_B2)
    return signal, noise


def _base_spectra(raw, l):
    """Padded, edge-normalised, whitened template spectra (FFT / l^2)."""
    t = torch.from_numpy(raw).to(DEV).double()
    n, ty, tx = t.shape
    p = torch.zeros(n, l, l, device=DEV, dtype=torch.float64)
    sy, sx = (l - ty) // 2, (l - tx) // 2
    p[:, sy:sy + ty, sx:sx + tx] = t
    q = (torch.arange(l, device=DEV) - l // 2).double()
    rr = q[:, None] ** 2 + q[None, :] ** 2
    r = l / 2.0 - 2.0
    ring = (rr >= (r - 1) ** 2) & (rr <= (r + 1) ** 2) if r > 1 else rr <= 0
    em = p[:, ring].mean(dim=1)
    sd = (p.square().mean(dim=(1, 2)) - p.mean(dim=(1, 2)) ** 2).clamp(min=0).sqrt()
    p = torch.where(sd[:, None, None] >= 1e-8, (p - em[:, None, None]) / sd[:, None, None], p)
    F = torch.fft.fft2(p) / (l * l)
    shell, inside, half = _half(l)
    idx = shell[half]
    count = torch.zeros(l // 2, device=DEV, dtype=torch.float64).index_add_(0, idx, torch.ones_like(idx, dtype=torch.float64))
    for k in range(n):
        s = torch.zeros(l // 2, device=DEV, dtype=torch.float64).index_add_(0, idx, F[k].abs().square()[half])
        d = torch.sqrt(s / count)
        F[k] = torch.where(inside, F[k] / d[shell.clamp(0, l // 2 - 1)], F[k])
    return F


def _weight(l, window, ctf):
    """Band-pass x |CTF| x Wiener weight of the templates; `ctf` may hold tensors (defocus, dfdiff, dfang)."""
    shell, rf = _shells(l, l)
    inside = (shell >= 0) & (shell < l // 2)
    hp, lp = _limits(l)
    x = torch.arange(l, device=DEV)[None, :].expand(l, l)
    y1 = (torch.arange(l, device=DEV)[:, None].expand(l, l) + l // 2) % l
    y1 = torch.where(x > l // 2, l - y1, y1)
    dx, dy = torch.minimum(x, l - x).double(), (y1 - l // 2).double()
    df = -ctf[0] + ctf[1] * torch.cos(2.0 * (ctf[2] * PI_REF / 180.0 - torch.atan2(dy, dx)))
    v = _ctf_value((dx * dx + dy * dy) / float(l * l), df).abs()
    ss = rf * _f32(np.float32(1.0) / np.float32(window))
    signal, noise = _curves(ss, KK)
    noise = noise / (signal / (KK + 1.0))
    w = v * torch.sqrt(1.0 / (noise + KK * v * v))
    return _band(shell, hp, lp, False) * torch.where(inside, w, torch.ones_like(w)), inside


def _prepared_templates(raw, l, window, ctf):
    F = _base_spectra(raw, l)
    w, _ = _weight(l, window, [_f32(v) for v in ctf])
    _, _, half = _half(l)
    F = F * w
    s = torch.stack([f.abs().square()[half].sum() for f in F])
    m = torch.sqrt(s) / float(half.sum())
    F = F / torch.where(m != 0, m, torch.ones_like(m))[:, None, None]
    return torch.fft.ifft2(F, norm="forward").real


def _rotation(l, angle):
    """Gather indices and weights of the bilinear rotation, source coordinates in float32."""
    a = _f32(angle) * PI_REF / 180.0
    c, s = _f32(math.cos(a)), _f32(math.sin(a))
    q = (torch.arange(l, device=DEV) - l // 2).double()
    x, y = q[None, :], q[:, None]
    x2 = ((c * x + (s * y).float().double()).float() + float(l // 2)).double()
    y2 = ((-s * x + (c * y).float().double()).float() + float(l // 2)).double()
    return _gather(l, x2, y2)


def _gather(l, x2, y2):
    inside = ~((x2 < 0) | (x2 > l - 1.0) | (y2 < 0) | (y2 > l - 1.0))
    ii = torch.floor(x2.detach()).clamp(0, l - 1).long()
    jj = torch.floor(y2.detach()).clamp(0, l - 1).long()
    t, u = x2 - ii, y2 - jj
    i1, j1 = (ii + 1).clamp(max=l - 1), (jj + 1).clamp(max=l - 1)
    return inside, ((jj * l + ii, (1 - t) * (1 - u)), (jj * l + i1, t * (1 - u)),
                    (j1 * l + i1, t * u), (j1 * l + ii, (1 - t) * u))


def _rotate(flat, how):
    inside, taps = how
    out = sum(flat[..., k.reshape(-1)].reshape(*flat.shape[:-1], *k.shape) * w for k, w in taps)
    return torch.where(inside, out, torch.zeros_like(out))


def _mask(l, d_m):
    q = (torch.arange(l, device=DEV) - l // 2).double()
    r = torch.sqrt(q[:, None] ** 2 + q[None, :] ** 2).float().double()
    dm = _f32(1.5 * _f32(d_m))
    outer = _f32(np.float32(dm / 2) + np.float32(12.0))
    m = torch.where(r > outer, torch.zeros_like(r), torch.ones_like(r))
    soft = (r <= outer) & (r >= dm / 2)
    return torch.where(soft, 0.5 * torch.cos(PI_REF * (r - dm / 2) / 12.0) + 0.5, m)


def _normal(t):
    mean = t.mean(dim=(-2, -1), keepdim=True)
    var = t.square().mean(dim=(-2, -1), keepdim=True) - mean * mean
    return (t - mean) / torch.where(var != 0, var.abs().sqrt(), torch.ones_like(var))


def _clamped(img, invert):
    ny, nx = img.shape
    v = img.ravel()
    s1 = np.add.accumulate((v / np.float32(nx)) / np.float32(ny))[-1]
    s2 = np.add.accumulate((v * v / np.float32(nx)) / np.float32(ny))[-1]
    out = torch.from_numpy(img).to(DEV)
    if s2 > s1 * s1:
        sd = np.float32(np.sqrt(s2 - s1 * s1))
        up, low = float(int(s1 + np.float32(6) * sd)), float(int(s1 - np.float32(6) * sd))
        out = torch.where((out > up) | (out < low), torch.full_like(out, float(s1)), out)
    return (-out if invert == 1 else out).double()


def _micrograph(case, img, ctf):
    ny, nx = img.shape
    F = torch.fft.fft2(_clamped(img, case["invert"])) / (nx * ny)
    if case["phase_flip"] == 1:
        L = max(nx, ny)
        v, s2 = _ctf_grid(nx, ny, ctf)
        F = F * torch.where(v > 0, 1.0, -1.0)
        v = v.abs()
        shell, _ = _shells(nx, ny)
        inside = (shell >= 0) & (shell < L // 2)
        half = inside & (torch.arange(nx, device=DEV)[None, :] <= nx // 2)
        idx = shell[half]
        total = torch.zeros(L // 2, device=DEV, dtype=torch.float64).index_add_(0, idx, F.abs().square()[half])
        count = torch.zeros(L // 2, device=DEV, dtype=torch.float64).index_add_(0, idx, torch.ones_like(idx, dtype=torch.float64))
        rms = torch.sqrt(total / count)[shell.clamp(0, L // 2 - 1)]
        # the frequencies by unfolded indices, for the curves and the damping
        fx = torch.minimum(torch.arange(nx, device=DEV), nx - torch.arange(nx, device=DEV)).double() / nx
        fy = torch.minimum(torch.arange(ny, device=DEV), ny - torch.arange(ny, device=DEV)).double() / ny
        ss = torch.sqrt(fx[None, :] ** 2 + fy[:, None] ** 2)
        signal, noise = _curves(ss, KK)
        f = torch.where(inside, torch.sqrt((signal * v * v + noise) / signal) / rms, torch.ones_like(ss))
        f = torch.where(inside & (shell > _f32(np.float32(L) / np.float32(6))), f * torch.exp(-100.0 * ss * ss), f)
        f = f * _band(shell, *_limits(L), True)
        noise = noise / (signal / (KK + 1.0))
        f = torch.where(inside, f * torch.sqrt(1.0 / (noise + KK * v * v)), f)
        F = F * f
    F[0, 0] = 0.0
    return torch.fft.ifft2(F, norm="forward").real


def _window_spectra(case, img, ctf):
    l = case["window"]
    m = _micrograph(case, img, ctf)
    ox, oy = _offsets(m.shape[1], l, case["overlap"]), _offsets(m.shape[0], l, case["overlap"])
    W = torch.stack([torch.fft.fft2(m[y:y + l, x:x + l]) / (l * l) for y in oy for x in ox])
    if case["phase_flip"] == 1:
        _, _, half = _half(l)
        s = torch.stack([w.abs().square()[half].sum() for w in W])
        a = torch.sqrt(s) / float(half.sum())
        W = W / torch.where(a != 0, a, torch.ones_like(a))[:, None, None]
    return W, ox, oy


def _maps(W, P):
    """Correlation maps of the window spectra W (w) with one pair spectrum, in
    fftshifted window coordinates: (w, 2, l, l)."""
    l = P.shape[-1]
    s = torch.fft.ifft2(W * P.conj(), norm="forward").roll((l // 2, l // 2), (-2, -1))
    sgn = 1.0 if (l // 2) % 2 == 0 else -1.0
    return torch.stack([s.real, s.imag], -3) * sgn


def _unit_scores(maps, d_m):
    l = maps.shape[-1]
    q = _f32(np.float32(d_m) / np.float32(4))
    k = torch.arange(l, device=DEV).double()
    keep = (k >= q) & (k <= _f32(np.float32(l) - np.float32(q)))
    flat = maps.reshape(*maps.shape[:-2], l * l)
    inner = torch.where(keep[:, None] & keep[None, :], maps, torch.zeros_like(maps)).reshape(flat.shape)
    peak, pos = inner.max(dim=-1)
    s1, s2 = flat.sum(-1), flat.square().sum(-1)
    rc = float(l * l - 1)
    sd = torch.sqrt((s2 - peak * peak) / rc - ((s1 - peak) / rc) ** 2)
    return peak / sd, pos, peak, sd


def _chunks(n, per):
    return [slice(a, min(n, a + per)) for a in range(0, n, max(1, per))]


def _search_exact(case, templates, mics):
    l, n = case["window"], case["templates"]
    T = _prepared_templates(templates, l, case["window"], mics[0][1]).reshape(n, l * l)
    mask = _mask(l, case["diameter"])
    spectra = [_window_spectra(case, img, ctf) for img, ctf, _ in mics]
    W = torch.cat([s[0] for s in spectra])
    angles = _angles(case["phistep"])
    per = max(1, int(2e8 / (l * l * 16)))
    norm1 = case["kind"] == "norm1"
    if norm1:
        s1 = torch.zeros(len(W), l, l, device=DEV, dtype=torch.float64)
        s2 = torch.zeros_like(s1)
    d_m, found = _f32(case["diameter"]), [[] for _ in mics]

    def pairs(angle):
        t = _normal(_rotate(T, _rotation(l, angle)) * mask)
        F = torch.fft.fft2(t) / (l * l)
        if n % 2:
            F = torch.cat([F, torch.zeros_like(F[:1])])
        return F[0::2] - 1j * F[1::2]

    if norm1:
        for a in angles:
            for p, P in enumerate(pairs(a)):
                for c in _chunks(len(W), per):
                    m = _maps(W[c], P)[:, : min(2, n - 2 * p)] / (l * l)
                    s1[c] += m.sum(1)
                    s2[c] += m.square().sum(1)
        mean = s1 / (n * len(angles))
        sd = torch.sqrt(s2 / (n * len(angles)) - mean * mean)
    for ai, a in enumerate(angles):
        got = [[], []]
        for p, P in enumerate(pairs(a)):
            for c in _chunks(len(W), per):
                m = _maps(W[c], P)[:, : min(2, n - 2 * p)]
                if norm1:
                    z = (m / (l * l) - mean[c, None]) / sd[c, None]
                    v, at = z.reshape(*z.shape[:2], -1, 1024).max(-1)
                    at = at + 1024 * torch.arange(v.shape[-1], device=DEV)
                else:
                    v, at, _, _ = _unit_scores(m, d_m)
                    v, at = v[..., None], at[..., None]
                keep = torch.nonzero(v >= case["thres"])
                for (w, q, b), sc, pos in zip(keep.tolist(), v[tuple(keep.T)].tolist(), at[tuple(keep.T)].tolist()):
                    got[0].append((c.start + w, 2 * p + q, b))
                    got[1].append((sc, pos))
        for (w, J, b), (sc, pos) in sorted(zip(*got)):
            first = 0
            for k, (Wm, ox, oy) in enumerate(spectra):
                if w < first + len(Wm):
                    cx, cy = ox[(w - first) % len(ox)] + pos % l, oy[(w - first) // len(ox)] + pos // l
                    ny, nx = mics[k][0].shape
                    if d_m <= cx < nx - d_m and d_m <= cy < ny - d_m:
                        found[k].append((sc, cx, cy))
                    break
                first += len(Wm)
    out = []
    for f in found:
        c = np.zeros((3, CAPACITY))
        c[:, : len(f)] = np.array(f, dtype=np.float64).reshape(-1, 3).T
        out.append(dict.fromkeys(("n",) + G.PICK_DTYPE.names) | dict(score=c[0], center_x=c[1], center_y=c[2]))
    return out if case["kind"] == "batch" else out[0]


def _grad_exact(case, templates, mics, picks):
    l = case["window"]
    B = _base_spectra(templates, l)
    W, _, _ = _window_spectra(case, mics[0][0], mics[0][1])
    mask = _mask(l, case["diameter"])
    _, _, half = _half(l)
    count = float(half.sum())
    k = torch.arange(l, device=DEV)
    k = torch.where(k < l // 2, k, k - l).double()
    q = (torch.arange(l, device=DEV) - l // 2).double()
    sgn = 1.0 if (l // 2) % 2 == 0 else -1.0
    scores, grads = [], []
    for p in picks:
        v = torch.tensor([float(p[c]) for c in ("angle", "dx", "dy", "defocus", "dfdiff", "dfang")], device=DEV,
                         dtype=torch.float64, requires_grad=True)
        w, _ = _weight(l, case["window"], (v[3], v[4], v[5]))
        F1 = B[int(p["template_index"])] * w
        a = torch.sqrt((F1.real.square() + F1.imag.square())[half].sum()) / count
        t = torch.fft.ifft2(F1 / a, norm="forward").real
        e = v[0] * PI_REF / 180.0
        x2 = torch.cos(e) * q[None, :] + torch.sin(e) * q[:, None] + l // 2
        y2 = -torch.sin(e) * q[None, :] + torch.cos(e) * q[:, None] + l // 2
        F = torch.fft.fft2(_normal(_rotate(t.reshape(-1), _gather(l, x2, y2)) * mask)) / (l * l)
        pos = int(p["pos"])
        x0, y0 = (pos % l - l // 2) % l, (pos // l - l // 2) % l
        ph = 2.0 * math.pi * (k[None, :] * (x0 + v[1]) + k[:, None] * (y0 + v[2])) / l
        Wp = W[int(p["window"])]
        c = (Wp * F.conj() * torch.complex(torch.cos(ph), torch.sin(ph))).real.sum()
        sig = torch.sqrt((Wp.abs().square() * (F.real.square() + F.imag.square())).sum())
        s = sgn * c / sig
        s.backward()
        scores.append(float(s.detach()))
        grads.append(v.grad.cpu().numpy())
    return dict(score=np.array(scores), gradient=np.stack(grads))


def exact(case, seed):
    kind = case["kind"]
    if kind == "merge" or case.get("precision"):
        # a keep mask; and which units the 16-bit mode puts above the threshold is its own
        return None
    if kind == "window":
        W, P = _window_inputs(case, seed)
        got = [_unit_scores(_maps(W[None].to(torch.complex128), p.to(torch.complex128))[0], case["diameter"]) for p in P]
        score, _, peak, sd = (torch.cat(v)[: case["templates"]] for v in zip(*got))
        return dict(score=score, pos=None, peak=peak, sigma=sd)
    templates, mics = _inputs(case, seed)
    if kind == "grad":
        return _grad_exact(case, templates, mics, _grad_picks(case, mics[0], seed))
    return _search_exact(case, templates, mics)
