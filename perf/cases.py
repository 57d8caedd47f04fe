"""The work a user of this package has it do, as measurable cases.

Every case is one pass through a public entry point on seeded synthetic data:
single filtering stages (``stage_device``), the learned pilot's inference and
training gradient (``PilotNet``), the device-resident two-stage run under
Gaussian noise (``bmnd_device``) and whole denoising calls (``bmnd``).  Sizes
follow the package's benchmark workloads and tests, plus ragged generic ones.
"""

import itertools
import math

import numpy as np
import torch

import bmnd_gb300 as bg
from bmnd_gb300 import api, gaussian
from bmnd_gb300 import pilot as pilot_mod
from bmnd_gb300.validation import resolve_profile


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a thumbnail through the drop-in call, NumPy in and out: launches and host work dominate
        {"name": "denoise_2d_small", "kind": "denoise", "noise": "poisson", "host": True, "d0": 64, "d1": 64, "d2": 0,
         "peak": 40.0},
        # a photograph-sized count image of ragged extents, both stages, resident on the device
        {"name": "denoise_2d_image", "kind": "denoise", "noise": "poisson", "host": False, "d0": 321, "d1": 481,
         "d2": 0, "peak": 40.0},
        # stage 1 of a large detector frame
        {"name": "ht_2d_large", "kind": "ht", "noise": "poisson", "d0": 2048, "d1": 2048, "d2": 0, "peak": 60.0},
        # stage 2 of a small image on a given stage-1 estimate
        {"name": "wiener_2d", "kind": "wiener", "noise": "poisson", "d0": 320, "d1": 256, "d2": 0, "peak": 50.0},
        # stage 1 of a ragged sub-volume
        {"name": "ht_3d", "kind": "ht", "noise": "poisson", "d0": 96, "d1": 104, "d2": 113, "peak": 30.0},
        # stage 2 of a volume: the largest part of the plain 3-D call
        {"name": "wiener_3d", "kind": "wiener", "noise": "poisson", "d0": 128, "d1": 144, "d2": 160, "peak": 30.0},
        # low counts (tomography at low dose), stage 2 of a small volume
        {"name": "wiener_3d_low", "kind": "wiener", "noise": "poisson", "d0": 40, "d1": 48, "d2": 56, "peak": 4.0},
        # the headline workload: the learned pilot's whole call on a 256^3 volume, NumPy in and out
        {"name": "learned_3d", "kind": "learned", "noise": "poisson", "host": True, "d0": 256, "d1": 256, "d2": 256,
         "peak": 30.0},
        # additive Gaussian noise, both stages of an image (SSD matching, covariance maps)
        {"name": "gauss_2d", "kind": "denoise_device", "noise": "gaussian", "d0": 768, "d1": 640, "d2": 0,
         "sigma": 5.0},
        # additive Gaussian noise, both stages of a volume
        {"name": "gauss_3d", "kind": "denoise_device", "noise": "gaussian", "d0": 80, "d1": 96, "d2": 90,
         "sigma": 2.0},
        # the learned pilot alone: BF16 inference of the 3-D net
        {"name": "net_forward", "kind": "net_forward", "noise": "poisson", "d0": 160, "d1": 144, "d2": 176,
         "peak": 30.0},
        # one gradient of the 3-D net at its training shape (4 crops of 48^3)
        {"name": "net_gradient", "kind": "net_gradient", "noise": "poisson", "batch": 4, "d0": 48, "d1": 48, "d2": 48,
         "peak": 30.0},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def extents(total_lo, total_hi, nd, least):
        """`nd` uneven extents with a product between the two totals, log-uniform."""
        total = math.exp(rng.uniform(math.log(total_lo), math.log(total_hi)))
        edge = total ** (1.0 / nd)
        out = [max(least, int(round(edge * math.exp(rng.uniform(-0.25, 0.25))))) for _ in range(nd - 1)]
        out.append(max(least, int(total / math.prod(out))))
        return out + [0] * (3 - nd)

    kind = rng.choice(["denoise2", "denoise3", "ht2", "ht3", "wiener2", "wiener3", "learned2", "learned3", "gauss2",
                       "gauss3", "net_forward", "net_gradient"])
    nd = 2 if kind.endswith("2") else 3
    peak = round(math.exp(rng.uniform(math.log(3.0), math.log(60.0))), 1)
    case = {"kind": kind.rstrip("23"), "noise": "poisson", "peak": peak}
    if kind in ("denoise2", "denoise3", "learned2", "learned3"):
        case["host"] = rng.random() < 0.5
    if kind.startswith("gauss"):
        case = {"kind": "denoise_device", "noise": "gaussian", "sigma": round(rng.uniform(1.0, 8.0), 1)}
    if kind == "net_gradient":
        case["batch"] = rng.randint(1, 4)
        d = [log_int(24, 48) for _ in range(3)]
    else:
        lo, hi = {"denoise2": (3e3, 1.2e6), "denoise3": (2e4, 8e5), "ht2": (2e4, 4e6), "ht3": (2e4, 1.1e6),
                  "wiener2": (1e4, 1.2e6), "wiener3": (2e4, 2.9e6), "learned2": (2e4, 1.2e6),
                  "learned3": (1e5, 1.6e7), "gauss2": (1e4, 8e5), "gauss3": (2e4, 7e5),
                  "net_forward": (1e5, 4e6)}[kind]
        d = extents(lo, hi, nd, 40 if nd == 2 else 20)
    case.update(d0=d[0], d1=d[1], d2=d[2])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _shape(case):
    return tuple(d for d in (case["d0"], case["d1"], case["d2"]) if d)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + 17)


def _scene(shape, seed, peak):
    """A piecewise smooth non-negative scene with maximum ``peak``: a low
    background, 24 ellipsoids of constant intensity and a slow illumination."""
    rng = np.random.default_rng([int(seed), 5])
    axes = [torch.arange(n, device="cuda", dtype=torch.float32).reshape([-1 if i == a else 1 for i in range(len(shape))])
            for a, n in enumerate(shape)]
    clean = torch.full(shape, 0.08, device="cuda")
    edge = min(shape)
    for _ in range(24):
        r2 = 0.0
        for a, n in enumerate(shape):
            semi = edge * rng.uniform(0.05, 0.3)
            r2 = r2 + ((axes[a] - rng.uniform(0, n)) / semi) ** 2
        clean = torch.where(r2 <= 1.0, torch.full_like(clean, rng.uniform(0.15, 1.0)), clean)
    for a, n in enumerate(shape):
        clean = clean * (1.0 + 0.15 * torch.sin(axes[a] * (2.0 * math.pi * rng.uniform(0.5, 1.5) / n)))
    return clean * (peak / float(clean.max()))


def _blur(x, times=3):
    """Separable box smoothing (the look of a first estimate's residual noise)."""
    nd = x.dim()
    pool = torch.nn.functional.avg_pool2d if nd == 2 else torch.nn.functional.avg_pool3d
    y = x[None, None]
    for _ in range(times):
        y = pool(y, 3, stride=1, padding=1, count_include_pad=False)
    return y[0, 0].contiguous()


def _inputs(case, seed):
    """(clean, noisy) CUDA float32 volumes; a batch where the case has one."""
    shape = _shape(case)
    gen = _generator(seed)
    if case["noise"] == "gaussian":
        clean = _scene(shape, seed, 100.0)
        return clean, clean + case["sigma"] * torch.randn(shape, generator=gen, device="cuda")
    if "batch" in case:
        clean = torch.stack([_scene(shape, 100 * int(seed) + b, case["peak"]) for b in range(case["batch"])])
    else:
        clean = _scene(shape, seed, case["peak"])
    return clean, torch.poisson(clean, generator=gen)


def _pilot_estimate(clean, noisy):
    """A first estimate of ordinary quality: the scene plus smoothed residual noise."""
    return (clean + 0.5 * _blur(noisy - clean)).clamp_min(0.0).contiguous()


def _fresh_params(seed, channels=48, layers=8):
    """Parameters of an untrained 3-D net (He-normal weights, zero biases), as
    at the start of a training run: layer by layer W[tap][ci][co], then b[co]."""
    rng = np.random.default_rng([int(seed), 9])
    parts = []
    for layer in range(layers):
        ci, co = 1 if layer == 0 else channels, 1 if layer == layers - 1 else channels
        std = math.sqrt(2.0 / (27 * ci)) * (0.1 if layer == layers - 1 else 1.0)
        parts += [rng.normal(0.0, std, size=27 * ci * co), np.zeros(co)]
    return np.concatenate(parts).astype(np.float32)


def _profile(case):
    noise = bg.NoiseModel.POISSON if case["noise"] == "poisson" else bg.NoiseModel.GAUSSIAN
    return (bg.BM3DProfile if len(_shape(case)) == 2 else bg.BM4DProfile)(noise_model=noise)


def prepare(case, seed):
    kind = case["kind"]
    clean, noisy = _inputs(case, seed)
    state = {"kind": kind}
    if kind in ("net_forward", "net_gradient"):
        state["noisy"] = noisy
        if kind == "net_forward":
            state["net"] = pilot_mod.PilotNet.load(pilot_mod.default_net_path("bm4d"))
        else:
            state["net"] = pilot_mod.PilotNet(3, 48, 8, params=_fresh_params(seed))
            state["target"] = torch.stack([_pilot_estimate(c, n) for c, n in zip(clean, noisy)])
        return state
    profile = _profile(case)
    resolved = resolve_profile(profile, _shape(case))
    state.update(profile=profile, resolved=resolved, noisy=noisy)
    if kind in ("denoise", "learned") and case["host"]:
        state["noisy"] = noisy.cpu().numpy()
    if kind == "wiener":
        state["pilot"] = _pilot_estimate(clean, noisy)
    if kind == "denoise_device":
        model = gaussian.build_model(_shape(case), profile.nf, sigma=case["sigma"])
        state["gauss"] = api.gaussian_tables(model, profile, _shape(case), resolved, noisy.device)
    return state


def run(state):
    kind = state["kind"]
    if kind == "denoise":
        return bg.bmnd(state["noisy"], state["profile"])
    if kind == "learned":
        return bg.bmnd(state["noisy"], state["profile"], pilot="learned")
    if kind == "denoise_device":
        return bg.bmnd_device(state["noisy"], state["profile"], resolved=state["resolved"], gauss=state["gauss"])
    if kind == "ht":
        return api.stage_device(state["noisy"], state["profile"], "ht", resolved=state["resolved"])
    if kind == "wiener":
        return api.stage_device(state["noisy"], state["profile"], "wiener", state["pilot"],
                                resolved=state["resolved"])
    if kind == "net_forward":
        pilot, y = state["net"].forward(state["noisy"], want_y=True)
        return {"pilot": pilot, "y": y}
    if kind == "net_gradient":
        loss, grad = state["net"].gradient(state["noisy"], state["target"])
        return {"loss": loss, "grad": grad}
    raise ValueError(kind)


# ---------------------------------------------------------------------------
# work that cannot be avoided
# ---------------------------------------------------------------------------
def work(case):
    shape = _shape(case)
    vox = float(math.prod(shape))
    nd = len(shape)
    kind = case["kind"]
    if kind in ("net_forward", "net_gradient"):
        channels, layers, taps = 48, 8, 27
        vox *= case.get("batch", 1)
        flops = 2.0 * vox * taps * ((layers - 2) * channels ** 2 + 2 * channels)
        weights = 4.0 * taps * ((layers - 2) * channels ** 2 + 2 * channels)
        if kind == "net_forward":
            return {"bytes": 12.0 * vox + weights / 2, "flops": flops}
        return {"bytes": 8.0 * vox + 2 * weights, "flops": 3.0 * flops}

    def stage(name):
        wiener = name == "wiener"
        block, radius, stack = ((8, 19, 32 if wiener else 16) if nd == 2 else (5, 7, 32) if wiener else (4, 7, 16))
        patch, window = block ** nd, (2 * radius + 1) ** nd
        step = 4 if kind == "learned" and nd == 3 else 3
        groups = 2.0 * vox / step ** nd
        # every voxel against every offset of half the window (the distance is
        # symmetric), about 8 operations a term with its share of the patch sum
        match = vox * window / 2 * 8
        transforms = groups * 2 * stack * patch * (stack + nd * block) * (3 if wiener else 2) * 2
        exact = 0.0 if kind == "learned" and nd == 3 else groups * 2 * stack * patch * 4 * patch
        return match + transforms + exact

    if kind == "ht":
        return {"bytes": 8.0 * vox, "flops": stage("ht")}
    if kind == "wiener":
        return {"bytes": 12.0 * vox, "flops": stage("wiener")}
    if kind == "learned":
        channels, layers, taps = (48, 8, 27) if nd == 3 else (32, 10, 9)
        net = 2.0 * vox * taps * ((layers - 2) * channels ** 2 + 2 * channels)
        return {"bytes": 8.0 * vox, "flops": net + stage("wiener")}
    return {"bytes": 8.0 * vox, "flops": stage("ht") + stage("wiener")}


# ---------------------------------------------------------------------------
# the outputs in 64 bits
# ---------------------------------------------------------------------------
def _schedule(counts, block, step):
    """Reference positions: a lattice whose odd rows are shifted (shift density
    2, two phases), the last position of every axis forced."""
    nd = len(counts)
    shifts, last, slots = [], [], []
    for d in range(nd):
        n = min(max(math.ceil(2.0 * (block - 1) / step), 1), block)
        vals = {0} if d == nd - 1 or n == 1 else {0} | {int(np.rint(v)) for v in np.linspace(0, block - 1, n)}
        shifts.append(sorted(vals))
        last.append(counts[d] - 1)
        slots.append(-(-last[d] // step) + 1)
    seen, out = set(), []
    for slot in itertools.product(*[range(s) for s in slots]):
        for phase in range(2):
            pos = []
            for d in range(nd):
                off = shifts[d][(slot[d + 1] + phase) % len(shifts[d])] if d < nd - 1 else 0
                a = min(max(min(slot[d] * step, last[d]) - off, 0), last[d])
                pos.append(last[d] if slot[d] == slots[d] - 1 else a)
            if tuple(pos) not in seen:
                seen.add(tuple(pos))
                out.append(pos)
    return torch.tensor(out, device="cuda", dtype=torch.int64)


def _key(d):
    """Distances rounded to 2^-18 of their power of two (at least 1): the
    quantised keys in which the matching compares, exact in float32."""
    e = (torch.frexp(d.abs().clamp_min(1.0))[1] - 1).float()
    return torch.round(d * torch.exp2(18 - e)) * torch.exp2(e - 18)


def _match(src, refs, counts, offs, offsets, radius, stack, threshold):
    """Match sets of `refs`: the smallest Poisson deviances in the window, in
    float32 term by term (the matching's definition), ties by position."""
    nd = len(counts)
    flat = src.reshape(-1)
    stride = [math.prod(src.shape[d + 1:]) for d in range(nd)]
    cand = refs[:, None, :] + offsets[None]
    ok = torch.ones(cand.shape[:2], dtype=torch.bool, device="cuda")
    base = torch.zeros(cand.shape[:2], dtype=torch.int64, device="cuda")
    lin = torch.zeros_like(base)
    for d in range(nd):
        c = cand[..., d]
        ok &= (c >= 0) & (c < counts[d])
        base += c.clamp(0, counts[d] - 1) * stride[d]
        lin = lin * counts[d] + c
    rbase = sum(refs[:, d] * stride[d] for d in range(nd))
    dist = torch.zeros(base.shape, device="cuda")
    for o in offs.tolist():
        r = flat[rbase + o][:, None]
        c = flat[base + o]
        s = r + c
        t = torch.where(r > 0, r * torch.log(2.0 * r / s), torch.zeros_like(s))
        t = torch.where(c > 0, t + c * torch.log(2.0 * c / s), t)
        dist = dist + torch.where(s > 0, 2.0 * t, torch.zeros_like(t))
    key = _key(dist.clamp_min(0.0) / torch.tensor(float(len(offs)), device="cuda"))
    accept = ok & (key < _key(torch.tensor(threshold, device="cuda", dtype=torch.float32)))
    order = key.view(torch.int32).long() * 4096 + torch.arange(offsets.shape[0], device="cuda")
    order = torch.where(accept, order, order + (1 << 50))
    order = torch.where(ok, order, torch.full_like(order, 1 << 60))
    best, at = torch.topk(order, stack, dim=1, largest=False)
    got = best < (1 << 50)
    if stack >= 2:
        got[:, :2] |= best[:, :2] < (1 << 60)  # filled up to two members
    centre = torch.zeros_like(lin[:, 0])
    for d in range(nd):
        centre = centre * counts[d] + refs[:, d]
    sel = torch.gather(lin, 1, at)
    got &= sel != centre[:, None]
    sel = torch.where(got, sel, torch.full_like(sel, -1))
    place = torch.where(got, got.cumsum(1), torch.full_like(sel, stack))
    out = torch.full((sel.shape[0], stack + 1), -1, dtype=torch.int64, device="cuda")
    out.scatter_(1, place.clamp_max(stack), sel)
    out[:, 0] = centre
    n = (got.sum(1) + 1).clamp_max(stack)
    n = torch.exp2(torch.floor(torch.log2(n.float() + 0.5))).long()
    return out[:, :stack], n


def _haar(n):
    s = np.float32(1.0 / np.sqrt(2.0))
    m = np.ones((1, 1), dtype=np.float32)
    while m.shape[0] < n:
        k = m.shape[0]
        m = np.vstack([np.kron(m, np.array([s, s])), np.kron(np.eye(k, dtype=np.float32), np.array([s, -s]))])
        m = m.astype(np.float32)
    return torch.tensor(m, device="cuda", dtype=torch.float64)


def _axis(kind, n):
    """One axis's forward matrix (float32 entries) and its inverse, in float64."""
    if kind == "dct":
        k, x = np.mgrid[0:n, 0:n]
        f = (np.sqrt(np.where(k == 0, 1.0, 2.0) / n) * np.cos(np.pi * (x + 0.5) * k / n)).astype(np.float32)
        return f.astype(np.float64), f.T.astype(np.float64)
    if n == 4:
        q = 0.70710677
        f = [[.5, .5, .5, .5], [.5, .5, -.5, -.5], [q, -q, 0, 0], [0, 0, q, -q]]
    else:
        a, b, c, d = 0.343550200747110, 0.225454819240296, 0.461645582253923, 0.569359398342840
        e, g, h = 0.402347308162280, 0.083506045090280, 0.707106781186550
        f = [[a] * 8, [-b, -c, -c, -b, b, c, c, b], [d, e, -e, -d, -g, g, -g, g], [-g, g, -g, g, d, e, -e, -d],
             [h, -h, 0, 0, 0, 0, 0, 0], [0, 0, h, -h, 0, 0, 0, 0], [0, 0, 0, 0, h, -h, 0, 0],
             [0, 0, 0, 0, 0, 0, h, -h]]
    f = np.array(f, dtype=np.float32).astype(np.float64)
    return f, np.linalg.inv(f).astype(np.float32).astype(np.float64)


def _stage64(noisy, pilot):
    """One filtering stage of the direct-Poisson method on float32 inputs:
    float32 matching, everything after it in float64.  `pilot` None: hard
    thresholding; else the Wiener stage, matched on the pilot."""
    nd, wiener = noisy.dim(), pilot is not None
    block, radius = (8, 19) if nd == 2 else (5 if wiener else 4, 7)
    stack = 32 if wiener else 16
    threshold = 2.9527 if not wiener else (0.3937 if nd == 2 else 0.7689)
    shape = tuple(noisy.shape)
    counts = tuple(s - block + 1 for s in shape)
    P = block ** nd
    f1, i1 = _axis("dct" if wiener else "bior", block)
    fwd, inv = np.ones((1, 1)), np.ones((1, 1))
    win = np.ones(())
    for _ in range(nd):
        fwd, inv, win = np.kron(fwd, f1), np.kron(inv, i1), np.multiply.outer(win, np.kaiser(block, 2.0))
    fwd, inv = (torch.tensor(m, device="cuda") for m in (fwd, inv))
    win = torch.tensor(win.astype(np.float32).astype(np.float64).reshape(-1), device="cuda")
    stride = [math.prod(shape[d + 1:]) for d in range(nd)]
    local = torch.tensor(list(itertools.product(range(block), repeat=nd)), device="cuda")
    offs = sum(local[:, d] * stride[d] for d in range(nd))
    offsets = torch.tensor(list(itertools.product(range(-radius, radius + 1), repeat=nd)), device="cuda")
    refs = _schedule(counts, block, 3)
    src = (pilot if wiener else noisy).float()
    x64 = noisy.double().reshape(-1)
    p64 = pilot.double().reshape(-1) if wiener else None
    var = (src.double().reshape(-1)).clamp_min(1e-10)
    num, den = torch.zeros_like(x64), torch.zeros_like(x64)
    span = 2 * radius + block
    cells = span ** nd
    for r0 in range(0, refs.shape[0], 4096):
        sel, size = _match(src, refs[r0:r0 + 4096], counts, offs, offsets, radius, stack, threshold)
        for n in (1, 2, 4, 8, 16, 32):
            rows = sel[size == n]
            if not rows.shape[0]:
                continue
            G, k = _haar(n), min(4, n)
            step = max(1, int(1.5e9 / (8.0 * cells * k * P)))
            for b0 in range(0, rows.shape[0], step):
                lins = rows[b0:b0 + step, :n]
                B = lins.shape[0]
                pos, rem = [], lins
                for d in reversed(range(nd)):
                    pos.insert(0, rem % counts[d])
                    rem = rem // counts[d]
                pos = torch.stack(pos, -1)
                idx = (sum(pos[..., d] * stride[d] for d in range(nd))[..., None] + offs)  # [B, n, P]

                def forward(v, group, space):
                    return torch.einsum("ig,bgp->bip", group, v) @ space.T

                X = forward(x64[idx], G, fwd)
                V = forward(var[idx], G * G, fwd * fwd).clamp_min(0.0)
                # exact planes: sum over union voxels of V (sum over their entries of G S)^2
                shift = pos - pos.amin(1, keepdim=True)
                cell = 0
                for d in range(nd):
                    cell = cell * span + shift[..., d, None] + local[:, d]
                cell = cell + torch.arange(B, device="cuda")[:, None, None] * cells
                acc = torch.zeros((B * cells, k * P), device="cuda", dtype=torch.float64)
                vol = torch.zeros(B * cells, device="cuda", dtype=torch.float64)
                for m in range(n):
                    row = (G[:k, m, None, None] * fwd[None]).permute(2, 0, 1).reshape(P, k * P)
                    acc.index_add_(0, cell[:, m].reshape(-1), row.repeat(B, 1))
                    vol[cell[:, m].reshape(-1)] = var[idx[:, m].reshape(-1)]
                exact = torch.einsum("bcq,bc->bq", acc.square_().reshape(B, cells, k * P), vol.reshape(B, cells))
                exact = exact.reshape(B, k, P)
                del acc
                rest = V[:, k:].sum(1)
                target = (V.sum(1) - exact.sum(1)).clamp_min(0.0)
                scale = torch.where(rest > 0, target / rest.clamp_min(1e-300), torch.zeros_like(rest))
                nv = torch.cat([exact, V[:, k:] * scale[:, None]], 1)
                if wiener:
                    eff = 0.4 * nv
                    power = (forward(p64[idx], G, fwd).square() - eff).clamp_min(0.0)
                    att = (power / (power + eff + 1e-10)).clamp(0.0, 1.0)
                else:
                    thr, mag = 3.0 * nv.sqrt(), X.abs()
                    top = torch.maximum(torch.maximum(mag, thr), torch.ones_like(mag))
                    att = (mag > thr + 2.0 ** -16 * top).double()
                risk = (att.square() * nv).sum(2)
                weight = 1.0 / (risk @ (G * G) + 1e-10)
                Y = torch.einsum("gi,bgp->bip", G, X * att) @ inv.T
                ww = weight[..., None] * win
                num.index_add_(0, idx.reshape(-1), (Y * ww).reshape(-1))
                den.index_add_(0, idx.reshape(-1), ww.reshape(-1))
    out = torch.where(den > 0, num / (den + 1e-10), x64)
    return out.reshape(shape)


def _net64(case, seed):
    """The pilot net in float64 with its float32 parameters: forward (the
    stored net), or the loss and its gradient (an untrained net)."""
    clean, noisy = _inputs(case, seed)
    channels, layers = 48, 8
    train = case["kind"] == "net_gradient"
    params = _fresh_params(seed) if train else np.load(pilot_mod.default_net_path("bm4d"))["params"]
    flat = torch.tensor(params.astype(np.float64), device="cuda", requires_grad=train)
    x = noisy.double() if noisy.dim() == 4 else noisy.double()[None]
    a = 2.0 * torch.sqrt(x.clamp_min(0.0) + 0.375)

    def conv(h, w, b):
        # one tap at a time: out[co] += w[tap][ci][co] h[ci] shifted by the tap
        hp = torch.nn.functional.pad(h, (1, 1) * 3)
        out = b[None, :, None, None, None]
        for t, (z, y, q) in enumerate(itertools.product(range(3), repeat=3)):
            part = hp[:, :, z:z + h.shape[2], y:y + h.shape[3], q:q + h.shape[4]]
            out = out + torch.einsum("bizyx,io->bozyx", part, w[t])
        return out

    h, at = a[:, None], 0
    for layer in range(layers):
        ci, co = 1 if layer == 0 else channels, 1 if layer == layers - 1 else channels
        w = flat[at:at + 27 * ci * co].reshape(27, ci, co)
        at += 27 * ci * co
        h = conv(h, w, flat[at:at + co])
        at += co
        if layer < layers - 1:
            h = torch.relu(h)
    y = a + h[:, 0]
    if case["kind"] == "net_forward":
        return {"pilot": ((y / 2.0) ** 2 - 0.375).clamp_min(0.0)[0].detach(), "y": y[0].detach()}
    target = torch.stack([_pilot_estimate(c, n) for c, n in zip(clean, noisy)]).double()
    loss = ((y - 2.0 * torch.sqrt(target.clamp_min(0.0) + 0.375)) ** 2).mean()
    loss.backward()
    return {"loss": loss.detach().reshape(1), "grad": flat.grad}


def exact(case, seed):
    """`run`'s outputs in 64 bits; None for the learned and the Gaussian whole
    calls (a BF16 net's or a covariance model's output feeds a matching), and
    for sizes whose float64 evaluation takes minutes."""
    kind, shape = case["kind"], _shape(case)
    vox = math.prod(shape)
    if kind in ("net_forward", "net_gradient"):
        vox *= case.get("batch", 1)
        return _net64(case, seed) if vox <= (1_200_000 if kind == "net_forward" else 450_000) else None
    if kind not in ("ht", "wiener", "denoise"):
        return None
    if vox > ({"ht": 1_300_000, "wiener": 250_000, "denoise": 160_000}[kind] if len(shape) == 3 else 600_000):
        return None
    clean, noisy = _inputs(case, seed)
    if kind == "ht":
        return _stage64(noisy, None)
    if kind == "wiener":
        return _stage64(noisy, _pilot_estimate(clean, noisy))
    out = _stage64(noisy, _stage64(noisy, None).float())
    return out.cpu().numpy() if case["host"] else out
