"""Performance cases: the work that a user of this framework has it do.

Each case is one call (or one kept handle's call) through the public entry
points, on seeded inputs made on the GPU. ``listed()`` names the cases,
``draw(rng)`` gives more of the same ranges, ``exact(case, seed)`` restates
what a case computes in plain torch, in 64 bits.

Inputs follow the generator of ``pymatting_b200.synthetic``: cubic colour
fields with N(0, 0.02) noise for foreground and background, a union of
ellipses with a soft edge as the matte, and a trimap whose unknown band is the
edge widened by a few pixels; the unknown fraction is between 5 and 25 %.
"""

import math
import random
import time

import numpy as np
import torch

import pymatting_b200 as pm
from pymatting_b200.laplacian import device_csr_arrays
from pymatting_b200.synthetic import batch_sizes

DEV = "cuda"
F64 = torch.float64
LAMBDA, EPS = 100.0, 1e-7
BATCH_SEED = 1000     # the sizes of bench.py's 64-image batch


def listed():
    return [
        # The smallest soft-constraint call, as an interactive preview makes
        # it for each new trimap stroke: latency, launches and setup count.
        dict(name="soft preview", kind="soft", count=1, h=240, w=320, precision="mixed"),
        # One ordinary photograph solved as accurately as the reference does,
        # with odd sides.
        dict(name="soft hd fp64", kind="soft", count=1, h=1079, w=1917, precision="fp64"),
        # The batch of bench.py: 64 images of six sizes, mixed precision.
        dict(name="soft batch64", kind="soft", count=64, h=0, w=0, precision="mixed"),
        # estimate_alpha_cf with its defaults (hard constraints, incomplete
        # Cholesky): the reference's headline call at its CPU-runnable size.
        dict(name="hard 320x240", kind="hard", h=240, w=320),
        # A training step through the differentiable alpha: forward solve,
        # adjoint solve and the image gradient, float32 images.
        dict(name="grad 4x512", kind="grad", count=4, h=512, w=512),
        # The preconditioner as a handle in a user's own solver loop: one
        # V-cycle in FP64 at full HD.
        dict(name="vcycle hd", kind="vcycle", h=1080, w=1920),
        # Assembly of the Laplacian as a CSR matrix on the device.
        dict(name="cf_laplacian 720p", kind="laplacian", h=720, w=1280),
        # One product with the large-kernel Laplacian, the step that a solver
        # over it repeats.
        dict(name="lkm apply 720p", kind="lkm", h=720, w=1280, radius=10),
        # The nearest-neighbour Laplacian of a small image.
        dict(name="knn 256", kind="knn", h=256, w=256),
        # Foreground colours of a solved matte, exact sweep order: a full-HD
        # frame, and a small odd-sided image with its background too.
        dict(name="fg ml hd", kind="fg", h=1080, w=1920, background=False),
        dict(name="fg ml small", kind="fg", h=227, w=341, background=True),
        # The fast (Jacobi) foreground variant on a full-HD frame.
        dict(name="fg jacobi hd", kind="fgj", h=1080, w=1920, background=True),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["soft", "soft", "soft", "hard", "grad", "vcycle", "laplacian", "lkm",
                       "knn", "fg", "fg", "fgj"])
    if kind == "soft":
        return dict(kind=kind, count=rng.choice([1, 1, 2, 3, 5, 8]), h=size(128, 1536),
                    w=size(128, 2048), precision=rng.choice(["mixed", "fp64"]))
    if kind == "hard":
        return dict(kind=kind, h=size(80, 240), w=size(80, 320))
    if kind == "grad":
        return dict(kind=kind, count=rng.randint(1, 4), h=size(96, 640), w=size(96, 640))
    if kind == "lkm":
        return dict(kind=kind, h=size(96, 1080), w=size(96, 1920), radius=rng.choice([3, 5, 10]))
    if kind == "knn":
        return dict(kind=kind, h=size(64, 300), w=size(64, 300))
    if kind in ("fg", "fgj"):
        return dict(kind=kind, h=size(64, 1536), w=size(64, 2048),
                    background=rng.choice([True, False]))
    return dict(kind=kind, h=size(128, 1536), w=size(128, 2048))


def _sizes(case):
    """(h, w) of every image: the case's own size first, the others of a
    batch smaller and odd."""
    if case["kind"] == "soft" and case["h"] == 0:
        return [(h, w) for h, w, _f, _s in batch_sizes(case["count"], BATCH_SEED)]
    sizes = [(case["h"], case["w"])] * case.get("count", 1)
    if case["kind"] == "soft":
        rng = random.Random(case["h"] * 4099 + case["w"])
        sizes[1:] = [(rng.randint(case["h"] // 2, case["h"]), rng.randint(case["w"] // 2, case["w"]))
                     for _ in sizes[1:]]
    return sizes


def work(case):
    px = float(sum(h * w for h, w in _sizes(case)))
    kind = case["kind"]
    # Flops: 3x3 windows of 81 colour pairs and their 3x3 covariance (about
    # 900 per pixel) wherever a matting Laplacian is made; one V-cycle is two
    # 25-point stencils on 4/3 of the pixels.
    if kind == "soft" or kind == "hard":
        return {"bytes": (24 + 8 + 8) * px, "flops": 900 * px}
    if kind == "grad":        # image, trimap, cotangent in; alpha, gradient out
        return {"bytes": (12 + 4 + 4 + 4 + 12) * px, "flops": 2 * 900 * px}
    if kind == "vcycle":      # 13 planes, r in; z out
        return {"bytes": (13 + 1 + 1) * 8 * px, "flops": 2 * 50 * 4 / 3 * px}
    if kind == "laplacian":   # 25 values and columns per row
        return {"bytes": (24 + 25 * 16 + 8) * px, "flops": 900 * px}
    if kind == "lkm":         # image, p, 10 coefficients per window in; L p out
        return {"bytes": (3 + 1 + 10 + 1) * 8 * px, "flops": 100 * px}
    if kind == "knn":         # up to 60 entries per row
        return {"bytes": (24 + 60 * 16) * px, "flops": 1000 * px}
    out = 24 if case["background"] else 12
    return {"bytes": (16 + out) * px, "flops": 2 * 4 / 3 * 80 * px}


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------

def _colour_field(g, h, w):
    y = torch.linspace(-1, 1, h, dtype=F64, device=DEV)[:, None, None]
    x = torch.linspace(-1, 1, w, dtype=F64, device=DEV)[None, :, None]
    c = torch.randn((10, 3), generator=g, dtype=F64).to(DEV)
    lo = (0.05 + 0.4 * torch.rand(3, generator=g, dtype=F64)).to(DEV)
    hi = (0.55 + 0.4 * torch.rand(3, generator=g, dtype=F64)).to(DEV)
    powers = [(i, j) for i in range(4) for j in range(4 - i)]
    f = sum(c[k] * (x ** i) * (y ** j) for k, (i, j) in enumerate(powers))
    f = f - f.amin((0, 1))
    f = f / f.amax((0, 1)).clamp_min(1e-12)
    return lo + (hi - lo) * f


def _problem(h, w, seed):
    """(image, trimap, alpha) float64 on the GPU."""
    g = torch.Generator().manual_seed(seed)
    gd = torch.Generator(device=DEV).manual_seed(seed)
    rng = random.Random(seed)
    s = min(h, w)
    sigma, band = (3.0, 10.0) if s >= 400 else (2.0, 3.0)
    half = 2.33 * sigma + band
    target = rng.uniform(0.05, 0.25) * h * w
    r_lo, r_hi = max(0.06 * s, half + 4), max(0.25 * s, half + 8)
    d = torch.full((h, w), -1e3, dtype=F64, device=DEV)
    ys = torch.arange(h, dtype=F64, device=DEV)[:, None]
    xs = torch.arange(w, dtype=F64, device=DEV)[None, :]
    done, first = 0.0, None
    while done < target and done >= 0.0:
        ry, rx = rng.uniform(r_lo, r_hi), rng.uniform(r_lo, r_hi)
        cy, cx, th = rng.uniform(0.1, 0.9) * h, rng.uniform(0.1, 0.9) * w, rng.uniform(0, math.pi)
        reach = max(ry, rx) + half + 2
        y0, y1 = max(int(cy - reach), 0), min(int(cy + reach) + 1, h)
        x0, x1 = max(int(cx - reach), 0), min(int(cx + reach) + 1, w)
        dy, dx = ys[y0:y1] - cy, xs[:, x0:x1] - cx
        u = (dx * math.cos(th) + dy * math.sin(th)) / rx
        v = (-dx * math.sin(th) + dy * math.cos(th)) / ry
        rho = (u * u + v * v).sqrt().clamp_min(1e-6)
        grad = ((u / rx) ** 2 + (v / ry) ** 2).sqrt().clamp_min(1e-9)
        d[y0:y1, x0:x1] = torch.maximum(d[y0:y1, x0:x1], (1 - rho) * rho / grad)
        first = first or (int(cy), int(cx))
        done += math.pi * (ry + rx) * 2 * half
    alpha = 0.5 * torch.erfc(-d / (sigma * math.sqrt(2.0)))
    alpha = torch.where(alpha > 0.99, 1.0, torch.where(alpha < 0.01, 0.0, alpha))
    trimap = torch.where(d > half, 1.0, torch.where(d < -half, 0.0, 0.5)).to(F64)
    # both classes present
    trimap[first[0], first[1]] = 1.0
    trimap[0, 0] = 0.0
    noise = 0.02 * torch.randn((2, h, w, 3), generator=gd, dtype=F64, device=DEV)
    fg = (_colour_field(g, h, w) + noise[0]).clamp(0, 1)
    bg = (_colour_field(g, h, w) + noise[1]).clamp(0, 1)
    image = (fg * alpha[..., None] + bg * (1 - alpha[..., None])).clamp(0, 1)
    return image.contiguous(), trimap.contiguous(), alpha.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    probs = [_problem(h, w, (seed * 1009 + k) % (1 << 31)) for k, (h, w) in enumerate(_sizes(case))]
    image, trimap, alpha = probs[0]
    st = {"case": case, "image": image, "trimap": trimap}
    gd = torch.Generator(device=DEV).manual_seed(seed + 77)
    if kind == "soft":
        st["images"] = [p[0] for p in probs]
        st["trimaps"] = [p[1] for p in probs]
    elif kind == "grad":
        st["images"] = torch.stack([p[0] for p in probs]).float().requires_grad_(True)
        st["trimaps"] = torch.stack([p[1] for p in probs]).float()
        st["g"] = torch.randn(st["trimaps"].shape, generator=gd, device=DEV)
    elif kind == "vcycle":
        A, _b = pm.make_linear_system(pm.cf_laplacian(image), trimap.cpu().numpy())
        st["M"] = pm.vcycle(A, (case["h"], case["w"]))
        st["r"] = torch.randn(case["h"] * case["w"], generator=gd, dtype=F64, device=DEV)
        st["M"](st["r"])      # builds the hierarchy, which the handle keeps
    elif kind == "lkm":
        st["op"] = pm.lkm_laplacian(image, radius=case["radius"], return_diagonal=False)
        st["p"] = torch.rand(case["h"] * case["w"], generator=gd, dtype=F64, device=DEV)
    elif kind in ("fg", "fgj"):
        st["image"], st["alpha"] = image.float(), alpha.float()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "soft":
        return pm.solve_alpha(st["images"], st["trimaps"], precision=case["precision"])
    if kind == "hard":
        return pm.estimate_alpha_cf(st["image"], st["trimap"])
    if kind == "grad":
        x = pm.cf_alpha(st["images"], st["trimaps"])
        grad, = torch.autograd.grad(x, st["images"], st["g"])
        return {"alpha": x.detach(), "grad": grad}
    if kind == "vcycle":
        return st["M"](st["r"])
    if kind == "laplacian":
        indptr, indices, data = device_csr_arrays(pm.cf_laplacian(st["image"]))
        return {"indptr": indptr, "indices": indices, "data": data}
    if kind == "lkm":
        return st["op"](st["p"])
    if kind == "knn":
        indptr, indices, data = device_csr_arrays(pm.knn_laplacian(st["image"]))
        return {"indptr": indptr, "indices": _padded(indices, indptr), "data": _padded(data, indptr)}
    if kind == "fg":
        return pm.estimate_foreground_ml(st["image"], st["alpha"],
                                         return_background=case["background"])
    return pm.estimate_foreground_ml_cupy(st["image"], st["alpha"], to_numpy=False,
                                          return_background=case["background"])


def _padded(a, indptr):
    """`a` at the largest size that a knn matrix can have (20 + 10 neighbours
    and their reverse entries): the number of entries varies with the image."""
    return torch.nn.functional.pad(a, (0, 60 * (len(indptr) - 1) - len(a)))


# --------------------------------------------------------------------------
# The same in plain torch, in 64 bits
# --------------------------------------------------------------------------

def _laplacian25(image, eps=EPS):
    """(h, w, 5, 5) entries of the closed-form Laplacian (Levin et al.)."""
    h, w, _ = image.shape
    shifts = [(dy, dx) for dy in range(3) for dx in range(3)]
    c = torch.stack([image[dy:dy + h - 2, dx:dx + w - 2] for dy, dx in shifts], 2)
    c = c - c.mean(2, keepdim=True)
    cov = torch.einsum("yxki,yxkj->yxij", c, c) + eps * torch.eye(3, dtype=F64, device=DEV)
    inv = _inverse3(cov / 9)
    m = (1 + torch.einsum("yxki,yxij,yxlj->yxkl", c, inv, c)) / 9
    V = torch.zeros((h, w, 5, 5), dtype=F64, device=DEV)
    parts = {}
    for k, (ky, kx) in enumerate(shifts):
        for l, (ly, lx) in enumerate(shifts):
            v = (1.0 if k == l else 0.0) - m[:, :, k, l]
            v = torch.nn.functional.pad(v, (kx, 2 - kx, ky, 2 - ky))
            parts.setdefault((ly - ky + 2, lx - kx + 2), []).append(v)
    cols = [sum(parts[(a, b)]) if (a, b) in parts else V[:, :, a, b]
            for a in range(5) for b in range(5)]
    return torch.stack(cols, 2).reshape(h, w, 5, 5)


def _inverse3(a):
    """Inverse of symmetric 3x3 matrices by the adjugate."""
    c0 = torch.linalg.cross(a[..., 1, :], a[..., 2, :])
    c1 = torch.linalg.cross(a[..., 2, :], a[..., 0, :])
    c2 = torch.linalg.cross(a[..., 0, :], a[..., 1, :])
    det = (a[..., 0, :] * c0).sum(-1)[..., None, None]
    return torch.stack([c0, c1, c2], -1) / det


def _apply25(V, x):
    xp = torch.nn.functional.pad(x, (2, 2, 2, 2))
    return (V * xp.unfold(0, 5, 1).unfold(1, 5, 1)).sum((2, 3))


def _solve25(V, b, keep, budget):
    """Jacobi-preconditioned cg on the pixels of `keep` to 1e-13, or None."""
    end = time.monotonic() + budget
    inv = keep / V[:, :, 2, 2].clamp_min(1e-300)
    x = torch.zeros_like(b)
    r = b * keep
    z = r * inv
    p, rz, nb = z.clone(), (r * z).sum(), r.norm()
    for it in range(200000):
        ap = _apply25(V, p) * keep
        a = rz / (p * ap).sum()
        x, r = x + a * p, r - a * ap
        z = r * inv
        rz, old = (r * z).sum(), rz
        p = z + (rz / old) * p
        if it % 50 == 49:
            if float(r.norm()) <= 1e-13 * float(nb):
                return x
            if time.monotonic() > end:
                return None
    return None


def _soft_system(image, trimap):
    V = _laplacian25(image)
    known = ((trimap >= 0.9) | (trimap <= 0.1)).to(F64)
    V[:, :, 2, 2] += LAMBDA * known
    return V, LAMBDA * (trimap >= 0.9).to(F64)


def _soft_exact(image, trimap, budget):
    V, b = _soft_system(image, trimap)
    return _solve25(V, b, torch.ones_like(b), budget)


def _hard_exact(image, trimap, budget):
    V = _laplacian25(image)
    known = (trimap >= 0.9) | (trimap <= 0.1)
    b = -_apply25(V, (trimap >= 0.9).to(F64))
    x = _solve25(V, b, (~known).to(F64), budget)
    return None if x is None else torch.where(known, trimap, x).clamp(0, 1)


def _grad_exact(images, trimaps, g, budget):
    xs, grads = [], []
    for image, trimap, gk in zip(images.double(), trimaps.double(), g.double()):
        V, b = _soft_system(image, trimap)
        x = _solve25(V, b, torch.ones_like(b), budget)
        mu = None if x is None else _solve25(V, gk, torch.ones_like(b), budget)
        if mu is None:
            return None
        leaf = image.detach().clone().requires_grad_(True)
        (mu * _apply25(_laplacian25(leaf), x)).sum().backward()
        xs.append(x)
        grads.append(-leaf.grad)
    return {"alpha": torch.stack(xs), "grad": torch.stack(grads)}


_WEIGHTS = [(oy, ox, (2 - abs(oy)) * (2 - abs(ox)) / 16) for oy in (-1, 0, 1) for ox in (-1, 0, 1)]


def _down(f):
    h2, w2 = f.shape[0] // 2, f.shape[1] // 2
    fp = torch.nn.functional.pad(f, (1, 1, 1, 1))
    return sum(wt * fp[1 + oy:1 + oy + 2 * h2:2, 1 + ox:1 + ox + 2 * w2:2][:h2, :w2]
               for oy, ox, wt in _WEIGHTS)


def _up(c, h, w):
    h2, w2 = c.shape
    fp = torch.zeros((h + 3, w + 3), dtype=F64, device=DEV)
    for oy, ox, wt in _WEIGHTS:
        fp[1 + oy:1 + oy + 2 * h2:2, 1 + ox:1 + ox + 2 * w2:2][:h2, :w2] += wt * c
    return fp[1:h + 1, 1:w + 1]


def _coarse25(V):
    """R A P as a 5x5 stencil, found by probing with 25 interleaved combs."""
    h, w = V.shape[:2]
    h2, w2 = h // 2, w // 2
    out = torch.zeros((h2, w2, 5, 5), dtype=F64, device=DEV)
    yy = torch.arange(h2, device=DEV)[:, None]
    xx = torch.arange(w2, device=DEV)[None, :]
    for a in range(5):
        for b in range(5):
            comb = ((yy % 5 == a) & (xx % 5 == b)).to(F64)
            col = _down(_apply25(V, _up(comb, h, w)))
            dy = (a - yy + 2) % 5 + 0 * xx       # offset + 2 of the comb pixel within reach
            dx = (b - xx + 2) % 5 + 0 * yy
            inside = ((yy + dy - 2 >= 0) & (yy + dy - 2 < h2) & (xx + dx - 2 >= 0) &
                      (xx + dx - 2 < w2)).to(F64)
            flat = (dy * 5 + dx).reshape(h2, w2, 1)
            out.view(h2, w2, 25).scatter_add_(2, flat, (col * inside)[..., None])
    return out


def _vcycle_exact(V, b, omega=0.8):
    h, w = b.shape
    if h * w <= 64:
        eye = torch.eye(h * w, dtype=F64, device=DEV).reshape(-1, h, w)
        dense = torch.stack([_apply25(V, e).reshape(-1) for e in eye], 1)
        return torch.linalg.solve(dense, b.reshape(-1)).reshape(h, w)
    d = V[:, :, 2, 2]
    x = omega * b / d
    x = x + _up(_vcycle_exact(_coarse25(V), _down(b - _apply25(V, x)), omega), h, w)
    return x + omega * (b - _apply25(V, x)) / d


def _box(a, r, full):
    """Box sums over (2r+1)^2 windows of a (channels, h, w) array."""
    if full:
        a = torch.nn.functional.pad(a, (2 * r, 2 * r, 2 * r, 2 * r))
    k = 2 * r + 1
    rows = sum(a[:, i:a.shape[1] - k + 1 + i] for i in range(k))
    return sum(rows[:, :, i:rows.shape[2] - k + 1 + i] for i in range(k))


def _lkm_exact(image, p, r):
    I = image.permute(2, 0, 1)
    h, w = I.shape[1:]
    area = (2 * r + 1) ** 2
    mean = _box(I, r, False) / area
    prod = (I[:, None] * I[None, :]).reshape(9, h, w)
    hv, wv = mean.shape[1:]
    cov = _box(prod, r, False).reshape(3, 3, hv, wv) / area - mean[:, None] * mean[None, :]
    V = _inverse3(cov.permute(2, 3, 0, 1) + EPS / area * torch.eye(3, dtype=F64, device=DEV))
    V = V.permute(2, 3, 0, 1) / area
    p = p.reshape(1, h, w)
    ps, pI = _box(p, r, False), _box(p * I, r, False)
    q = torch.einsum("ijyx,jyx->iyx", V, pI - ps * mean)       # area * cov(p, I) / area
    out = _box(torch.ones_like(ps), r, True) * p
    out = out - (I * _box(q, r, True)).sum(0, keepdim=True)
    out = out - _box(ps / area - (q * mean).sum(0, keepdim=True), r, True)
    return out.reshape(-1)


def _knn_exact(image, ks=(20, 10), weights=(2.0, 0.1)):
    h, w, _ = image.shape
    n = h * w
    x = torch.linspace(0, 1, w, dtype=F64, device=DEV).repeat(h)
    y = torch.linspace(0, 1, h, dtype=F64, device=DEV).repeat_interleave(w)
    keys = []
    for k, dw in zip(ks, weights):
        f = torch.cat([image.reshape(n, 3), (dw * x)[:, None], (dw * y)[:, None]], 1).float()
        for i0 in range(0, n, 2048):
            i1 = min(i0 + 2048, n)
            dist = torch.zeros((i1 - i0, n), dtype=F64, device=DEV)
            for c in range(5):
                dc = f[i0:i1, c, None] - f[None, :, c]
                dist += (dc * dc).double()
            nbr = dist.topk(k, 1, largest=False).indices.reshape(-1)
            i = torch.arange(i0, i1, device=DEV).repeat_interleave(k)
            keys += [i * n + nbr, nbr * n + i]
    keys, counts = torch.unique(torch.cat(keys), return_counts=True)
    rows, cols = keys // n, keys % n
    rs = torch.zeros(n, dtype=F64, device=DEV).index_add_(0, rows, counts.to(F64))
    # I - W with the identity as entries of its own row; every pixel is its
    # own nearest neighbour, so the diagonal is always stored.
    data = (rows == cols).to(F64) - counts.to(F64) / rs[rows]
    return {"indptr": None, "indices": None, "data": torch.nn.functional.pad(data, (0, 60 * n - len(data)))}


def _levels(h, w):
    n = math.ceil(math.log2(max(h, w)))
    return [(round(h ** (i / n)), round(w ** (i / n))) for i in range(n + 1)]


def _resize(a, h, w):
    ys = (torch.arange(h, device=a.device) * a.shape[0] // h).clamp_max(a.shape[0] - 1)
    xs = (torch.arange(w, device=a.device) * a.shape[1] // w).clamp_max(a.shape[1] - 1)
    return a[ys][:, xs]


def _fg_terms(image, alpha, reg=1e-5):
    """Neighbour indices, their weights, the data term and the inverse 2x2
    matrices of every pixel of a level, flattened."""
    h, w = alpha.shape
    y = torch.arange(h, device=DEV)[:, None].expand(h, w)
    x = torch.arange(w, device=DEV)[None, :].expand(h, w)
    nbr = torch.stack([y * w + (x - 1).clamp_min(0), y * w + (x + 1).clamp_max(w - 1),
                       (y - 1).clamp_min(0) * w + x, (y + 1).clamp_max(h - 1) * w + x],
                      2).reshape(-1, 4)
    a0 = alpha.reshape(-1)
    a1 = 1 - a0
    da = reg + (a0[:, None] - a0[nbr]).abs()
    s = da.sum(1)
    img = image.reshape(-1, 3)
    base = torch.stack([a0[:, None] * img, a1[:, None] * img], 1)
    m00, m01, m11 = a0 * a0 + s, a0 * a1, a1 * a1 + s
    det = m00 * m11 - m01 * m01
    inv = torch.stack([m11, -m01, -m01, m00], 1).reshape(-1, 2, 2) / det[:, None, None]
    return nbr, da, base, inv


def _fg_step(FB, nbr, da, base, inv):
    b = base + (da[:, :, None, None] * FB[nbr]).sum(1)
    return (inv @ b).clamp(0, 1)


def _fg_exact(image, alpha, background):
    """Gauss-Seidel in raster order: the pixels of one anti-diagonal at once."""
    image, alpha = image.double(), alpha.double()
    h0, w0 = alpha.shape
    seeds = []
    for mask in (alpha > 0.9, alpha < 0.1):
        seeds.append((image * mask[..., None]).sum((0, 1)) / (mask.sum() + 1e-5))
    FB = torch.stack(seeds)[None, None]
    for h, w in _levels(h0, w0):
        nbr, da, base, inv = _fg_terms(_resize(image, h, w), _resize(alpha, h, w))
        FB = _resize(FB, h, w).reshape(-1, 2, 3).contiguous()
        s = (torch.arange(h, device=DEV)[:, None] + torch.arange(w, device=DEV)[None, :]).reshape(-1)
        order = torch.argsort(s, stable=True)
        bounds = np.cumsum([0] + torch.bincount(s).tolist())
        nbr, da, base, inv = nbr[order], da[order], base[order], inv[order]
        for _ in range(10 if max(h, w) <= 32 else 2):
            for a, b in zip(bounds[:-1], bounds[1:]):
                FB[order[a:b]] = _fg_step(FB, nbr[a:b], da[a:b], base[a:b], inv[a:b])
        FB = FB.reshape(h, w, 2, 3)
    F, B = FB[:, :, 0], FB[:, :, 1]
    return (F, B) if background else F


def _fgj_exact(image, alpha, background):
    """Jacobi sweeps from the colour of pixel (0, 0); every level starts from,
    and the result is, the second newest iterate of the last sweeps."""
    image, alpha = image.double(), alpha.double()
    h0, w0 = alpha.shape
    n = (max(w0, h0) - 1).bit_length()
    FB = image[:1, :1, None].expand(1, 1, 2, 3)
    for i in range(n + 1):
        h, w = round(h0 ** (i / n)), round(w0 ** (i / n))
        terms = _fg_terms(_resize(image, h, w), _resize(alpha, h, w))
        new = _resize(FB, h, w).reshape(-1, 2, 3)
        for _ in range(10 if min(h, w) <= 32 else 2):
            old, new = new, _fg_step(new, *terms)
        FB = old.reshape(h, w, 2, 3)
    F, B = FB[:, :, 0], FB[:, :, 1]
    return (F, B) if background else F


def exact(case, seed):
    kind = case["kind"]
    if kind == "soft" and sum(h * w for h, w in _sizes(case)) > 4e6:
        return None          # beyond the time that a plain solve may take
    st = prepare(case, seed)
    if kind == "soft":
        budget = 15.0 / len(st["images"])
        xs = [_soft_exact(i, t, budget) for i, t in zip(st["images"], st["trimaps"])]
        return [None if x is None else x.clamp(0, 1) for x in xs]
    if kind == "hard":
        return _hard_exact(st["image"], st["trimap"], 15.0)
    if kind == "grad":
        return _grad_exact(st["images"].detach(), st["trimaps"], st["g"], 7.0 / case["count"])
    if kind == "vcycle":
        V, _b = _soft_system(st["image"], st["trimap"])
        return _vcycle_exact(V, st["r"].reshape(case["h"], case["w"])).reshape(-1)
    if kind == "laplacian":
        return {"indptr": None, "indices": None, "data": _laplacian25(st["image"]).reshape(-1)}
    if kind == "lkm":
        return _lkm_exact(st["image"], st["p"], case["radius"])
    if kind == "knn":
        return _knn_exact(st["image"])
    if kind == "fg":
        return _fg_exact(st["image"], st["alpha"], case["background"])
    return _fgj_exact(st["image"], st["alpha"], case["background"])
