"""The calls a user of this package makes, with the sizes they make them at.

Matting has four kinds of work, and each has its cases here: assembling the
Laplacian of a new image, solving for the matte (one image, a batch, the
drop-in cgSolve of the reference's layout), differentiating through both, and
the plain matrix product that a caller's own iteration uses.  Every case goes
through gpumatting_b200.api or gpumatting_b200.autograd.

Inputs follow the recipe of gpumatting_b200.synth (smooth colour fields
blended by a sigmoid matte, sensor noise, about 10 % scribbled in strokes),
made on the GPU from the seed.  Stores, batches and output buffers are made
once in prepare(), as a program that processes a stream of images keeps them;
images, scribbles and initial guesses are a pass's inputs.
"""
import math

import numpy as np
import torch

from gpumatting_b200 import api, autograd

DEV = "cuda"
GAMMA = 100.0
EPS = 1e-5  # where a case does not say


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
# A matte is solved either to a tolerance or for a fixed number of iterations.
# rtol 1e-9 is what an accurate matte takes: it puts alpha within about 1e-4 of
# the direct solution, where 1e-6 leaves it 0.1 to 0.3 away at weakly
# constrained pixels.  A fixed count (rtol 0) is a time budget per image, the
# way the reference's cgSolve is called.
ACCURATE = 1e-9
BUDGET = {"mg": 20, "cg": 100}


def listed():
    return [
        # A thumbnail: the smallest assembly, bound by launches.
        {"name": "assemble_thumb", "kind": "assemble", "w": 160, "h": 120, "prec": "fp16", "image": "rgb8",
         "weights": "map", "eps": 1e-5},
        # A video frame, in the store the mixed solvers use.
        {"name": "assemble_1080p", "kind": "assemble", "w": 1920, "h": 1080, "prec": "fp16", "image": "rgb8",
         "weights": "map", "eps": 1e-5},
        # A photograph of ragged size with float colours and per-pixel weights
        # (the inputs of the differentiable path), FP32 store.
        {"name": "assemble_photo_fp32", "kind": "assemble", "w": 4001, "h": 2999, "prec": "fp32", "image": "rgba32f",
         "weights": "maps", "eps": 1e-7},
        # The reference's own 25-band layout and arithmetic, at the size of
        # its sample photograph.
        {"name": "bands25_reference", "kind": "bands", "w": 800, "h": 552, "arith": "reference", "eps": 1e-5},
        # One matrix product of a caller's own iteration, operands beyond L2.
        {"name": "apply_photo", "kind": "apply", "w": 3001, "h": 2003, "prec": "fp16", "true_op": False},
        # A new image to its matte, assembly and solve: an interactive preview
        # of odd size, the plain method's standard size, a video frame.
        {"name": "matte_preview", "kind": "matte", "w": 317, "h": 211, "prec": "fp16", "solver": "mg", "eps": 1e-5,
         "rtol": ACCURATE},
        {"name": "matte_vga", "kind": "matte", "w": 640, "h": 480, "prec": "fp16", "solver": "mg", "eps": 1e-5,
         "rtol": ACCURATE},
        {"name": "matte_1080p", "kind": "matte", "w": 1920, "h": 1080, "prec": "fp16", "solver": "mg", "eps": 1e-5,
         "rtol": ACCURATE},
        # The largest single image, within a time budget.
        {"name": "matte_4096_budget", "kind": "matte", "w": 4096, "h": 4096, "prec": "fp16", "solver": "mg",
         "eps": 1e-7, "rtol": 0.0},
        # The video frame with the unpreconditioned fused CG (the reference's
        # algorithm) for a fixed number of iterations.
        {"name": "matte_1080p_cg_budget", "kind": "matte", "w": 1920, "h": 1080, "prec": "fp16", "solver": "cg",
         "eps": 1e-5, "rtol": 0.0},
        # A training step through the matte: forward, loss, backward to the
        # image and to the scribble weights.
        {"name": "gradient_512", "kind": "grad", "w": 512, "h": 512, "prec": "fp16", "eps": 1e-3},
        # A folder of images of uneven sizes in one call.
        {"name": "batch_uneven", "kind": "batch", "count": 12, "lo": 256, "hi": 1024, "prec": "fp16"},
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["assemble", "matte", "bands", "apply", "grad", "batch"], [25, 40, 8, 9, 10, 8])[0]
    prec = rng.choice(["fp16", "fp16", "bf16", "fp32"])
    if kind == "assemble":
        return {"kind": kind, "w": _side(rng, 64, 4096), "h": _side(rng, 48, 4096), "prec": prec,
                "image": rng.choice(["rgb8", "rgb8", "rgba32f"]), "weights": rng.choice(["map", "map", "maps"]),
                "eps": rng.choice([1e-5, 1e-6, 1e-7])}
    if kind == "matte":
        solver = rng.choice(["mg", "mg", "mg", "cg"])
        return {"kind": kind, "w": _side(rng, 96, 2048), "h": _side(rng, 96, 2048), "prec": prec, "solver": solver,
                "eps": 1e-5, "rtol": 0.0 if solver == "cg" or rng.random() < 0.4 else ACCURATE}
    if kind == "bands":
        return {"kind": kind, "w": _side(rng, 64, 2048), "h": _side(rng, 48, 2048),
                "arith": rng.choice(["reference", "fp64"]), "eps": 1e-5}
    if kind == "apply":
        return {"kind": kind, "w": _side(rng, 320, 4096), "h": _side(rng, 240, 4096), "prec": prec,
                "true_op": rng.random() < 0.4}
    if kind == "grad":
        return {"kind": kind, "w": _side(rng, 96, 768), "h": _side(rng, 96, 768), "prec": prec, "eps": 1e-3}
    lo = rng.choice([128, 256])
    return {"kind": kind, "count": rng.randint(3, 16), "lo": lo, "hi": rng.choice([512, 768, 1024]), "prec": prec}


# ---------------------------------------------------------------------------
# Inputs (the recipe of gpumatting_b200.synth, on the GPU)
# ---------------------------------------------------------------------------
def _field(rng, W, H):
    g = torch.from_numpy(rng.uniform(0.0, 255.0, size=(8, 8, 3))).to(DEV)

    def axis(n):
        t = torch.arange(n, device=DEV, dtype=torch.float64) * (7.0 / max(n - 1, 1))
        i = t.floor().clamp(0, 6).long()
        return i, t - i

    (y, fy), (x, fx) = axis(H), axis(W)
    fy, fx = fy[:, None, None], fx[None, :, None]
    top = g[y][:, x] * (1 - fx) + g[y][:, x + 1] * fx
    bot = g[y + 1][:, x] * (1 - fx) + g[y + 1][:, x + 1] * fx
    return (top * (1 - fy) + bot * fy).float()


def _smooth(z, sigma):
    """Gaussian smoothing along both axes, edges mirrored; a plain sum of
    shifted copies, so that the same seed gives the same bits everywhere."""
    for dim in (0, 1):
        n = z.shape[dim]
        r = min(int(3 * sigma), n - 1)
        k = [math.exp(-0.5 * (d / sigma) ** 2) for d in range(-r, r + 1)]
        s = sum(k)
        idx = torch.arange(-r, n + r, device=DEV)
        idx = idx.abs()
        idx = torch.where(idx > n - 1, 2 * (n - 1) - idx, idx)
        p = z.index_select(dim, idx)
        out = torch.zeros_like(z)
        for d in range(2 * r + 1):
            out += p.narrow(dim, d, n) * (k[d] / s)
        z = out
    return z


def _strokes(rng, W, H, frac, eligible):
    """Mask of 20 smooth strokes, 7 px wide."""
    n = max(8, int(frac * W * H / (140 * max(eligible, 0.05))))
    t = np.arange(n)
    m = torch.zeros((H, W), device=DEV)
    start = rng.uniform(0.0, 1.0, size=(20, 2)) * np.array([W, H])
    turn, bend = rng.uniform(0.0, 2.0 * np.pi, size=20), rng.normal(0.0, 1.0, size=20)
    for s in range(20):
        a = turn[s] + bend[s] * 2.0 * t / n
        px = np.mod(start[s, 0] + np.cumsum(np.cos(a)), W).astype(np.int64).clip(0, W - 1)
        py = np.mod(start[s, 1] + np.cumsum(np.sin(a)), H).astype(np.int64).clip(0, H - 1)
        m.view(-1)[torch.from_numpy(py * W + px).to(DEV)] = 1.0
    for dim in (0, 1):
        n = m.shape[dim]
        idx = (torch.arange(-3, n + 3, device=DEV)).clamp(0, n - 1)
        p = m.index_select(dim, idx)
        m = torch.stack([p.narrow(dim, d, n) for d in range(7)]).amax(0)
    return m > 0


def _problem(W, H, seed):
    """Image (uint8), scribbles (0 / 128 / 255) and the matte they came from."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    large = W * H >= 2048 * 2048
    z = torch.rand((H, W), generator=gen, device=DEV) * 2 - 1
    z = _smooth(z, 24.0 if large else 6.0)
    z = z - z.mean()
    alpha = torch.sigmoid(8.0 * z / z.std())
    img = alpha[..., None] * _field(rng, W, H) + (1 - alpha[..., None]) * _field(rng, W, H)
    img = (img + 4.0 * torch.randn((H, W, 3), generator=gen, device=DEV)).round().clamp(0, 255).to(torch.uint8)
    fg, bg = alpha > 0.98, alpha < 0.02
    mask = _strokes(rng, W, H, 0.05 if large else 0.10, float((fg | bg).float().mean()))
    scr = torch.full((H, W), 128, dtype=torch.uint8, device=DEV)
    scr[mask & bg] = 0
    scr[mask & fg] = 255
    if not bool((scr != 128).any()):
        scr[H // 2, W // 2] = 255
    return img, scr, alpha


def _float_image(img):
    out = torch.ones((img.shape[0], img.shape[1], 4), device=DEV)
    out[..., :3] = img.float() / 255.0
    return out


def _weights(scr):
    """Per-pixel weights and targets of a scribble map."""
    gamma = torch.where(scr != 128, GAMMA, 0.0).float()
    return gamma, (scr == 255).float()


def _sizes(case):
    """The sizes are the case's (a folder keeps its images); the seed draws their contents."""
    rng = np.random.default_rng(case["count"] * 1000 + case["lo"] + case["hi"])
    return [(int(w), int(h)) for w, h in rng.integers(case["lo"], case["hi"] + 1, size=(case["count"], 2))]


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k == "batch":
        s["sizes"] = _sizes(case)
        s["batch"] = api.LevinBatch(s["sizes"], case["prec"])
        s["alpha"] = []
        for i, (w, h) in enumerate(s["sizes"]):
            img, scr, _ = _problem(w, h, seed * 100 + i)
            s["batch"].assemble(i, img, scr, eps=EPS, gamma_value=GAMMA)
            s["alpha"].append(torch.empty((h, w), device=DEV))
        return s
    W, H = case["w"], case["h"]
    eps = case.get("eps", EPS)
    img, scr, gt = _problem(W, H, seed)
    if k == "grad":
        gamma, target = _weights(scr)
        s["image"] = (img.float() / 255.0).requires_grad_()
        s["gamma"], s["target"] = gamma.requires_grad_(), target
        s["gt"] = gt
        return s
    s["img"], s["scr"] = img, scr
    if k == "bands":
        s["img"] = _float_image(img)
        return s
    s["store"] = api.LevinStore(W, H, case["prec"])
    if k == "assemble":
        if case["image"] == "rgba32f":
            s["img"] = _float_image(img)
        s["scribbles"] = {"scribbles": scr, "gamma_value": GAMMA}
        if case["weights"] == "maps":
            gamma, target = _weights(scr)
            s["scribbles"] = {"gamma_map": gamma, "s_map": target}
        st = s["store"]
        # Views of the store's planes without the padding columns, which no call
        # writes.  They do not own the memory, so each keeps the store alive.
        s["planes"] = {n: st.planes(n)[..., :W] for n in ("w", "w32", "gamma", "b", "d", "d32")}
        for view in s["planes"].values():
            view.store = st
        if case["prec"] == "fp32":
            del s["planes"]["w"]  # the same memory as w32
    elif k == "apply":
        s["store"].assemble(img, scr, eps=eps, gamma_value=GAMMA)
        pw = (W + 3) // 4 * 4
        gen = torch.Generator(device=DEV).manual_seed(seed + 1)
        s["x"] = torch.rand((H, pw), generator=gen, device=DEV)
        s["y"] = torch.zeros((H, pw), device=DEV)
    else:
        s["alpha"] = torch.empty((H, W), device=DEV)
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "assemble":
        s["store"].assemble(s["img"], eps=case["eps"], **s["scribbles"])
        return s["planes"]
    if k == "apply":
        s["store"].apply(s["x"], s["y"], true_op=case["true_op"])
        return s["y"][:, :case["w"]]
    if k == "bands":
        return api.levin_bands25(s["img"], s["scr"], eps=case["eps"], gamma_value=1.0, arithmetic=case["arith"])
    if k == "matte":
        s["store"].assemble(s["img"], s["scr"], eps=case["eps"], gamma_value=GAMMA)
        s["alpha"].fill_(0.5)
        s["store"].solve(s["alpha"], case["solver"], rtol=case["rtol"],
                         max_iters=20000 if case["rtol"] > 0 else BUDGET[case["solver"]])
        return s["alpha"]
    if k == "grad":
        image, gamma = s["image"], s["gamma"]
        image.grad = gamma.grad = None
        alpha = autograd.levin_matte(image, gamma, s["target"], eps=case["eps"], precision=case["prec"],
                                     rtol=ACCURATE)
        loss = ((alpha - s["gt"]) ** 2).mean()
        loss.backward()
        return {"alpha": alpha.detach(), "dimage": image.grad, "dgamma": gamma.grad}
    for a in s["alpha"]:
        a.fill_(0.5)
    s["batch"].solve(s["alpha"], "mg", rtol=ACCURATE, max_iters=20000)
    return s["alpha"]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
# Bytes per pixel and operations per pixel of the parts.  An assembly reads the
# image and the scribbles and writes its planes; its operations are the window
# statistics, their inverses and the 12 coupling sums in 64 bits.  A CG
# iteration on 2-byte planes moves 60 B (planes 24, diagonal 4, vectors 32), a
# multigrid iteration with the outer product on the FP32 planes 180 B (156 B on
# the FP16 planes); both do about 2 operations per coupling and vector entry.
def _esize(case):
    return 4 if case["prec"] == "fp32" else 2


def _assembly(case, n):
    esize = 0 if case["prec"] == "fp32" else 2
    image = 16 if case.get("image") == "rgba32f" else 3
    weights = 8 if case.get("weights") == "maps" else 1
    return n * (image + weights + 12 * (esize + 4) + 16), n * 500


# Multigrid iterations to 1e-9 grow slowly with the size; this is what they
# come to on these inputs.
def _mg_iterations(n):
    return 60.0 * n ** 0.107


def work(case):
    k = case["kind"]
    if k == "batch":
        by = fl = 0.0
        for w, h in _sizes(case):
            n, it = w * h, _mg_iterations(w * h)
            by, fl = by + n * it * (132 + 24 * _esize(case) // 2), fl + n * it * 200
        return {"bytes": by, "flops": fl}
    n = case["w"] * case["h"]
    if k == "assemble":
        by, fl = _assembly(case, n)
    elif k == "bands":
        by, fl = n * (16 + 1 + 25 * 4 + 4), n * 1500
    elif k == "apply":
        by, fl = n * (12 * (4 if case["true_op"] else _esize(case)) + 12), n * 50
    elif k == "matte":
        by, fl = _assembly(case, n)
        if case["solver"] == "cg":
            by, fl = by + n * BUDGET["cg"] * (36 + 12 * _esize(case)), fl + n * BUDGET["cg"] * 70
        else:
            it = BUDGET["mg"] if case["rtol"] == 0 else _mg_iterations(n)
            outer = 24 if case["rtol"] == 0 and case["prec"] == "fp16" else 48
            by, fl = by + n * it * (84 + outer + 24 * _esize(case)), fl + n * it * 200
    else:
        by, fl = _assembly(dict(case, image="rgba32f", weights="maps"), n)
        it = 2 * _mg_iterations(n)
        by, fl = by + n * (it * (132 + 24 * _esize(case)) + 60), fl + n * (it * 200 + 500)
    return {"bytes": float(by), "flops": float(fl)}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
_OFFS = [(((k + 2) % 5) - 2, (k + 2) // 5) for k in range(1, 13)]  # upper couplings (du, dv)


def _couplings(x, eps):
    """12 upper coupling planes of the Levin Laplacian of x (H, W, 3), FP64:
    sum over the 3x3 windows that hold both pixels of
    (1 + (x_i - mu)^T (Sigma + eps / 9)^-1 (x_j - mu)) / 9."""
    H, W, _ = x.shape
    hh, ww = H - 2, W - 2
    planes = [torch.zeros((H, W), dtype=torch.float64, device=x.device) for _ in _OFFS]
    if hh < 1 or ww < 1:
        return planes
    win = [[x[j:j + hh, i:i + ww] for i in range(3)] for j in range(3)]
    mu = sum(win[j][i] for j in range(3) for i in range(3)) / 9.0
    c = {}
    for a in range(3):
        for b in range(a, 3):
            c[a, b] = sum((win[j][i][..., a] - mu[..., a]) * (win[j][i][..., b] - mu[..., b])
                          for j in range(3) for i in range(3)) / 9.0
        c[a, a] = c[a, a] + eps / 9.0
    k00 = c[1, 1] * c[2, 2] - c[1, 2] ** 2
    k01 = c[0, 2] * c[1, 2] - c[0, 1] * c[2, 2]
    k02 = c[0, 1] * c[1, 2] - c[0, 2] * c[1, 1]
    det = c[0, 0] * k00 + c[0, 1] * k01 + c[0, 2] * k02
    k11 = c[0, 0] * c[2, 2] - c[0, 2] ** 2
    k12 = c[0, 1] * c[0, 2] - c[0, 0] * c[1, 2]
    k22 = c[0, 0] * c[1, 1] - c[0, 1] ** 2
    inv = [[k00, k01, k02], [k01, k11, k12], [k02, k12, k22]]
    for j in range(3):
        for i in range(3):
            d = [win[j][i][..., a] - mu[..., a] for a in range(3)]
            g = [(inv[a][0] * d[0] + inv[a][1] * d[1] + inv[a][2] * d[2]) / det for a in range(3)]
            for n, (du, dv) in enumerate(_OFFS):
                i2, j2 = i + du, j + dv
                if 0 <= i2 < 3 and 0 <= j2 < 3:
                    t = 1.0 + sum(g[a] * (win[j2][i2][..., a] - mu[..., a]) for a in range(3))
                    if t.requires_grad:
                        planes[n] = planes[n] + torch.nn.functional.pad(t / 9.0, (i, 2 - i, j, 2 - j))
                    else:
                        planes[n][j:j + hh, i:i + ww] += t / 9.0
    return planes


def _pair(n, H, W):
    """Slices of the pixels that have an n-th upper neighbour, and of those neighbours."""
    du, dv = _OFFS[n]
    i = (slice(0, H - dv), slice(max(0, -du), W - max(0, du)))
    j = (slice(dv, H), slice(max(0, du), W + min(0, du)))
    return i, j


def _row_sums(planes, gamma):
    d = gamma.clone()
    H, W = gamma.shape
    for n, w in enumerate(planes):
        i, j = _pair(n, H, W)
        d[i] += w[i]
        d[j] += w[i]
    return d


def _product(planes, d, x):
    y = d * x
    H, W = x.shape
    for n, w in enumerate(planes):
        i, j = _pair(n, H, W)
        y[i] -= w[i] * x[j]
        y[j] -= w[i] * x[i]
    return y


def _solve(planes, gamma, b, x):
    """Conjugate gradients with the diagonal as preconditioner, to 1e-12 of b."""
    d = _row_sums(planes, gamma)
    m = torch.where(d > 0, 1.0 / d, 0.0)
    r = b - _product(planes, d, x)
    z = m * r
    p, rz, stop = z.clone(), (r * z).sum(), float(b.square().sum()) * 1e-24
    for it in range(40000):
        q = _product(planes, d, p)
        a = rz / (p * q).sum()
        x = x + a * p
        r = r - a * q
        if it % 50 == 49 and float(r.square().sum()) <= stop:
            break
        z = m * r
        rz2 = (r * z).sum()
        p = z + (rz2 / rz) * p
        rz = rz2
    return x


def _cg(planes, gamma, b, x, count):
    d = _row_sums(planes, gamma)
    r = b - _product(planes, d, x)
    p, rr = r.clone(), r.square().sum()
    for _ in range(count):
        q = _product(planes, d, p)
        a = rr / (p * q).sum()
        x = x + a * p
        r = r - a * q
        rr2 = r.square().sum()
        p = r + (rr2 / rr) * p
        rr = rr2
    return x


def _rounded(w, prec):
    """w as a store of this precision holds it, in 64 bits."""
    return w if prec == "fp32" else w.to(torch.float16 if prec == "fp16" else torch.bfloat16).double()


def exact(case, seed):
    k = case["kind"]
    if k == "batch":
        return None
    W, H = case["w"], case["h"]
    s = prepare(case, seed)
    if k == "grad":
        x = s["image"].detach().double().requires_grad_()
        gamma, target = s["gamma"].detach().double(), s["target"].double()
        w = _couplings(x, case["eps"])
        fixed = [p.detach() for p in w]
        half = torch.full((H, W), 0.5, dtype=torch.float64, device=DEV)
        alpha = _solve(fixed, gamma, gamma * target, half)
        lam = _solve(fixed, gamma, 2.0 * (alpha - s["gt"].double()) / (W * H), torch.zeros_like(half))
        e = 0.0
        for n, p in enumerate(w):
            i, j = _pair(n, H, W)
            e = e - (p[i] * (lam[i] - lam[j]) * (alpha[i] - alpha[j])).sum()
        e.backward()
        return {"alpha": alpha, "dimage": x.grad, "dgamma": lam * (target - alpha)}
    img = s["img"]
    x = img.double() / 255.0 if img.dtype == torch.uint8 else img[..., :3].double()
    gamma, target = _weights(s["scr"])
    gamma, target = gamma.double(), target.double()
    if k == "matte" and (case["solver"] == "mg" and case["rtol"] == 0 or W * H > 2_200_000):
        return None
    w = _couplings(x, case.get("eps", EPS))
    if k == "assemble":
        low = [_rounded(p, case["prec"]) for p in w]
        out = {"w": torch.stack(w), "w32": torch.stack(w), "gamma": gamma, "b": gamma * target,
               "d": _row_sums(low, gamma), "d32": _row_sums(w, gamma)}
        if case["prec"] == "fp32":
            del out["w"]
        return out
    if k == "bands":
        gamma = gamma / GAMMA
        a = torch.zeros((25, H, W), dtype=torch.float64, device=DEV)
        for n, p in enumerate(w):
            du, dv = _OFFS[n]
            i, j = _pair(n, H, W)
            a[12 + du + 5 * dv][i] = -p[i]
            a[12 - du - 5 * dv][j] = -p[i]
        a[12] = _row_sums(w, gamma)
        return a.reshape(25, -1), (gamma * target).reshape(-1)
    if k == "apply":
        low = w if case["true_op"] else [_rounded(p, case["prec"]) for p in w]
        return _product(low, _row_sums(low, gamma), s["x"][:, :W].double())
    half = torch.full((H, W), 0.5, dtype=torch.float64, device=DEV)
    if case["rtol"] == 0:
        return _cg(w, gamma, gamma * target, half, BUDGET["cg"])
    return _solve(w, gamma, gamma * target, half)
