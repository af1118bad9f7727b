"""Performance cases of the DIC path through its public Python entry points.

A case is one pass of a user's program: a target frame registered against a
reference on a POI grid (DICFrame.process), the same with a new reference
(a camera loop's reference refresh), the FFT-CC and IC-GN classes used one
after the other (cuFFTCC2D, cuICGN2D), integer-pixel tracking alone
(cuFFTCC2D), and several uneven image pairs in one call (DICBatch).  Geometry
follows the repository's own workloads: the 192x160 check case, the 512x512
pair, 640x480 to 4096x3072 cameras, subset radii 8 to 30, POI steps 3 to 12,
a one-pixel image border around the ROI and a margin of 20.

Images are Gaussian speckle patterns (radius 2-4 px, peaks of 40-200 gray
levels on a background of 20) and their deformed targets (affine plus a
sinusoid: a few pixels of translation, strains and rotations up to 1 %) with
noise of 2 gray levels, made on the GPU from the seed.
"""
import math

import torch

from tw_gb300 import INTERP_BICUBIC, INTERP_BSPLINE, DICBatch, DICFrame, cuFFTCC2D, cuICGN2D, make_params

MARGIN = 20
MAX_ITER = 20
DELTA_P = 0.001


def _case(name, kind, w, h, r, grid, interp="bicubic", host=False):
    return {"name": name, "kind": kind, "w": w, "h": h, "r": r, "grid": grid, "interp": interp, "host": host}


def listed():
    return [
        # a handful of strain-gauge points on a cropped image: one small call, latency counts
        _case("frame_192x160", "frame", 192, 160, 10, 7),
        # a low-resolution measurement, 33x33 subsets every 10 px
        _case("frame_512", "frame", 512, 512, 16, 10),
        # one image of a live VGA camera, from and to host memory
        _case("camera_640x480", "frame", 640, 480, 15, 8, host=True),
        # one image of a 1.3-megapixel camera already on the device
        _case("frame_1280x1024", "frame", 1280, 1024, 15, 8),
        # the B-spline interpolation option on an odd-sized crop
        _case("bspline_1279x1021", "frame", 1279, 1021, 13, 7, interp="bspline"),
        # a dense displacement map of a 4-megapixel image: the benchmark's workload
        _case("frame_2048", "frame", 2048, 2048, 20, 5),
        # coarse speckles: the largest subsets on a ragged ROI, few POIs
        _case("subset61_2045x1531", "frame", 2045, 1531, 30, 11),
        # a 12-megapixel image, the largest frame
        _case("frame_4096x3072", "frame", 4096, 3072, 24, 6),
        # the reference moves on (every image is compared with the one before it)
        _case("refresh_2048x1536", "refresh", 2048, 1536, 17, 6),
        # integer-pixel tracking alone, small subsets on a fine grid
        _case("fftcc_1024x768", "fftcc", 1024, 768, 12, 3),
        # an engine that calls the FFT-CC class and then the IC-GN class
        _case("classes_1280x1024", "classes", 1280, 1024, 11, 6, host=False),
        # several cameras' pairs of uneven sizes and subsets in one call
        {"name": "batch_uneven", "kind": "batch", "interp": "bicubic", "host": False,
         "pairs": "512x384:10:5 1024x768:17:4 1280x1024:15:8 2048x1536:27:9 1024x768:22:12 512x384:13:3"},
    ]


def _pois(w, h, r, grid):
    nx = (w - 2 - 2 * r - 2 * MARGIN) // grid + 1
    ny = (h - 2 - 2 * r - 2 * MARGIN) // grid + 1
    return max(nx, 0) * max(ny, 0), nx, ny


_MOST = 320_000 * 49 * 49  # subset samples of the largest listed frame, nearly


def _draw_geometry(rng, most=_MOST, w_most=4096):
    r = rng.randint(8, 30)
    w = int(round(math.exp(rng.uniform(math.log(192), math.log(w_most)))))
    h = int(round(w * rng.uniform(0.6, 1.0)))
    w, h = max(w, 2 * r + 2 * MARGIN + 40), min(max(h, 2 * r + 2 * MARGIN + 40), 3072)
    grid = rng.randint(3, 12)
    while _pois(w, h, r, grid)[0] * (2 * r + 1) ** 2 > most:
        grid += 1
    return w, h, r, grid


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "refresh", "fftcc", "classes", "batch"])
    if kind == "batch":
        pairs = []
        for _ in range(rng.randint(2, 6)):
            w, h, r, grid = _draw_geometry(rng, _MOST // 8, 2048)
            pairs.append("%dx%d:%d:%d" % (w, h, r, grid))
        return {"kind": kind, "interp": "bicubic", "host": False, "pairs": " ".join(pairs)}
    w, h, r, grid = _draw_geometry(rng, _MOST if kind in ("frame", "classes") else _MOST // 2)
    interp = "bspline" if kind in ("frame", "classes") and rng.random() < 0.25 else "bicubic"
    host = kind == "frame" and rng.random() < 0.3
    return {"kind": kind, "w": w, "h": h, "r": r, "grid": grid, "interp": interp, "host": host}


def _geometries(case):
    if case["kind"] != "batch":
        return [(case["w"], case["h"], case["r"], case["grid"])]
    out = []
    for text in case["pairs"].split():
        size, r, grid = text.split(":")
        w, h = size.split("x")
        out.append((int(w), int(h), int(r), int(grid)))
    return out


# ------------------------------------------------------------------ images --
def _speckles(w, h, gen):
    """Gaussian speckles I = A exp(-d^2 / R^2) on a background of 20, summed
    in fixed point (the same image whatever the order of the additions)."""
    dev = "cuda"
    n = int(6000 * h * w / (512 * 512))

    def uniform(lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=gen, device=dev)

    cy, cx, rad, amp = uniform(-4, h + 4), uniform(-4, w + 4), uniform(2.0, 4.0), uniform(40.0, 200.0)
    off = torch.arange(-12, 13, device=dev)
    acc = torch.zeros(h * w, dtype=torch.int64, device=dev)
    for s in range(0, n, 32768):
        e = min(n, s + 32768)
        iy = cy[s:e].floor().long()[:, None, None] + off[None, :, None]
        ix = cx[s:e].floor().long()[:, None, None] + off[None, None, :]
        d2 = (iy - cy[s:e, None, None]) ** 2 + (ix - cx[s:e, None, None]) ** 2
        val = (amp[s:e, None, None] * torch.exp(-d2 / rad[s:e, None, None] ** 2) * 4096).round().long()
        ok = (iy >= 0) & (iy < h) & (ix >= 0) & (ix < w)
        acc.index_add_(0, (iy.clamp(0, h - 1) * w + ix.clamp(0, w - 1)).reshape(-1), (val * ok).reshape(-1))
    return (acc.float() / 4096 + 20.0).reshape(h, w)


def _catmull_rom(t):
    return (t * (t * (1 - 0.5 * t) - 0.5), t * t * (1.5 * t - 2.5) + 1, t * (t * (2 - 1.5 * t) + 0.5),
            t * t * (0.5 * t - 0.5))


def _deformed(img, r, gen):
    """img sampled at the inverse of X -> X + u(X): translation of a few
    pixels, affine part and sinusoid with gradients up to 1 %."""
    h, w = img.shape
    most = min(6.0, 0.3 * r)  # what an FFT-CC window of 2r pixels follows
    k = (2 * torch.rand(10, generator=gen, device="cuda") - 1).tolist()
    u0, v0, rot = 0.5 * most * k[0], 0.5 * most * k[1], 0.004 * k[2]
    ux, uy, vx, vy = 0.006 * k[3], 0.002 * k[4] - rot, 0.002 * k[5] + rot, 0.006 * k[6]
    lu, lv = 400.0 + 200.0 * k[7], 500.0 + 200.0 * k[8]
    su, sv = 0.003 * lu / (2 * math.pi), 0.003 * lv / (2 * math.pi)
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                          torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    X, Y = x, y
    for _ in range(10):
        dx, dy = X - w / 2, Y - h / 2
        u = u0 + ux * dx + uy * dy + su * torch.sin(dx * (2 * math.pi / lu))
        v = v0 + vx * dx + vy * dy + sv * torch.cos(dy * (2 * math.pi / lv))
        # (a strained or turned large image would move its far ends by more)
        X, Y = x - most * torch.tanh(u / most), y - most * torch.tanh(v / most)
    ix, iy = X.floor(), Y.floor()
    wx, wy = _catmull_rom(X - ix), _catmull_rom(Y - iy)
    ix, iy = ix.long(), iy.long()
    flat, out = img.reshape(-1), torch.zeros_like(img)
    for a in range(4):
        row = torch.zeros_like(img)
        base = (iy + (a - 1)).clamp(0, h - 1) * w
        for b in range(4):
            row += wx[b] * flat[base + (ix + (b - 1)).clamp(0, w - 1)]
        out += wy[a] * row
    return out


def _pair(w, h, r, gen):
    """(reference, target) as uint8 tensors on the GPU."""
    img = _speckles(w, h, gen)
    tar = _deformed(img, r, gen) + 2.0 * torch.randn(h, w, generator=gen, device="cuda")
    return img.round().clamp(0, 255).to(torch.uint8), tar.round().clamp(0, 255).to(torch.uint8)


def _pairs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [_pair(w, h, r, gen) for w, h, r, _ in _geometries(case)]


def _params(w, h, r, grid):
    return make_params(w, h, 1, 1, w - 2, h - 2, r, r, grid, grid, MARGIN, MARGIN, MAX_ITER, DELTA_P)


# --------------------------------------------------------------- the passes --
def prepare(case, seed):
    kind, geoms, pairs = case["kind"], _geometries(case), _pairs(case, seed)
    torch.cuda.synchronize()
    state = {"kind": kind, "keep": pairs}
    interp = INTERP_BSPLINE if case["interp"] == "bspline" else INTERP_BICUBIC
    if kind in ("fftcc", "classes"):
        (w, h, r, grid), (ref, tar) = geoms[0], pairs[0]
        fft = cuFFTCC2D(w, h, w - 2, h - 2, 1, 1, r, r, grid, grid, MARGIN, MARGIN)
        u, v, z = fft.cuInitializeFFTCC(ref)
        n = fft.GetNumPOIs()
        state.update(fft=fft, tar=tar, u=u, v=v, z=z, status=torch.zeros(n, dtype=torch.uint8, device="cuda"))
        if kind == "classes":
            icgn = cuICGN2D(w, h, 1, 1, w - 2, h - 2, r, r, fft.GetNumPOIsX(), fft.GetNumPOIsY(), MAX_ITER, DELTA_P,
                            Iflag=interp)
            icgn.cuInitialize(ref)
            state.update(icgn=icgn, poi=fft.POIPositions("cuda"), p6=torch.zeros(n, 6, device="cuda"),
                         iters=torch.zeros(n, dtype=torch.int32, device="cuda"),
                         flags=torch.zeros(n, dtype=torch.uint8, device="cuda"))
        return state
    frames = []
    for (w, h, r, grid), (ref, _) in zip(geoms, pairs):
        f = DICFrame(_params(w, h, r, grid))
        f.set_interpolation(interp)
        f.set_reference(ref)
        frames.append(f)
    if case["host"]:
        outs = {k: torch.from_numpy(a).pin_memory() for k, a in frames[0].alloc_outputs().items()}
        state.update(frame=frames[0], ref=pairs[0][0], tar=pairs[0][1].cpu().pin_memory(), outs=outs)
    elif kind == "batch":
        state.update(batch=DICBatch(), frames=frames, tars=[t for _, t in pairs],
                     outs=[f.alloc_outputs("cuda") for f in frames])
    else:
        state.update(frame=frames[0], ref=pairs[0][0], tar=pairs[0][1], outs=frames[0].alloc_outputs("cuda"))
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].process(state["frames"], state["tars"], state["outs"])
        return state["outs"]
    if kind in ("fftcc", "classes"):
        out = {k: state[k] for k in ("u", "v", "z", "status")}
        state["fft"].cuComputeFFTCC(out["u"], out["v"], out["z"], state["tar"], out["status"])
        if kind == "classes":
            out.update({k: state[k] for k in ("p6", "iters", "flags")})
            state["icgn"].cuCompute(state["tar"], state["poi"], out["u"], out["v"], out["p6"], out["iters"],
                                    out["flags"])
        return out
    if kind == "refresh":
        state["frame"].set_reference(state["ref"])
    state["frame"].process(state["tar"], **state["outs"])
    return state["outs"]


def work(case):
    """Bytes: the images and outputs, each once.  Operations: two real 2D FFTs
    of the window per POI (target forward, correlation inverse; three, and
    the subset statistics, where the reference is new), and four IC-GN passes
    (the workloads' mean is 3.9) of 52 operations per subset sample: 16-tap
    interpolation, coordinates and the eight sums."""
    total = {"bytes": 0, "flops": 0}
    for w, h, r, grid in _geometries(case):
        n, win, sub = _pois(w, h, r, grid)[0], (2 * r) ** 2, (2 * r + 1) ** 2
        fresh = case["kind"] == "refresh"
        total["bytes"] += w * h * (2 if fresh else 1) + n * 12
        total["flops"] += n * (3 if fresh else 2) * 2.5 * win * math.log2(win)
        if case["kind"] != "fftcc":
            total["bytes"] += n * 29
            total["flops"] += n * (4 * 52 + (60 if fresh else 0)) * sub
    return total


# ------------------------------------------------- the same in 64 bits -------
def _exact_fftcc(ref, tar, py, px, r):
    """First maximum of the circular correlation of the 2r x 2r windows and
    its ZNCC (the correlations are whole numbers: rounded, so ties are ties)."""
    n, N = len(py), 2 * r
    o = torch.arange(N, device="cuda") - r
    out = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 25) // (N * N))
    for s in range(0, n, step):
        y, x = py[s:s + step, None, None] + o[:, None], px[s:s + step, None, None] + o
        f, g = ref[y, x].double(), tar[y, x].double()
        c = torch.fft.irfft2(torch.fft.rfft2(f).conj() * torch.fft.rfft2(g), s=(N, N)).round().flatten(1)
        best = c.max(1).values
        at = torch.where(c == best[:, None], torch.arange(N * N, device="cuda"), N * N).min(1).values
        du, dv = at % N, at // N
        f, g, area = f.flatten(1), g.flatten(1), N * N
        num = best - f.sum(1) * g.sum(1) / area
        den = ((f * f).sum(1) - f.sum(1) ** 2 / area) * ((g * g).sum(1) - g.sum(1) ** 2 / area)
        out[s:s + step, 0] = torch.where(du > r, du - N, du)
        out[s:s + step, 1] = torch.where(dv > r, dv - N, dv)
        out[s:s + step, 2] = num / den.sqrt()
    return out[:, 0], out[:, 1], out[:, 2]


def _bspline(t):
    """The B-spline option's four weights (rows of basis times prefilter)."""
    a, b, c = 3 / 56, 3 / 56, 1 / 7
    return (t * (-11 * a + t * (19 * b + t * (-3 * c))), 1 + t * (-a + t * (-39 * b + t * (8 * c))),
            t * (15 * a + t * (25 * b + t * (-8 * c))), t * (-3 * a + t * (-5 * b + t * (3 * c))))


def _exact_icgn(ref, tar, py, px, u, v, r, bspline):
    """First-order IC-GN: whole-pixel first pass, then interpolated passes
    until the scaled step is below DELTA_P.  Returns p6 [n, 6]."""
    h, w = tar.shape
    SW = 2 * r + 1
    d = torch.arange(-r, r + 1, device="cuda")
    dy, dx = (t.reshape(-1) for t in torch.meshgrid(d, d, indexing="ij"))
    fdx, fdy = dx.double(), dy.double()
    weights = _bspline if bspline else _catmull_rom
    rf, tf = ref.double(), tar.double()
    padded = torch.nn.functional.pad(tf, (2, 2, 2, 2)).reshape(-1)
    P6 = torch.zeros(len(py), 6, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 24) // (SW * SW))
    for s in range(0, len(py), step):
        Y, X = py[s:s + step], px[s:s + step]
        y, x = Y[:, None] + dy, X[:, None] + dx
        R = rf[y, x]
        gx, gy = 0.5 * (rf[y, x + 1] - rf[y, x - 1]), 0.5 * (rf[y + 1, x] - rf[y - 1, x])
        SD = torch.stack((gx, gx * fdx, gx * fdy, gy, gy * fdx, gy * fdy), 1)
        Hinv = torch.linalg.inv(SD @ SD.transpose(1, 2))
        R = R - R.mean(1, keepdim=True)
        Rs = R.norm(dim=1, keepdim=True)
        P = torch.zeros(len(Y), 6, dtype=torch.float64, device="cuda")
        P[:, 0], P[:, 3] = u[s:s + step], v[s:s + step]
        live = torch.arange(len(Y), device="cuda")
        for it in range(MAX_ITER):
            p = P[live]
            wx = X[live, None] + fdx * (1 + p[:, 1:2]) + fdy * p[:, 2:3] + p[:, 0:1]
            wy = Y[live, None] + fdx * p[:, 4:5] + fdy * (1 + p[:, 5:6]) + p[:, 3:4]
            ix, iy = wx.trunc().long(), wy.trunc().long()
            # a subset that leaves the ROI ends its POI where it is
            inside = ((ix >= 1) & (ix < w - 1) & (iy >= 1) & (iy < h - 1)).all(1)
            live, wx, wy, ix, iy, p = live[inside], wx[inside], wy[inside], ix[inside], iy[inside], p[inside]
            if not len(live):
                break
            if it == 0:
                T = tf[iy, ix]
            else:
                cx, cy = weights(wx - ix), weights(wy - iy)
                base = (iy + 1) * (w + 4) + ix + 1
                T = torch.zeros_like(wx)
                for a in range(4):
                    row = torch.zeros_like(wx)
                    for b in range(4):
                        row += cx[b] * padded[base + (a * (w + 4) + b)]
                    T += cy[a] * row
                if not bspline:  # the bicubic table has no last row and column
                    T[(ix == w - 2) | (iy == h - 2)] = 0.0
            T = T - T.mean(1, keepdim=True)
            e = Rs[live] / T.norm(dim=1, keepdim=True) * T - R[live]
            q = (Hinv[live] @ (SD[live] @ e[:, :, None]))[:, :, 0]
            one, zero = torch.ones_like(p[:, 0]), torch.zeros_like(p[:, 0])

            def matrix(m):
                return torch.stack((1 + m[:, 1], m[:, 2], m[:, 0], m[:, 4], 1 + m[:, 5], m[:, 3], zero, zero, one),
                                   1).reshape(-1, 3, 3)

            W = matrix(p) @ torch.linalg.inv(matrix(q))
            P[live] = torch.stack((W[:, 0, 2], W[:, 0, 0] - 1, W[:, 0, 1], W[:, 1, 2], W[:, 1, 0], W[:, 1, 1] - 1), 1)
            scale = torch.tensor([1, r, r, 1, r, r], dtype=torch.float64, device="cuda")
            live = live[(q * scale).norm(dim=1) >= DELTA_P]
            if not len(live):
                break
        P6[s:s + step] = P
    return P6


def exact(case, seed):
    results = []
    for (w, h, r, grid), (ref, tar) in zip(_geometries(case), _pairs(case, seed)):
        _, nx, ny = _pois(w, h, r, grid)
        i, j = torch.meshgrid(torch.arange(ny, device="cuda"), torch.arange(nx, device="cuda"), indexing="ij")
        py, px = (1 + MARGIN + r + grid * i).reshape(-1), (1 + MARGIN + r + grid * j).reshape(-1)
        u, v, z = _exact_fftcc(ref, tar, py, px, r)
        if case["kind"] == "fftcc":
            return {"u": u, "v": v, "z": z, "status": None}
        P = _exact_icgn(ref, tar, py, px, u, v, r, case["interp"] == "bspline")
        results.append({"u": P[:, 0].clone(), "v": P[:, 3].clone(), "zncc": z, "p6": P, "iters": None, "flags": None})
    if case["kind"] == "batch":
        return results
    if case["kind"] == "classes":
        return {"u": results[0]["u"], "v": results[0]["v"], "z": results[0]["zncc"], "status": None,
                "p6": results[0]["p6"], "iters": None, "flags": None}
    return results[0]
