"""Performance cases: the work that a program built on umi_gb300 has it do.

Each case is one call (or one step of a loop) through the package's public
entry points, at sizes of this repository's own benchmark workloads and
tests and at ragged ones beside them:

  filter3x3   one 3x3 filter of a float frame (the smallest call: a thumbnail)
  iimg        integral image of a uint8 frame
  full_me     exhaustive block search with argmin, 16x16 or 8x8 blocks
  coarse_me   4K-style motion estimation by the coarse proposal, its refine,
              audit and fallback
  menet       one gradient of the motion-proposal network (forward + backward)
  window      the window operators (census, dilate, erode, box sum, Gaussian)
  batch       bilateral, per-pixel filter and cost volume over uneven images
              in one fused launch
  gemm        C = A B^T in bf16, f16 or fp32 (split precision)
  fprop       convolution in bf16

`listed()` gives the measured cases, `draw(rng)` further ones of the same
ranges.  Inputs are made on the GPU from the seed alone.
"""
import math
import random

import torch
import torch.nn.functional as F

import umi_gb300 as U
from umi_gb300 import apps

DEV = "cuda"
BATCH_ND, BATCH_C = 64, 32  # disparities and feature channels of the cost volume


def listed():
    return [
        # a thumbnail with odd sides: latency of one small call
        {"name": "filter3x3_small", "op": "filter3x3", "h": 97, "w": 131, "pad": 0.0},
        # 4K luma plane: the largest frame whose sums fit int32
        {"name": "iimg_4k", "op": "iimg", "h": 2160, "w": 3840},
        # 1080p frame pair, 16x16 blocks, +-32: the benchmark's motion search (every block moved by itself)
        {"name": "full_me_1080p", "op": "full_me", "h": 1080, "w": 1920, "block": 16, "search": 32, "content": "shift"},
        # cropped 720p video with 8x8 blocks: a panning camera, rows that are not a multiple of 4 bytes
        {"name": "full_me_b8_ragged", "op": "full_me", "h": 717, "w": 1278, "block": 8, "search": 16, "content": "pan"},
        # 4K motion estimation at video rate: proposal, refine, audit of every 64th block, fallback
        {"name": "coarse_me_4k", "op": "coarse_me", "h": 2160, "w": 3840, "audit": 64},
        # one training gradient of the proposal network on a 4K pair
        {"name": "menet_grad_4k", "op": "menet", "h": 2160, "w": 3840},
        # stereo preprocessing: census transform of a 1080p frame
        {"name": "census_1080p", "op": "window", "kind": "census", "h": 1080, "w": 1920, "radius": 2},
        # denoising: separable Gaussian blur, sigma 2, of a 1080p frame
        {"name": "gaussian_1080p", "op": "window", "kind": "gaussian", "h": 1080, "w": 1920, "radius": 6},
        # a batch of uneven images through the three image operators
        {"name": "batch_uneven", "op": "batch", "n": 6, "lo": 256, "hi": 2048, "sizes": 3},
        # large square product in bf16
        {"name": "gemm_bf16_4096", "op": "gemm", "m": 4096, "n": 4096, "k": 4096, "dtype": "bf16"},
        # ragged fp32 product
        {"name": "gemm_f32_ragged", "op": "gemm", "m": 1000, "n": 1540, "k": 2056, "dtype": "f32"},
        # convolution layer of the benchmark
        {"name": "fprop_n32", "op": "fprop", "n": 32, "c": 64, "h": 128, "w": 128, "k": 128, "r": 3},
    ]


def _log(rng, lo, hi, step=1):
    """A size of [lo, hi], spread over its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return int(min(hi, max(lo, round(v / step) * step)))


def _draw(rng):
    op = rng.choice(["filter3x3", "iimg", "full_me", "coarse_me", "menet", "window", "batch", "gemm", "fprop"])
    if op == "filter3x3":
        return {"op": op, "h": _log(rng, 64, 4096), "w": _log(rng, 64, 4096), "pad": rng.choice([0.0, 0.5])}
    if op == "iimg":
        return {"op": op, "h": _log(rng, 64, 2160), "w": _log(rng, 64, 3840)}
    if op == "full_me":
        block = rng.choice([16, 16, 8])
        search = rng.choice([7, 16, 24, 32, 64] if block == 16 else [7, 16, 32])
        w = _log(rng, 160, 3840)
        return {"op": op, "h": _log(rng, 96, 2160), "w": w if rng.random() < 0.3 else (w + 15) // 16 * 16,
                "block": block, "search": search, "content": rng.choice(["shift", "pan"])}
    if op == "coarse_me":
        return {"op": op, "h": _log(rng, 96, 2160, 16), "w": _log(rng, 160, 3840, 16), "audit": rng.choice([16, 64])}
    if op == "menet":
        return {"op": op, "h": _log(rng, 256, 2160, 16), "w": _log(rng, 256, 3840, 16)}
    if op == "window":
        kind = rng.choice(["census", "dilate", "erode", "box", "gaussian"])
        radius = {"census": [1, 2], "dilate": [1, 2, 3], "erode": [1, 2, 3], "box": [2, 3, 7],
                  "gaussian": [3, 6]}[kind]
        return {"op": op, "kind": kind, "h": _log(rng, 64, 2160), "w": _log(rng, 64, 3840), "radius": rng.choice(radius)}
    if op == "batch":
        return {"op": op, "n": rng.randint(1, 8), "lo": 256, "hi": rng.choice([512, 1024, 2048]),
                "sizes": rng.randint(0, 10 ** 6)}
    if op == "gemm":
        return {"op": op, "m": _log(rng, 64, 4096), "n": _log(rng, 64, 4096), "k": _log(rng, 64, 4096, 8),
                "dtype": rng.choice(["bf16", "f16", "f32"])}
    return {"op": op, "n": _log(rng, 1, 32), "c": rng.choice([64, 128]), "h": _log(rng, 7, 128), "w": _log(rng, 7, 160),
            "k": rng.choice([16, 64, 96, 128, 256]), "r": rng.choice([1, 3, 3, 5])}


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng):
    top = max(_cost(c) for c in listed())
    while True:
        c = _draw(rng)
        if _cost(c) <= top:
            return c


# ---------------------------------------------------------------- inputs

def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1009 * int(seed) + salt)


def _texture(g, h, w):
    """A scene: N(128, 40^2) noise blurred by a Gaussian of sigma 2, as uint8."""
    a = torch.normal(128.0, 40.0, size=(h, w), generator=g, device=DEV)
    t = torch.arange(-6, 7, dtype=torch.float64, device=DEV)
    k = torch.exp(-t * t / 8.0)
    k = (k / k.sum()).float()
    x = F.pad(a[None, None], (6, 6, 0, 0), mode="replicate")
    x = sum(k[i] * x[..., i:i + w] for i in range(13))
    x = F.pad(x, (0, 0, 6, 6), mode="replicate")
    x = sum(k[i] * x[..., i:i + h, :] for i in range(13))
    return x[0, 0].round().clamp(0, 255)


def _noisy(g, x):
    return (x + torch.normal(0.0, 2.0, size=x.shape, generator=g, device=DEV)).round().clamp(0, 255).to(torch.uint8)


def _pair(seed, h, w, block, reach, content):
    """(cur, ref) uint8.  shift: every block of ref moved by its own round(N(0, (reach/4)^2)) vector; pan: a camera
    that moves over a still scene.  Both with N(0, 2^2) sensor noise."""
    g = _gen(seed, 1)
    if content == "pan":
        vy, vx = (int(v) for v in torch.randint(-(reach // 2), reach // 2 + 1, (2,), generator=g, device=DEV))
        big = _texture(g, h + abs(vy), w + abs(vx))
        y0, x0 = max(-vy, 0), max(-vx, 0)
        ref = _noisy(g, big[y0:y0 + h, x0:x0 + w])
        cur = _noisy(g, big[y0 + vy:y0 + vy + h, x0 + vx:x0 + vx + w])
        return cur.contiguous(), ref.contiguous()
    a = _texture(g, h, w)
    nby, nbx = max(h // block, 1), max(w // block, 1)
    sh = torch.normal(0.0, reach / 4.0, size=(nby, nbx, 2), generator=g, device=DEV).round().clamp(-reach, reach).long()
    by = (torch.arange(h, device=DEV) // block).clamp(max=nby - 1)
    bx = (torch.arange(w, device=DEV) // block).clamp(max=nbx - 1)
    yy = (torch.arange(h, device=DEV)[:, None] + sh[by[:, None], bx[None, :], 0]).clamp(0, h - 1)
    xx = (torch.arange(w, device=DEV)[None, :] + sh[by[:, None], bx[None, :], 1]).clamp(0, w - 1)
    return _noisy(g, a[yy, xx]).contiguous(), a.to(torch.uint8).contiguous()


def _batch_sizes(case):
    r = random.Random(case["sizes"])
    return [(r.randint(case["lo"], case["hi"]), r.randint(case["lo"], case["hi"])) for _ in range(case["n"])]


def _gauss_kernel(radius):
    """exp(-i^2 / 8) (sigma 2), normalised, as the float32 weights the blur uses."""
    t = torch.arange(-radius, radius + 1, dtype=torch.float64)
    k = torch.exp(-t * t / 8.0)
    return (k / k.sum()).float()


def prepare(case, seed):
    op, g = case["op"], _gen(seed)
    s = {"case": case}

    def rand(*shape):
        return torch.rand(*shape, generator=g, device=DEV)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEV)

    if op == "filter3x3":
        s["x"] = rand(case["h"], case["w"])
        s["w9"] = randn(9).tolist()
        s["out"] = torch.empty_like(s["x"])
    elif op == "iimg":
        s["x"] = torch.randint(0, 256, (case["h"], case["w"]), generator=g, device=DEV, dtype=torch.uint8)
        s["out"] = torch.empty(s["x"].shape, dtype=torch.int32, device=DEV)
        s["ws"] = torch.empty(max(16, U.iimg_workspace_bytes(case["h"], case["w"])), dtype=torch.uint8, device=DEV)
    elif op == "full_me":
        b = case["block"]
        s["cur"], s["ref"] = _pair(seed, case["h"], case["w"], b, case["search"], case["content"])
        s["out"] = torch.empty(((case["h"] // b) * (case["w"] // b), 3), dtype=torch.int32, device=DEV)
    elif op == "coarse_me":
        s["cur"], s["ref"] = _pair(seed, case["h"], case["w"], 16, 64, "shift")
        s["me"] = U.CoarseMe(case["h"], case["w"], device=DEV)
        # 1.2 x the 99th percentile of a matched block's SAD under this sensor noise
        s["thr"] = 576
        s["mv"] = torch.empty((s["me"].nblk, 3), dtype=torch.int32, device=DEV)
        s["sums"] = torch.zeros(2, dtype=torch.int64, device=DEV)
        s["nf"] = torch.zeros(1, dtype=torch.int32, device=DEV)
    elif op == "menet":
        s["cur"], s["ref"] = _pair(seed, case["h"], case["w"], 16, 64, "shift")
        s["net"] = U.MeNet(case["h"], case["w"], device=DEV, seed=int(seed) % 97)
        s["target"] = (16.0 * randn(s["net"].nblk, 2)).round().clamp(-64, 64).int().contiguous()
        s["pred"] = torch.empty((s["net"].nblk, 2), dtype=torch.float32, device=DEV)
    elif op == "window":
        h, w = case["h"], case["w"]
        if case["kind"] == "gaussian":
            s["x"], s["out"], s["tmp"] = rand(h, w), torch.empty(h, w, device=DEV), torch.empty(h, w, device=DEV)
        elif case["kind"] == "box":
            s["x"] = torch.randint(0, 256, (h, w), generator=g, device=DEV, dtype=torch.uint8)
            s["out"] = torch.empty((h, w), dtype=torch.int32, device=DEV)
            s["J"] = torch.zeros((h + 1, w + 1), dtype=torch.int32, device=DEV)
            s["ii"] = torch.empty((h, w), dtype=torch.int32, device=DEV)
            s["ws"] = torch.empty(max(16, U.iimg_workspace_bytes(h, w)), dtype=torch.uint8, device=DEV)
        else:
            s["x"] = torch.randint(0, 256, (h, w), generator=g, device=DEV, dtype=torch.int32)
            s["out"] = torch.empty((h, w), dtype=torch.int32, device=DEV)
    elif op == "batch":
        bil, wf, cv = [], [], []
        for h, w in _batch_sizes(case):
            x = rand(h, w)
            wts = rand(h, w, 3, 3)
            left = randn(BATCH_C, h, w)
            d = torch.randint(0, BATCH_ND, (h, w), generator=g, device=DEV)
            src = (torch.arange(w, device=DEV)[None, :] - d).clamp(min=0)  # right = left moved by its disparity + noise
            right = torch.gather(left, 2, src[None].expand(BATCH_C, h, w)) + 0.1 * randn(BATCH_C, h, w)
            bil.append((x, None, torch.empty_like(x)))
            wf.append((x, wts, torch.empty_like(x)))
            cv.append((left, right.contiguous(), torch.empty((h, w, BATCH_ND), device=DEV)))
        s["jobs"] = [(U.OP_BILATERAL, bil, U.BatchParams(2, 2.0, 0.1, 0, 0), None),
                     (U.OP_WFILTER_PP, wf, U.BatchParams(), None),
                     (U.OP_COST_VOLUME, cv, U.BatchParams(0, 0.0, 0.0, BATCH_C, BATCH_ND), None)]
    elif op == "gemm":
        dt = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}[case["dtype"]]
        s["A"], s["B"] = randn(case["m"], case["k"]).to(dt), randn(case["n"], case["k"]).to(dt)
        s["out"] = torch.empty((case["m"], case["n"]), device=DEV)
        if case["dtype"] == "f32":
            nb = int(U.lib().umi_gemm_f32_f16x3_workspace_bytes(case["m"], case["n"], case["k"]))
            s["ws"] = torch.empty(max(nb, 256), dtype=torch.uint8, device=DEV)
    else:
        n, c, h, w, k, r = (case[q] for q in ("n", "c", "h", "w", "k", "r"))
        s["x"] = randn(n, h, w, c).bfloat16()
        s["wt"] = (randn(k, r, r, c) / math.sqrt(r * r * c)).bfloat16()
        s["out"] = torch.empty((n, k, h, w), device=DEV)
    return s


# ---------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    op = case["op"]
    if op == "filter3x3":
        return U.filter3x3_f32(s["x"], s["w9"], pad=case["pad"], out=s["out"])
    if op == "iimg":
        return U.iimg_u8_i32(s["x"], out=s["out"], workspace=s["ws"])
    if op == "full_me":
        return U.full_me_u8(s["cur"], s["ref"], case["block"], case["search"], out=s["out"])
    if op == "coarse_me":
        mv, sums, nf = s["me"].estimate(s["cur"], s["ref"], sad_threshold=s["thr"], audit_stride=case["audit"],
                                        out=s["mv"], audit_sums=s["sums"], n_fallback=s["nf"])
        return {"mv": mv, "audit": sums, "fallback": nf}
    if op == "menet":
        pred = s["net"].forward(s["cur"], s["ref"], pred=s["pred"])
        grads = s["net"].backward(s["target"])
        return {"pred": pred, "loss": s["net"].loss, "grads": grads}
    if op == "window":
        kind, x, r = case["kind"], s["x"], case["radius"]
        if kind == "gaussian":
            return apps.gaussian(x, 2.0, radius=r, out=s["out"], tmp=s["tmp"])
        if kind == "box":
            return apps.box_sum(x, r, out=s["out"], J=s["J"], ii=s["ii"], workspace=s["ws"])
        return {"census": apps.census, "dilate": apps.dilate, "erode": apps.erode}[kind](x, r, out=s["out"])
    if op == "batch":
        U.batch_run_fused(s["jobs"])
        return [[im[2] for im in job[1]] for job in s["jobs"]]
    if op == "gemm":
        if case["dtype"] == "f32":
            return U.gemm_f32_f16x3(s["A"], s["B"], out=s["out"], workspace=s["ws"])
        return U.gemm(s["A"], s["B"], out=s["out"])
    return U.conv2d_fprop_bf16(s["x"], s["wt"], out=s["out"])


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    op = case["op"]
    if op == "filter3x3":
        px = case["h"] * case["w"]
        return {"bytes": 8 * px, "flops": 18 * px}
    if op == "iimg":
        px = case["h"] * case["w"]
        return {"bytes": 5 * px, "flops": 2 * px}
    if op in ("full_me", "coarse_me"):
        h, w = case["h"], case["w"]
        b = case.get("block", 16)
        nblk = (h // b) * (w // b)
        # bytes: both frames in, the vectors out.  Operations: the |a - b| and the addition of every candidate that
        # the definition compares (coarse_me: of the proposal's cells and of the refine)
        cand = (2 * case["search"] + 1) ** 2 * b * b if op == "full_me" else 61 * 61 * 16 + 81 * 256
        return {"bytes": 2 * h * w + 12 * nblk, "flops": 2 * nblk * cand}
    if op == "menet":
        cells = (case["h"] // 4) * (case["w"] // 4)
        layer = 2 * 32 * 9 * cells  # per input channel
        fwd = layer * (2 + 32 * 3)
        params = 32 * 9 * (2 + 96) + 128 + 1026
        return {"bytes": 2 * case["h"] * case["w"] + 8 * params + 16 * (cells // 16), "flops": 3 * fwd - layer * 2}
    if op == "window":
        px, k = case["h"] * case["w"], 2 * case["radius"] + 1
        per = {"census": 2 * k * k, "dilate": k * k, "erode": k * k, "box": 5, "gaussian": 4 * k}[case["kind"]]
        return {"bytes": (5 if case["kind"] == "box" else 8) * px, "flops": per * px}
    if op == "batch":
        px = sum(h * w for h, w in _batch_sizes(case))
        return {"bytes": px * (8 + 44 + 4 * (2 * BATCH_C + BATCH_ND)), "flops": px * (25 * 6 + 18 + 2 * BATCH_C * BATCH_ND)}
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        e = 4 if case["dtype"] == "f32" else 2
        return {"bytes": e * k * (m + n) + 4 * m * n, "flops": 2 * m * n * k}
    n, c, h, w, k, r = (case[q] for q in ("n", "c", "h", "w", "k", "r"))
    return {"bytes": 2 * n * h * w * c + 2 * k * r * r * c + 4 * n * k * h * w, "flops": 2 * n * h * w * c * k * r * r}


# ---------------------------------------------------------------- the same in 64 bits

def _exact_me(cur, ref, b, r):
    """(mv_y, mv_x, sad) per block: every displacement in raster order, reference pixels clamped to the frame."""
    h, w = cur.shape
    nby, nbx = h // b, w // b
    H, W = nby * b, nbx * b
    c = cur[:H, :W].to(torch.int16)
    p = F.pad(ref.float()[None, None], (r, r + b, r, r + b), mode="replicate")[0, 0].to(torch.int16)
    best = torch.full((nby, nbx), 1 << 40, dtype=torch.int64, device=DEV)
    arg = torch.zeros((nby, nbx), dtype=torch.int64, device=DEV)
    for dy in range(2 * r + 1):
        for dx in range(2 * r + 1):
            d = (c - p[dy:dy + H, dx:dx + W]).abs()
            sad = d.view(nby, b, nbx, b).sum(dim=(1, 3), dtype=torch.int64)
            less = sad < best
            best = torch.where(less, sad, best)
            arg = torch.where(less, torch.full_like(arg, dy * (2 * r + 1) + dx), arg)
    n = 2 * r + 1
    return torch.stack([arg // n - r, arg % n - r, best], dim=-1).view(-1, 3).int()


def _windows(x, r):
    p = F.pad(x[None, None], (r, r, r, r), mode="replicate")[0, 0]
    h, w = x.shape
    return [p[dy:dy + h, dx:dx + w] for dy in range(2 * r + 1) for dx in range(2 * r + 1)]


def _exact_menet(s):
    case, net = s["case"], s["net"]
    H, W = case["h"] // 4, case["w"] // 4
    p = net.params.double()
    x = torch.stack([f.double().view(H, 4, W, 4).sum(dim=(1, 3)) / 512.0 - 4.0 for f in (s["cur"], s["ref"])])
    o, leaves = 0, []

    def take(n, weights):
        nonlocal o
        v = p[o:o + n]
        o += n
        v = (v.bfloat16().double() if weights else v).clone().requires_grad_(True)
        leaves.append(v)
        return v

    for cin, dil in zip((2, 32, 32, 32), (1, 2, 4, 8)):
        wt, bias = take(32 * cin * 9, True), take(32, False)
        xp = F.pad(x, (dil, dil, dil, dil))
        y = bias[:, None].expand(32, H * W)
        for t in range(9):
            dy, dx = (t // 3) * dil, (t % 3) * dil
            y = y + wt.view(32, cin, 9)[:, :, t] @ xp[:, dy:dy + H, dx:dx + W].reshape(cin, -1)
        x = torch.relu(y).view(32, H, W)
    wh, bh = take(2 * 512, True), take(2, False)
    feat = x.view(32, H // 4, 4, W // 4, 4).permute(1, 3, 0, 2, 4).reshape(-1, 512)
    pred = feat @ wh.view(2, 512).T + bh
    loss = F.smooth_l1_loss(pred, s["target"].double() / 16.0, reduction="sum") / pred.shape[0]
    grads = torch.autograd.grad(loss, leaves)
    return {"pred": pred.detach(), "loss": loss.detach().view(1), "grads": torch.cat([v.reshape(-1) for v in grads])}


def _exact_batch(s):
    out = [[], [], []]
    for (x, _, _), (_, wts, _), (left, right, _) in zip(*(job[1] for job in s["jobs"])):
        h, w = x.shape
        xd = x.double()
        p = F.pad(xd, (2, 2, 2, 2))
        ws, wx = torch.zeros_like(xd), torch.zeros_like(xd)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                v = p[2 + dy:2 + dy + h, 2 + dx:2 + dx + w]
                wt = torch.exp(-(v - xd) ** 2 / (2 * 0.1 ** 2)) * math.exp(-(dy * dy + dx * dx) / (2 * 2.0 ** 2))
                ws += wt
                wx += wt * v
        out[0].append(wx / ws)
        p = F.pad(xd, (1, 1, 1, 1))
        out[1].append(sum(wts[:, :, dy, dx].double() * p[dy:dy + h, dx:dx + w] for dy in range(3) for dx in range(3)))
        cv = torch.zeros((h, w, BATCH_ND), dtype=torch.float64, device=DEV)
        for d in range(min(BATCH_ND, w)):
            for c0 in range(0, BATCH_C, 8):
                cv[:, :w - d, d] += (left[c0:c0 + 8, :, :w - d].double() * right[c0:c0 + 8, :, d:].double()).sum(0)
        out[2].append(cv)
    return out


def exact(case, seed):
    if case["op"] == "coarse_me":
        return None  # a proposal: its vectors are whole numbers and have no closed form
    s = prepare(case, seed)
    op = case["op"]
    if op == "filter3x3":
        h, w = case["h"], case["w"]
        p = F.pad(s["x"].double(), (1, 1, 1, 1), value=case["pad"])
        w9 = torch.tensor(s["w9"], dtype=torch.float32).double().tolist()
        return sum(w9[3 * dy + dx] * p[dy:dy + h, dx:dx + w] for dy in range(3) for dx in range(3))
    if op == "iimg":
        return s["x"].long().cumsum(0).cumsum(1).int()
    if op == "full_me":
        if case["search"] > 32 or case["h"] * case["w"] * (2 * case["search"] + 1) ** 2 > 2e10:
            return None
        return _exact_me(s["cur"], s["ref"], case["block"], case["search"])
    if op == "menet":
        return _exact_menet(s)
    if op == "window":
        x, r, kind = s["x"], case["radius"], case["kind"]
        h, w = x.shape
        if kind == "gaussian":
            k = _gauss_kernel(r).double().tolist()
            p = F.pad(x.double()[None, None], (r, r, 0, 0), mode="replicate")
            y = sum(k[i] * p[..., i:i + w] for i in range(2 * r + 1))
            p = F.pad(y, (0, 0, r, r), mode="replicate")
            return sum(k[i] * p[..., i:i + h, :] for i in range(2 * r + 1))[0, 0]
        if kind == "box":
            j = F.pad(x.long().cumsum(0).cumsum(1), (1, 0, 1, 0))
            y0, y1 = ((torch.arange(h, device=DEV) + d).clamp(0, h) for d in (-r, r + 1))
            x0, x1 = ((torch.arange(w, device=DEV) + d).clamp(0, w) for d in (-r, r + 1))
            return (j[y1][:, x1] - j[y0][:, x1] - j[y1][:, x0] + j[y0][:, x0]).int()
        win = _windows(x.double(), r)
        if kind == "census":
            bits = torch.zeros((h, w), dtype=torch.int64, device=DEV)
            for v in win:
                bits = (bits << 1) | (v < x.double()).long()
            return bits.int()
        y = win[0]
        for v in win[1:]:
            y = torch.maximum(y, v) if kind == "dilate" else torch.minimum(y, v)
        return y.int()
    if op == "batch":
        return _exact_batch(s)
    if op == "gemm":
        return s["A"].double() @ s["B"].double().T
    n, c, h, w, k, r = (case[q] for q in ("n", "c", "h", "w", "k", "r"))
    out = torch.empty((n, k, h, w), dtype=torch.float64, device=DEV)
    p = F.pad(s["x"].double(), (0, 0, r // 2, r // 2, r // 2, r // 2))
    wt = s["wt"].double()
    for i in range(n):
        y = sum(p[i, dy:dy + h, dx:dx + w].reshape(-1, c) @ wt[:, dy, dx].T for dy in range(r) for dx in range(r))
        out[i] = y.T.reshape(k, h, w)
    return out
