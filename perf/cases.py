"""The work that users have this framework do, as measurable cases.

Six kinds, each through a public entry point, on seeded synthetic scenes (a smooth gradient
with blobs and polygons; sites half spread evenly, half drawn to the image's edges, with the
spread of softness, radius and anisotropy that fitted sites have):

  autograd    SADRenderFunction forward and backward: gradients of a rendered image with
              respect to its sites, as a program with its own loss asks for them.
  step        one optimisation step written with the torch.ops.sad operators, as the
              reference's PyTorch training loop runs it: render, gradients, four tau
              diffusion passes, Adam, and the refresh of the candidate field.
  candidates  CandidateUpdater from its random start down the jump schedule, and the render.
  render      an image from a list of sites: the serving path, on device buffers
              (sad_render_from_sites) or from host arrays through the Executor.
  fit         a whole fit from a host image (Trainer.fit_host) and its rendered result.
  batch       several images of mixed sizes fitted in one lockstep Batch.

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a
program has in hand before the call, run() is one pass, work() what a pass cannot do without
and exact() the outputs in 64 bits where they are a plain function of the inputs.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

DEV = "cuda"


def listed():
    return [
        # the smallest call: latency and launches (64x48 with 300 sites, the smoke test's size)
        {"name": "autograd_64x48", "kind": "autograd", "w": 64, "h": 48, "n": 300},
        # the size that the autograd render is quoted at: 512x512, 16,384 sites
        {"name": "autograd_512", "kind": "autograd", "w": 512, "h": 512, "n": 16384},
        # a photograph-sized image, odd sides
        {"name": "autograd_1999x1503", "kind": "autograd", "w": 1999, "h": 1503, "n": 46941},
        # a step of a PyTorch training loop on a Kodak-sized image, many sites (early in a fit)
        {"name": "step_768x512", "kind": "step", "w": 768, "h": 512, "n": 24576,
         "ssim": 0.0, "removal": False, "masked": False},
        # the same late in a fit, ragged, with the SSIM term, a mask and a prune step's removal deltas
        {"name": "step_1237x941_ssim", "kind": "step", "w": 1237, "h": 941, "n": 18187,
         "ssim": 0.2, "removal": True, "masked": True},
        # candidate search from scratch for a PyTorch program
        {"name": "candidates_512", "kind": "candidates", "w": 512, "h": 512, "n": 16384,
         "passes": 12, "inject": 4, "probes": 0},
        # serving: a thumbnail from host sites through the executor, 1 bpp
        {"name": "render_256_host", "kind": "render", "w": 256, "h": 256, "n": 512, "host": True},
        # serving on device buffers: an ordinary image and the largest, 1 bpp
        {"name": "render_1024", "kind": "render", "w": 1024, "h": 1024, "n": 8192, "host": False},
        {"name": "render_4096", "kind": "render", "w": 4096, "h": 4096, "n": 131072, "host": False},
        # the command line's fixed-site fit: 256x256, 4,096 sites, 200 iterations
        {"name": "fit_256_fixed", "kind": "fit", "w": 256, "h": 256, "n": 4096, "iters": 200, "bpp": 0.0},
        # the headline fit at 1 bpp over the serving mix's 500 iterations (128,000 sites pruned)
        {"name": "fit_1024_1bpp", "kind": "fit", "w": 1024, "h": 1024, "n": 128000, "iters": 500, "bpp": 1.0},
        # a folder of images of mixed sizes and aspect ratios
        {"name": "batch_6_mixed", "kind": "batch", "sizes": "301x199,256x256,512x340,187x410,640x427,1024x683",
         "iters": 200},
    ]


def _sides(rng, lo, hi):
    side = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = math.exp(rng.uniform(math.log(0.5), math.log(2.0)))
    clip = lambda v: max(32, min(int(hi * 1.25), int(round(v))))  # noqa: E731
    return clip(side * math.sqrt(aspect)), clip(side / math.sqrt(aspect))


def _sites_for(rng, w, h, sparse=128.0, dense=8.0):
    """A site count between one site per `sparse` and one per `dense` pixels."""
    return max(64, int(w * h / math.exp(rng.uniform(math.log(dense), math.log(sparse)))))


def draw(rng):
    kind = rng.choice(["autograd", "autograd", "step", "step", "candidates", "render", "render", "fit", "batch"])
    if kind == "autograd":
        w, h = _sides(rng, 48, 1800)
        return {"kind": kind, "w": w, "h": h, "n": _sites_for(rng, w, h)}
    if kind == "step":
        w, h = _sides(rng, 128, 1200)
        return {"kind": kind, "w": w, "h": h, "n": _sites_for(rng, w, h),
                "ssim": rng.choice([0.0, 0.0, 0.2]), "removal": rng.random() < 0.4, "masked": rng.random() < 0.4}
    if kind == "candidates":
        w, h = _sides(rng, 64, 1000)
        return {"kind": kind, "w": w, "h": h, "n": _sites_for(rng, w, h), "passes": rng.randint(6, 14),
                "inject": rng.choice([0, 4, 4]), "probes": rng.choice([0, 0, 1])}
    if kind == "render":
        w, h = _sides(rng, 128, 2600)
        return {"kind": kind, "w": w, "h": h, "n": _sites_for(rng, w, h, 128.0, 32.0),
                "host": max(w, h) <= 1024 and rng.random() < 0.4}
    if kind == "fit":
        if rng.random() < 0.4:
            w, h = _sides(rng, 128, 512)
            return {"kind": kind, "w": w, "h": h, "n": _sites_for(rng, w, h, 64.0, 8.0), "iters": 200, "bpp": 0.0}
        w, h = _sides(rng, 256, 800)
        return {"kind": kind, "w": w, "h": h, "n": 128000, "iters": rng.randint(200, 500), "bpp": 1.0}
    sizes = [_sides(rng, 128, 600) for _ in range(rng.randint(2, 6))]
    return {"kind": kind, "sizes": ",".join("%dx%d" % s for s in sizes), "iters": rng.randint(100, 200)}


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 2654435761 % (1 << 62) + 17)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV)


def _image(w, h, seed):
    """Gradient, Gaussian blobs and hard-edged convex polygons, [h,w,3] f32 in [0,1]."""
    rng = np.random.default_rng(seed)
    side = math.sqrt(w * h)
    yy, xx = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32),
                            torch.arange(w, device=DEV, dtype=torch.float32), indexing="ij")
    col = lambda: torch.tensor(rng.uniform(0, 1, 3), device=DEV, dtype=torch.float32)  # noqa: E731
    c0, c1, th = col(), col(), rng.uniform(0, 2 * math.pi)
    t = xx * math.cos(th) + yy * math.sin(th)
    t = (t - t.min()) / (t.max() - t.min()).clamp_min(1e-6)
    img = c0 + (c1 - c0) * t[..., None]
    blobs = max(4, min(192, round(32 * (side / 256) ** 1.5)))
    for _ in range(blobs):
        sig, cx, cy, c = rng.uniform(4, 40), rng.uniform(0, w), rng.uniform(0, h), col()
        x0, x1 = max(0, int(cx - 3 * sig)), min(w, int(cx + 3 * sig) + 1)
        y0, y1 = max(0, int(cy - 3 * sig)), min(h, int(cy + 3 * sig) + 1)
        gx, gy = xx[y0:y1, x0:x1], yy[y0:y1, x0:x1]
        a = torch.exp(-((gx - cx) ** 2 + (gy - cy) ** 2) / (2 * sig * sig))[..., None]
        img[y0:y1, x0:x1] += (c - img[y0:y1, x0:x1]) * a
    for _ in range(max(2, blobs // 4)):
        cx, cy, r, c = rng.uniform(0, w), rng.uniform(0, h), rng.uniform(0.02, 0.1) * side, col()
        ang = np.sort(rng.uniform(0, 2 * math.pi, int(rng.integers(3, 8))))
        px, py = cx + r * np.cos(ang), cy + r * np.sin(ang)
        x0, x1 = max(0, int(px.min())), min(w, int(px.max()) + 2)
        y0, y1 = max(0, int(py.min())), min(h, int(py.max()) + 2)
        if x0 >= x1 or y0 >= y1:
            continue
        gx, gy = xx[y0:y1, x0:x1], yy[y0:y1, x0:x1]
        inside = torch.ones_like(gx, dtype=torch.bool)
        for i in range(len(ang)):
            j = (i + 1) % len(ang)
            inside &= float(px[j] - px[i]) * (gy - float(py[i])) - float(py[j] - py[i]) * (gx - float(px[i])) >= 0
        img[y0:y1, x0:x1] = torch.where(inside[..., None], c, img[y0:y1, x0:x1])
    return img.clamp(0, 1).contiguous()


def _sites(img, n, seed):
    """[n,10] sites like a fit's: half spread evenly, half where the image changes."""
    h, w = img.shape[:2]
    g = _gen(seed)
    lum = img.mean(dim=2)
    edge = torch.zeros_like(lum)
    edge[:, 1:] += (lum[:, 1:] - lum[:, :-1]).abs()
    edge[1:, :] += (lum[1:, :] - lum[:-1, :]).abs()
    cdf = ((edge * 1e6).long() + 100).flatten().cumsum(0)  # whole numbers: the same sums in any order
    at = torch.searchsorted(cdf, (_rand(g, n - n // 2).double() * cdf[-1]).long()).clamp_max(w * h - 1)
    x = torch.cat([_rand(g, n // 2) * w, (at % w).float() + 4 * (_rand(g, n - n // 2) - 0.5)])
    y = torch.cat([_rand(g, n // 2) * h, torch.div(at, w, rounding_mode="floor").float() + 4 * (_rand(g, n - n // 2) - 0.5)])
    x, y = x.clamp(0, w - 1), y.clamp(0, h - 1)
    order = torch.randperm(n, generator=g, device=DEV)
    x, y = x[order], y[order]
    s = torch.empty(n, 10, device=DEV)
    s[:, 0], s[:, 1] = x, y
    s[:, 2] = 5 + 0.6 * torch.randn(n, generator=g, device=DEV)
    s[:, 3] = (4 + 1.5 * torch.randn(n, generator=g, device=DEV)).clamp(1, 512)
    s[:, 4:7] = (img[y.long(), x.long()] + 0.05 * torch.randn(n, 3, generator=g, device=DEV)).clamp(0, 1)
    th = math.pi * _rand(g, n)
    s[:, 7], s[:, 8] = torch.cos(th), torch.sin(th)
    s[:, 9] = (0.6 * torch.randn(n, generator=g, device=DEV)).clamp(-4, 4)
    return s


def _inv(w, h):
    return float(np.float32(1.0) / np.float32(max(w, h) * max(w, h)))


def _metric(s, ux, uy, inv):
    """tau and the soft distance of sites s ([...,10]) at pixels (ux, uy)."""
    dx, dy = ux - s[..., 0], uy - s[..., 1]
    proj = s[..., 7] * dx + s[..., 8] * dy
    l1 = s[..., 9].exp()
    d2 = (l1 * proj ** 2 + (dx ** 2 + dy ** 2 - proj ** 2).clamp_min(0) / l1) * inv
    return s[..., 2].exp(), d2.clamp_min(1e-8).sqrt() - s[..., 3] * math.sqrt(inv)


def _nearest_field(sites, w, h):
    """The eight nearest sites of every pixel, nearest first, as two [w*h,4] int32 fields
    (searched among the sites around each 16x16 tile): a converged candidate field."""
    n, t = sites.shape[0], 16
    tx, ty = (w + t - 1) // t, (h + t - 1) // t
    k = min(n, 96)
    out = torch.empty(h, w, 8, dtype=torch.int32, device=DEV)
    px = torch.arange(t, device=DEV)
    inv = _inv(w, h)
    rows = max(1, 6_000_000 // max(1, tx * max(n // 8, t * t * k // 8)))
    for r0 in range(0, ty, rows):
        r1 = min(ty, r0 + rows)
        cy, cx = torch.meshgrid(torch.arange(r0, r1, device=DEV), torch.arange(tx, device=DEV), indexing="ij")
        c = torch.stack([cx.flatten() * t + 7.5, cy.flatten() * t + 7.5], 1).float()
        near = torch.cdist(c, sites[:, :2], compute_mode="donot_use_mm_for_euclid_dist").topk(k, 1, largest=False).indices
        ux = (cx.flatten()[:, None] * t + px[None, :])[:, None, :, None].float()  # [tiles,1,t,1]
        uy = (cy.flatten()[:, None] * t + px[None, :])[:, :, None, None].float()  # [tiles,t,1,1]
        tau, d = _metric(sites[near][:, None, None], ux, uy, inv)
        best = (tau * d).topk(min(8, k), 3, largest=False).indices  # [tiles,t,t,8]
        ids = torch.gather(near[:, None, None].expand(-1, t, t, -1), 3, best).to(torch.int32)
        ids = ids.view(r1 - r0, tx, t, t, 8).permute(0, 2, 1, 3, 4).reshape((r1 - r0) * t, tx * t, 8)
        y1 = min(h, r1 * t)
        out[r0 * t:y1] = ids[: y1 - r0 * t, :w]
    out = out.view(w * h, 8)
    return out[:, :4].contiguous(), out[:, 4:].contiguous()


def _scene(case, seed):
    img = _image(case["w"], case["h"], seed)
    return img, _sites(img, case["n"], seed)


def _mask(case, seed):
    """An object mask: 1 inside an ellipse and 0 outside, or all 1."""
    w, h = case["w"], case["h"]
    m = torch.ones(h, w, device=DEV)
    if case["masked"]:
        rng = np.random.default_rng(seed + 5)
        cx, cy = w * rng.uniform(0.4, 0.6), h * rng.uniform(0.4, 0.6)
        yy, xx = torch.meshgrid(torch.arange(h, device=DEV), torch.arange(w, device=DEV), indexing="ij")
        m = (((xx - cx) / (0.45 * w)) ** 2 + ((yy - cy) / (0.45 * h)) ** 2 < 1).float().contiguous()
    return m


def _moments(n, seed):
    """Adam state of a fit some hundreds of steps in, [n,20]."""
    g = _gen(seed + 3)
    scale = 3e-6 * torch.exp(0.7 * torch.randn(n, 20, generator=g, device=DEV))
    state = 0.5 * scale * torch.randn(n, 20, generator=g, device=DEV)
    second = [2, 4, 6, 10, 11, 12, 15, 17]
    state[:, second] = scale[:, second] ** 2
    state[:, 18:] = 0
    return state


ADAM = {"lr_pos": 0.025, "lr_tau": 0.01, "lr_radius": 0.01, "lr_color": 0.01, "lr_dir": 0.0025, "lr_aniso": 0.025,
        "beta1": 0.9, "beta2": 0.999, "eps": 1e-8, "t": 400}
TAU_LAMBDA = 0.03
TAU_PASSES = 4


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def _step_inputs(case, seed):
    img, sites = _scene(case, seed)
    c0, c1 = _nearest_field(sites, case["w"], case["h"])
    return {"target": img, "sites": sites, "c0": c0, "c1": c1, "mask": _mask(case, seed),
            "adam": _moments(case["n"], seed)}


def _autograd_inputs(case, seed):
    img, sites = _scene(case, seed)
    c0, c1 = _nearest_field(sites, case["w"], case["h"])
    g = _gen(seed + 9)
    grad = 0.1 * torch.randn(case["h"], case["w"], 3, generator=g, device=DEV)  # a loss's dL/dimage
    return {"sites": sites, "c0": c0, "c1": c1, "grad": grad}


def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "autograd":
        from sad_gb300 import ops  # noqa: F401  (registers torch.ops.sad)
        from sad_gb300.modules import SADRenderFunction
        s = _autograd_inputs(case, seed)
        s["sites"].requires_grad_(True)
        s.update(case=case, inv=_inv(case["w"], case["h"]), apply=SADRenderFunction.apply)
        return s
    if kind == "step":
        from sad_gb300 import _lib, ops
        s = _step_inputs(case, seed)
        w, h, n = case["w"], case["h"], case["n"]
        bits = _lib.fn("sad_hilbert_bits_for_size")(w, h)
        pairs = torch.empty((n + 1023) // 1024 * 1024, 2, dtype=torch.int32, device=DEV)
        ops.build_hilbert_pairs(s["sites"], pairs, n, pairs.shape[0], w, h, bits)
        pairs = ops.radix_sort_pairs(pairs, 1 << (2 * bits))
        order, pos = (torch.empty(n, dtype=torch.int32, device=DEV) for _ in range(2))
        ops.write_hilbert_order(pairs, order, pos, n)
        s.update(case=case, inv=_inv(w, h), ops=ops, order=order, pos=pos,
                 packed=torch.empty(n, 8, dtype=torch.float16, device=DEV),
                 out0=torch.empty_like(s["c0"]), out1=torch.empty_like(s["c1"]))
        return s
    if kind == "candidates":
        from sad_gb300 import ops
        from sad_gb300.modules import CandidateUpdater
        img, sites = _scene(case, seed)
        up = CandidateUpdater(case["w"], case["h"], case["n"], seed=1 + seed % 1000)
        pow2 = 1 << max(1, math.ceil(math.log2(max(case["w"], case["h"]))))
        jumps = [max(1, pow2 >> (i + 1)) for i in range(case["passes"])]
        return {"case": case, "sites": sites, "up": up, "jumps": jumps, "inv": _inv(case["w"], case["h"]),
                "render": ops.render_sad}
    if kind == "render":
        from sad_gb300 import _lib
        from sad_gb300.executor import Executor
        _, sites = _scene(case, seed)
        w, h, n = case["w"], case["h"], case["n"]
        if case["host"]:
            return {"case": case, "sites": sites.cpu().numpy(), "executor": Executor(workers=2)}
        cfg = _lib.RenderConfig()
        _lib.fn("sad_render_config_default")(ctypes.byref(cfg))
        size = _lib.fn("sad_render_scratch_bytes")(n, w, h, 1)
        return {"case": case, "sites": sites, "cfg": cfg, "call": _lib.call,
                "scratch": torch.empty(size, dtype=torch.uint8, device=DEV),
                "out": torch.empty(h, w, 3, device=DEV)}
    if kind == "fit":
        from sad_gb300 import Trainer
        w, h, n = case["w"], case["h"], case["n"]
        more = {} if case["bpp"] > 0 else {"prune_percentile": 0.0, "densify_percentile": 0.0}
        tr = Trainer(w, h, n_sites=n, max_sites=n, iterations=case["iters"], target_bpp=case["bpp"], log_freq=0, **more)
        return {"case": case, "trainer": tr, "image": _image(w, h, seed).cpu().numpy(),
                "sites": np.empty((n, 10), np.float32), "out": torch.empty(h, w, 3, device=DEV)}
    from sad_gb300.batch import Batch
    sizes = _sizes(case)
    images = [_image(w, h, seed * 64 + i).cpu().numpy() for i, (w, h) in enumerate(sizes)]
    return {"case": case, "batch": Batch(sizes, iterations=case["iters"], log_freq=0), "images": images}


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def _run_step(s):
    case, ops, inv = s["case"], s["ops"], s["inv"]
    w, h, n = case["w"], case["h"], case["n"]
    c0, c1, mask, target = s["c0"], s["c1"], s["mask"], s["target"]
    sites, adam = s["sites"].clone(), s["adam"].clone()
    rendered = ops.render_sad(c0, c1, sites, inv, w, h)
    grads = torch.zeros(11, n, device=DEV)
    rows = grads.unbind(0)
    ops.compute_gradients_tiled(c0, c1, target, rendered, mask, sites, *rows, inv, n, int(case["removal"]),
                                case["ssim"], w, h)
    raw, src = rows[2], rows[2]
    ping, pong = torch.empty(2, n, device=DEV).unbind(0)
    for _ in range(TAU_PASSES):
        ops.tau_diffuse(c0, c1, sites, raw, src, ping, n, TAU_LAMBDA, 1, w, h)
        src, ping, pong = ping, pong, ping
    a = ADAM
    ops.adam_update(sites, adam, rows[0], rows[1], src, *rows[3:10], a["lr_pos"], a["lr_tau"], a["lr_radius"],
                    a["lr_color"], a["lr_dir"], a["lr_aniso"], a["beta1"], a["beta2"], a["eps"], a["t"], w, h)
    ops.pack_candidate_sites(s["sites"], s["packed"], n)
    ops.update_candidates_compact(c0, c1, s["out0"], s["out1"], s["packed"], s["order"], s["pos"], inv, n,
                                  (1 << 16) | 50, 0, 64.0, 0, 4, 1, 32, 1, w, h, w, h)
    return {"rendered": rendered, "grads": grads[:10], "removal": grads[10], "tau": src, "sites": sites,
            "adam": adam[:, :18], "cand0": s["out0"], "cand1": s["out1"]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "autograd":
        out = state["apply"](state["sites"], state["c0"], state["c1"], state["inv"], case["w"], case["h"])
        (grad,) = torch.autograd.grad(out, state["sites"], state["grad"])
        return {"image": out.detach(), "grad": grad}
    if kind == "step":
        return _run_step(state)
    if kind == "candidates":
        up = state["up"]
        up.reset()
        for jump in state["jumps"]:
            up.update(state["sites"], state["inv"], jump, radius_probes=case["probes"], radius_scale=64.0,
                      inject_count=case["inject"])
        c0, c1 = up.get()
        return {"cand0": c0, "cand1": c1,
                "image": state["render"](c0, c1, state["sites"], state["inv"], case["w"], case["h"])}
    if kind == "render":
        w, h, n = case["w"], case["h"], case["n"]
        if case["host"]:
            return state["executor"].submit_render(state["sites"], w, h).result()
        scratch, out = state["scratch"], state["out"]
        state["call"]("sad_render_from_sites", ctypes.byref(state["cfg"]), state["sites"].data_ptr(), n, w, h,
                      out.data_ptr(), scratch.data_ptr(), scratch.numel(), torch.cuda.current_stream().cuda_stream)
        return out
    if kind == "fit":
        sites, psnr = state["trainer"].fit_host(state["image"], state["sites"])
        return {"sites": sites, "psnr": psnr, "image": state["trainer"].render(state["out"])}
    b = state["batch"]
    for i, img in enumerate(state["images"]):
        b.set_target(i, img)
    b.init()
    b.run()
    b.synchronize()
    n = len(state["images"])
    return {"sites": [b.sites(i) for i in range(n)], "psnr": [b.psnr(i) for i in range(n)]}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
# Floating-point operations of one (pixel, candidate): the soft distance, its place in the
# softmax and the blend, and the ten parameter gradients with their sums.
DIST, BLEND, GRADS = 20, 15, 75
VPT_VISITS, JFA_VISITS = 45, 36  # candidates that one pixel of a pass looks at


def _search(px, n, vpt, jfa):
    """Bytes and operations of a candidate search of `vpt` + `jfa` passes."""
    return (vpt * (64 * px + 32 * n) + jfa * (32 * px + 32 * n),
            px * DIST * (vpt * VPT_VISITS + jfa * JFA_VISITS))


def _fit_work(px, start, final, iters):
    active = 0.5 * (start + final)
    b, f = _search(px, active, (iters + 7) // 8, 0)
    return (b + iters * (48 * px + 420 * active) + 40 * final + 12 * px,
            f + iters * px * 8 * (DIST + BLEND + GRADS))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_fit_work(w * h, 128000, w * h / 128, case["iters"]) for w, h in _sizes(case)]
        return {"bytes": int(sum(b for b, _ in parts)), "flops": int(sum(f for _, f in parts))}
    px, n = case["w"] * case["h"], case["n"]
    if kind == "autograd":
        b, f = px * (44 + 44) + 120 * n, px * 8 * (2 * DIST + 2 * BLEND + GRADS)
    elif kind == "step":
        b, f = _search(px, n, 1, 0)
        ssim = case["ssim"] > 0
        b += px * (44 + 48 + (12 if ssim else 0)) + n * (40 + 44 + 4 * 44 + 240)
        f += px * 8 * (2 * DIST + 2 * BLEND + GRADS)
    elif kind == "candidates":
        b, f = _search(px, n, case["passes"], 0)
        b, f = b + px * (32 + 44) + 40 * n, f + px * 8 * (DIST + BLEND)
    elif kind == "render":
        jfa = max(1, math.ceil(math.log2(max(case["w"], case["h"]))))
        b, f = _search(px, n, 16, jfa)
        b, f = b + px * 44 + 40 * n, f + px * 8 * (DIST + BLEND)
    else:
        b, f = _fit_work(px, n, px / 128 if case["bpp"] > 0 else n, case["iters"])
    return {"bytes": int(b), "flops": int(f)}


# ---------------------------------------------------------------------------
# exact
# ---------------------------------------------------------------------------
def _forward64(s, ids, ux, uy, inv):
    """Softmax weights [p,8], colours [p,8,3] and the blend [p,3] of pixels with lists ids."""
    c = s[ids]
    tau, d = _metric(c, ux[:, None], uy[:, None], inv)
    wt = torch.softmax(-tau * d, 1)
    return wt, c, (wt[..., None] * c[..., 4:7]).sum(1)


def _grads64(s, ids, ux, uy, inv, wt, c, pred, dldp, acc):
    """Adds the ten parameter gradients of each (pixel, candidate) into acc [n,10]."""
    tau, l1 = c[..., 2].exp(), c[..., 9].exp()
    l2 = 1 / l1
    dx, dy = ux[:, None] - c[..., 0], uy[:, None] - c[..., 1]
    gx, gy = c[..., 7], c[..., 8]
    proj = gx * dx + gy * dy
    perp2 = (dx ** 2 + dy ** 2 - proj ** 2).clamp_min(0)
    d2 = ((l1 * proj ** 2 + l2 * perp2) * inv).clamp_min(1e-8)
    isq, scale = d2.rsqrt(), math.sqrt(inv)
    dm = d2.sqrt() - c[..., 3] * scale
    dlogit = wt * (dldp[:, None, :] * (c[..., 4:7] - pred[:, None, :])).sum(2)
    kpos = dlogit * tau * inv * isq
    kang = dlogit * -tau * 0.5 * isq
    kdir = 2 * (l1 - l2) * proj * inv
    col = wt[..., None] * dldp[:, None, :]
    v = torch.stack([kpos * (l2 * dx + (l1 - l2) * gx * proj), kpos * (l2 * dy + (l1 - l2) * gy * proj),
                     -dlogit * dm * tau, dlogit * tau * scale, col[..., 0], col[..., 1], col[..., 2],
                     kang * kdir * dx, kang * kdir * dy, kang * (l1 * proj ** 2 - l2 * perp2) * inv], 2)
    acc.index_add_(0, ids.flatten(), v.view(-1, 10))


def _chunks64(case, c0, c1):
    """Row ranges of the image with their pixel coordinates and candidate lists."""
    w, h = case["w"], case["h"]
    rows = max(1, 400_000 // w)
    lists = torch.cat([c0, c1], 1).long()
    for y0 in range(0, h, rows):
        y1 = min(h, y0 + rows)
        p = torch.arange(y0 * w, y1 * w, device=DEV)
        yield slice(y0 * w, y1 * w), lists[p], (p % w).double(), torch.div(p, w, rounding_mode="floor").double()


def _ssim64(ren, tgt):
    """d(SSIM term)/d(luma) at every pixel, 3x3 windows with clamped taps, [h,w]."""
    k = torch.tensor([0.299, 0.587, 0.114], device=DEV, dtype=torch.float32).double()
    x, y = (ren.double() * k).sum(2), (tgt.double() * k).sum(2)
    invn = float(np.float32(0.111111111))

    def mean(a):
        return 9 * invn * F.avg_pool2d(F.pad(a[None, None], (1, 1, 1, 1), mode="replicate"), 3, stride=1)[0, 0]
    mx, my, xx, yy, xy = mean(x), mean(y), mean(x * x), mean(y * y), mean(x * y)
    c1, c2 = float(np.float32(0.0001)), float(np.float32(0.0009))
    a, b = 2 * mx * my + c1, 2 * (xy - mx * my) + c2
    c = mx * mx + my * my + c1
    d = (xx - mx * mx).clamp_min(0) + (yy - my * my).clamp_min(0) + c2
    den = (c * d).clamp_min(1e-8)
    da, db, dc, dd = 2 * my * invn, 2 * invn * (y - my), 2 * mx * invn, 2 * invn * (x - mx)
    return (da * b + a * db) / den - a * b * (dc * d + c * dd) / (den * den), k


def _exact_autograd(case, seed):
    i = _autograd_inputs(case, seed)
    s, inv = i["sites"].double(), _inv(case["w"], case["h"])
    image = torch.empty(case["h"] * case["w"], 3, dtype=torch.float64, device=DEV)
    grad = torch.zeros(case["n"], 10, dtype=torch.float64, device=DEV)
    dl = i["grad"].double().view(-1, 3)
    for at, ids, ux, uy in _chunks64(case, i["c0"], i["c1"]):
        wt, c, pred = _forward64(s, ids, ux, uy, inv)
        image[at] = pred
        _grads64(s, ids, ux, uy, inv, wt, c, pred, dl[at], grad)
    return {"image": image.view(case["h"], case["w"], 3), "grad": grad}


def _exact_tau(case, s, c0, c1, raw):
    w, h, n = case["w"], case["h"], case["n"]
    px = (s[:, 0].float() + 0.5).long().clamp(0, w - 1)
    py = (s[:, 1].float() + 0.5).long().clamp(0, h - 1)
    ids = torch.cat([c0, c1], 1).long()[py * w + px]
    keep = (ids != torch.arange(n, device=DEV)[:, None]).double()
    lam = float(np.float32(TAU_LAMBDA))
    g = raw
    for _ in range(TAU_PASSES):
        g = (raw + lam * (keep * g[ids]).sum(1)) / (1 + lam * keep.sum(1))
    return g


def _exact_adam(case, s, m, g):
    a = {k: float(np.float32(v)) if k != "t" else v for k, v in ADAM.items()}
    b1, b2, eps = a["beta1"], a["beta2"], a["eps"]
    k1, k2 = 1 / (1 - b1 ** a["t"]), 1 / (1 - b2 ** a["t"])
    s, m, w, h = s.clone(), m.clone(), case["w"], case["h"]
    g = [x / (w * h) for x in g]

    def move(first, second, grads, lr):
        for f, gr in zip(first, grads):
            m[:, f] = b1 * m[:, f] + (1 - b1) * gr
        m[:, second] = b2 * m[:, second] + (1 - b2) * sum(gr ** 2 for gr in grads)
        return [lr * m[:, f] * k1 / ((m[:, second] * k2).sqrt() + eps) for f in first]
    st = move([0, 1], 2, [g[0], g[1]], a["lr_pos"])
    s[:, 0], s[:, 1] = (s[:, 0] - st[0]).clamp(0, w - 1), (s[:, 1] - st[1]).clamp(0, h - 1)
    s[:, 2] -= move([3], 4, [g[2]], a["lr_tau"])[0]
    s[:, 3] = (s[:, 3] - move([5], 6, [g[3]], a["lr_radius"])[0]).clamp(1, 512)
    for c in range(3):
        s[:, 4 + c] = (s[:, 4 + c] - move([7 + c], 10 + c, [g[4 + c]], a["lr_color"])[0]).clamp(0, 1)
    dx, dy = s[:, 7].clone(), s[:, 8].clone()
    along = g[7] * dx + g[8] * dy
    st = move([13, 14], 15, [g[7] - dx * along, g[8] - dy * along], a["lr_dir"])
    dx, dy = dx - st[0], dy - st[1]
    il = (dx * dx + dy * dy).rsqrt()
    s[:, 7], s[:, 8] = dx * il, dy * il
    s[:, 9] = (s[:, 9] - move([16], 17, [g[9]], a["lr_aniso"])[0]).clamp(-4, 4)
    return s, m


def _exact_step(case, seed):
    i = _step_inputs(case, seed)
    w, h, n = case["w"], case["h"], case["n"]
    s, inv = i["sites"].double(), _inv(w, h)
    tgt, mask = i["target"].double().view(-1, 3), i["mask"].flatten() > 0
    image = torch.empty(h * w, 3, dtype=torch.float64, device=DEV)
    for at, ids, ux, uy in _chunks64(case, i["c0"], i["c1"]):
        image[at] = _forward64(s, ids, ux, uy, inv)[2]
    dl = 2 * (image - tgt)
    if case["ssim"] > 0:
        ds, k = _ssim64(image.view(h, w, 3), i["target"])
        dl = dl - float(np.float32(case["ssim"])) * ds.view(-1, 1) * k
    dl = dl * mask.double()[:, None]
    grads = torch.zeros(n, 10, dtype=torch.float64, device=DEV)
    for at, ids, ux, uy in _chunks64(case, i["c0"], i["c1"]):
        wt, c, pred = _forward64(s, ids, ux, uy, inv)
        _grads64(s, ids, ux, uy, inv, wt, c, pred, dl[at], grads)
    g = list(grads.unbind(1))
    g[2] = _exact_tau(case, s, i["c0"], i["c1"], g[2])
    sites, adam = _exact_adam(case, s, i["adam"].double(), g)
    # removal deltas jump to a sentinel at a threshold, and candidate ids are whole numbers
    return {"rendered": image.view(h, w, 3), "grads": grads.t().contiguous(), "removal": None, "tau": g[2],
            "sites": sites, "adam": adam[:, :18], "cand0": None, "cand1": None}


def exact(case, seed):
    if case["kind"] == "autograd":
        return _exact_autograd(case, seed)
    if case["kind"] == "step":
        return _exact_step(case, seed)
    return None  # searches and fits: discrete choices and thousands of dependent steps
