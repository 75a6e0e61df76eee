"""Degenerate image sizes through the whole fit and the render from sites: one pixel, one
row, one column, odd sizes, more sites than pixels.  The oracle's fit runs the same cases
(tests/test_oracle_cpu.py covers its side); here the device path must stay finite,
reproducible and improving."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 2), (1, 64), (64, 1), (3, 2), (17, 5)]


@pytest.mark.parametrize("w,h", SIZES)
def test_fit_at_degenerate_sizes(cuda, w, h):
    from sad_gb300.config import train_config
    from sad_gb300.trainer import Trainer
    img = np.random.default_rng(w * 100 + h).uniform(0, 1, (h, w, 3)).astype(np.float32)
    cfg = train_config(log_freq=0, n_sites=4, max_sites=8, iterations=40, target_bpp=0.0, prune_start=5,
                       prune_freq=5, prune_end=30, cand_hilbert_window=4)
    out = []
    for _ in range(2):
        with Trainer(w, h, cfg) as tr:
            tr.set_target(img)
            tr.init()
            p0 = tr.psnr()
            tr.run()
            p1 = tr.psnr()
            out.append((p0, p1, tr.sites(active_only=False)))
    (p0, p1, s0), (q0, q1, s1) = out
    assert np.isfinite(p0) and np.isfinite(p1) and np.isfinite(s0).all()
    assert p1 >= p0 - 1e-3
    assert (p0, p1) == (q0, q1)
    np.testing.assert_array_equal(s0, s1)


@pytest.mark.parametrize("w,h,n", [(1, 1, 1), (1, 1, 3), (2, 3, 1), (1, 50, 7), (50, 1, 7), (9, 7, 200)])
def test_render_from_sites_at_degenerate_sizes(cuda, w, h, n):
    from sad_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(n)
    s = np.zeros((n, 10), np.float32)
    s[:, 0] = rng.uniform(0, w, n)
    s[:, 1] = rng.uniform(0, h, n)
    s[:, 2], s[:, 3] = 5.0, 4.0
    s[:, 4:7] = rng.uniform(0.2, 0.8, (n, 3))
    s[:, 7] = 1.0
    cfg = _lib.RenderConfig()
    lib.sad_render_config_default(C.byref(cfg))
    nb = lib.sad_render_scratch_bytes(n, w, h, cfg.cand_downscale)
    scratch = torch.empty(nb, dtype=torch.uint8, device="cuda")
    d = torch.from_numpy(s).cuda()
    out = torch.full((h, w, 3), -1.0, device="cuda")
    assert lib.sad_render_from_sites(C.byref(cfg), C.c_void_p(d.data_ptr()), n, w, h, C.c_void_p(out.data_ptr()),
                                     C.c_void_p(scratch.data_ptr()), nb, None) == 0, lib.sad_last_error()
    torch.cuda.synchronize()
    o = out.cpu().numpy()
    # every pixel is written, and is a convex combination of the site colours
    assert np.isfinite(o).all()
    assert o.min() >= 0.2 - 1e-5 and o.max() <= 0.8 + 1e-5


def _tall(w, h, n):
    """Sites down a tall image, with exact FP32 distances (whole pixels, unit softness, no
    anisotropy; max side 2^18 for the scale)."""
    rng = np.random.default_rng(h)
    s = np.zeros((n, 10), np.float32)
    s[:, 0], s[:, 1] = rng.integers(0, w, n), np.sort(rng.integers(0, h, n))
    s[:, 3], s[:, 7] = rng.integers(1, 9, n), 1.0
    s[:, 4:7] = rng.uniform(0.2, 0.8, (n, 3))
    return s


@pytest.mark.parametrize("w,h,step", [(2, 262140, 1), (2, 262141, 1), (1, 300001, 4), (2, 524280, 2),
                                      (80, 264000, 8)])
def test_flood_of_tall_fields(cuda, orc, w, h, step):
    """Rows of blocks on either side of the grid's y limit (four texel rows a block)."""
    from sad_gb300 import ops
    sites = _tall(w, h, 5000)
    rng = np.random.default_rng(w)
    f = rng.integers(0, 5000, (w * h, 4)).astype(np.uint32)
    f[(np.arange(w * h) // w) % 3 == 1] = 0xFFFFFFFF
    near = np.searchsorted(sites[:, 1], np.arange(h)).clip(0, 4999).repeat(w)
    f[:, 0] = np.where(f[:, 0] == 0xFFFFFFFF, f[:, 0], near)
    inv = 2.0 ** -36
    out = torch.full((w * h, 4), -2, dtype=torch.int32, device="cuda")
    ops.jfa_flood(torch.from_numpy(f.view(np.int32)).cuda(), out, torch.from_numpy(sites).cuda(), inv, 0, step, 1, w, h)
    want = orc.jfa_flood(f, sites, step, w, h, inv_s2=inv)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("w,h", [(1, 524280), (1, 524281), (2, 600000), (1, 1048560)])
def test_gradients_of_tall_images(cuda, orc, w, h):
    """Rows of blocks on either side of the grid's y limit (eight pixel rows a block), every pixel
    with the sites around it, against the FP64 sums (the FP32 oracle's texel of a pixel overflows
    above 46,340 rows).  FP32 terms with exact distances and some 1,000 of them a site: 1e-3 of
    each parameter's norm allows for sums that cancel to a thousandth."""
    from sad_gb300 import ops
    n = 4000
    sites = _tall(w, h, n)
    near = np.searchsorted(sites[:, 1], np.arange(h)).repeat(w)[:, None] + np.arange(-4, 4)
    ids = near.clip(0, n - 1).astype(np.uint32)
    c0, c1 = np.ascontiguousarray(ids[:, :4]), np.ascontiguousarray(ids[:, 4:])
    img = np.random.default_rng(3).uniform(0, 1, (h, w, 3)).astype(np.float32)
    dev = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()  # noqa: E731
    bufs = [torch.zeros(n, device="cuda") for _ in range(11)]
    inv = 1.0 / max(w, h) ** 2
    ops.compute_gradients_tiled(dev(c0), dev(c1), dev(img), dev(img), torch.ones(h, w, device="cuda"), dev(sites), *bufs,
                                inv, 0, 0, 0.0, w, h)
    want = orc.compute_gradients_d(c0, c1, img, sites, w, h)
    for b, g in zip(bufs, want):
        assert np.linalg.norm(b.cpu().numpy() - g) <= 1e-3 * np.linalg.norm(g)


@pytest.mark.parametrize("n", [8, 4000])  # sums by table, and by groups of lanes
def test_gradients_of_too_tall_an_image_are_refused(cuda, n):
    from sad_gb300 import ops
    w, h = 1, 1048561
    c = torch.zeros(w * h, 4, dtype=torch.int32, device="cuda")
    img, bufs = torch.zeros(h, w, 3, device="cuda"), [torch.zeros(n, device="cuda") for _ in range(11)]
    with pytest.raises(RuntimeError, match="invalid configuration|invalid argument"):
        ops.compute_gradients_tiled(c, c, img, img, torch.ones(h, w, device="cuda"),
                                    torch.from_numpy(_tall(w, h, n)).cuda(), *bufs, 1.0 / h ** 2, 0, 0, 0.0, w, h)


def test_render_of_a_tall_image(cuda):
    """A render from sites whose flood has more rows of blocks than the grid's y takes: pixels
    between 0.2 and 0.8, the range of the sites' colours."""
    from sad_gb300 import _lib
    w, h, n = 2, 300000, 3000
    sites = torch.from_numpy(_tall(w, h, n)).cuda()
    cfg = _lib.RenderConfig()
    _lib.fn("sad_render_config_default")(C.byref(cfg))
    nb = _lib.fn("sad_render_scratch_bytes")(n, w, h, cfg.cand_downscale)
    scratch = torch.empty(nb, dtype=torch.uint8, device="cuda")
    out = torch.full((h, w, 3), -1.0, device="cuda")
    _lib.call("sad_render_from_sites", C.byref(cfg), C.c_void_p(sites.data_ptr()), n, w, h,
              C.c_void_p(out.data_ptr()), C.c_void_p(scratch.data_ptr()), nb, None)
    torch.cuda.synchronize()
    o = out.cpu().numpy()
    assert o.min() >= 0.2 - 1e-5 and o.max() <= 0.8 + 1e-5
