"""The work a user of this library has it do, as cases that can be timed.

Each case is one pass through the public entry points of
libmeshlessvis_b200.meshless (the C ABI of libmeshless_vis.so), as a program
that renders particle data calls them:

  slice     vis_fourier_volume_rendering of a registered dataset: one view;
  frame     the interactive loop: register, set the view, render, copy the
            image to the host, unregister;
  spectrum  vis_spectrum_compute on a 3D lattice, then vis_spectrum_render_views;
  views     vis_spectrum_render_views alone (a spectrum computed before);
  batch     vis_batch_execute: many particle sets, each with lattice and views;
  post      vis_images_normalize_to_rgb and vis_images_colormap of rendered images.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
inputs and handles, run() is one pass, exact() the same outputs from plain
torch in FP64, and work() the bytes and flops a pass cannot do without (one
particle x frequency term is a complex multiply-accumulate, 8 flops).
"""
import ctypes
import math

import numpy as np
import torch

SPH, GAUSSIAN, WENDLAND, DECAYING = "sph", "gaussian", "wendland", "gaussian_decaying"
MOST_TENSOR_TERMS = 2.9e13  # a drawn case costs no more than the largest listed one
MOST_PLAIN_TERMS = 4e11


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: a preview of a small uniform cloud (4096 particles, one h, 64 x 64)
        _slice("slice-preview", 4096, GAUSSIAN, "uniform", "cube", 0.02, 0.02, 32, 64, 64, 1.0, 1.0, 1),
        # vis_config_get_default's image (cutoff 128, 512 x 512, step 0.1) of an SPH snapshot in a box of 10
        _slice("slice-default", 100003, SPH, "varying", "plummer", 0.05, 0.4, 128, 512, 512, 0.1, 10.0, 1),
        # the timing driver's call without radii and with partial sums
        _slice("slice-no-radii", 262144, WENDLAND, "none", "cube", 0.0, 0.0, 64, 128, 128, 1.0, 1.0, 4),
        # the viewer's frame: every frame registers the data again and fetches the image
        dict(_slice("frame", 30011, WENDLAND, "varying", "plummer", 0.01, 0.08, 96, 192, 192, 1.0, 1.0, 1), kind="frame"),
        # the small half-spectrum: 4096 particles on 64^3, one view
        _spectrum("spectrum-small", 4096, GAUSSIAN, "uniform", "cube", 0.02, 0.02, 1, 64, 64, 64, 1, 64, 64),
        # SPH-like data: clustered, radii over a factor of 60, 64 views
        _spectrum("sph-views", 262144, WENDLAND, "varying", "plummer", 0.004, 0.24, 1, 128, 128, 128, 64, 128, 128),
        # a lattice and sizes that fit no tile: ragged extents, odd images, three groups
        _spectrum("spectrum-ragged", 20011, SPH, "varying", "plummer", 0.01, 0.1, 3, 100, 90, 70, 8, 101, 77),
        # the precision form's headline: 2^20 Gaussians in 16 h-bins on 256^3
        _spectrum("gauss-256", 1 << 20, DECAYING, "varying", "cube", 0.005, 0.05, 16, 256, 256, 256, 1, 256, 256),
        # one frame of a time series: 384^3 and 360 views
        _spectrum("gauss-384", 1000003, DECAYING, "varying", "plummer", 0.002, 0.02, 8, 384, 384, 384, 360, 384, 384),
        # many particle sets of uneven size and lattice, 16 views each, in one call
        dict(name="batch", kind="batch", sets=16, least=1024, most=1 << 19, views=16),
        # turning around a spectrum that is there: a full rotation at 384 x 384
        dict(name="views-384", kind="views", gx=384, gy=384, gz=384, views=360, nx=384, ny=384),
        # the display of that rotation: file output's grey levels and the viewer's colour map
        dict(name="post-384", kind="post", images=360, nx=384, ny=384, log=True, map=1),
    ]


def _slice(name, n, basis, radii, where, h_min, h_max, cutoff, nx, ny, step, box, partial):
    return dict(name=name, kind="slice", n=n, basis=basis, radii=radii, where=where, h_min=h_min, h_max=h_max,
                cutoff=cutoff, nx=nx, ny=ny, step=step, box=box, partial=partial)


def _spectrum(name, n, basis, radii, where, h_min, h_max, groups, gx, gy, gz, views, nx, ny):
    return dict(name=name, kind="spectrum", n=n, basis=basis, radii=radii, where=where, h_min=h_min, h_max=h_max,
                groups=groups, gx=gx, gy=gy, gz=gz, views=views, nx=nx, ny=ny)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_particles(rng, n, kmax):
    """basis, radii and positions; radii so that |k| h stays where the transform is not yet negligible."""
    radii = rng.choice(["none", "uniform", "varying", "varying"])
    basis = rng.choice([SPH, WENDLAND, DECAYING, SPH, WENDLAND, GAUSSIAN])
    if basis == GAUSSIAN:  # exp(+pi r^2) grows: small supports only
        radii = "uniform" if radii == "none" else radii
    h_max = min(0.24, rng.uniform(0.3, 1.0) * (1.1 if basis == GAUSSIAN else 8.0) / kmax)
    h_min = h_max if radii == "uniform" else h_max / rng.uniform(2.0, 40.0)
    if radii == "none":
        basis = rng.choice([SPH, WENDLAND])
        h_min = h_max = 0.0
    return basis, radii, rng.choice(["cube", "plummer"]), h_min, h_max


def draw(rng):
    kind = rng.choice(["slice", "slice", "slice", "frame", "spectrum", "spectrum", "spectrum", "spectrum", "batch",
                       "views", "post"])
    if kind in ("slice", "frame"):
        cutoff = rng.choice([32, 48, 64, 80, 96, 112, 128])
        n = _log(rng, 1000, 300000 if kind == "slice" else 60000)
        basis, radii, where, h_min, h_max = _draw_particles(rng, n, cutoff * 1.42)
        nx, ny = (rng.randint(2 * cutoff, min(512, 4 * cutoff)) for _ in range(2))
        c = _slice("", n, basis, radii, where, h_min, h_max, cutoff, nx, ny, 1.0, 1.0, rng.choice([1, 1, 2, 4]))
        del c["name"]
        return dict(c, kind=kind)
    if kind == "spectrum":
        ragged = rng.random() < 0.25
        if ragged:
            gx, gy, gz = (2 * rng.randint(20, 70) for _ in range(3))
        else:
            gx = gy = gz = rng.choice([48, 64, 96, 128, 160, 192, 256])
            if rng.random() < 0.3:
                gz = rng.choice([64, 96, 128])
        kmax = 0.5 * math.sqrt(gx * gx + gy * gy + gz * gz)
        n = _log(rng, 2000, 1000000)
        basis, radii, where, h_min, h_max = _draw_particles(rng, n, kmax)
        slow = ragged or radii == "varying" and basis in (SPH, WENDLAND, GAUSSIAN)
        per = gx * gy * (gz // 2 + 1)
        n = max(1000, min(n, int((MOST_PLAIN_TERMS if slow else MOST_TENSOR_TERMS) / per)))
        groups = rng.choice([1, 2, 8]) if n >= 16000 else 1
        nx, ny = (gx, gy) if rng.random() < 0.5 else (rng.randint(48, 300), rng.randint(48, 300))
        c = _spectrum("", n, basis, radii, where, h_min, h_max, groups, gx, gy, gz, rng.choice([1, 4, 16, 64]), nx, ny)
        del c["name"]
        return c
    if kind == "batch":
        return dict(kind="batch", sets=rng.randint(2, 20), least=1000, most=_log(rng, 20000, 400000),
                    views=rng.randint(1, 24))
    if kind == "views":
        g = rng.choice([64, 96, 128, 192, 256, 384])
        nx, ny = (g, g) if rng.random() < 0.5 else (rng.randint(g // 2, g), rng.randint(g // 2, g))
        return dict(kind="views", gx=g, gy=g, gz=g, views=_log(rng, 4, 360), nx=nx, ny=ny)
    return dict(kind="post", images=_log(rng, 1, 360), nx=rng.randint(64, 384), ny=rng.randint(64, 384),
                log=rng.random() < 0.5, map=rng.choice([1, 2, 3]))


# ------------------------------------------------------------------ the inputs
def _positions(rng, n, where, box):
    """Uniform in [0, box)^3, or a Plummer sphere of scale box / 10 in its middle."""
    if where == "cube":
        return (rng.random((n, 3), dtype=np.float32) * np.float32(box)).astype(np.float32)
    out = np.empty((0, 3))
    while len(out) < n:
        m = int(1.3 * (n - len(out))) + 256
        r = 0.1 / np.sqrt(np.clip(rng.random(m), 1e-12, 1 - 1e-12) ** (-2.0 / 3.0) - 1.0)
        d = rng.standard_normal((m, 3))
        p = 0.5 + r[:, None] * d / np.linalg.norm(d, axis=1, keepdims=True)
        out = np.concatenate([out, p[np.all((p >= 0) & (p < 1), axis=1)]])
    return (out[:n] * box).astype(np.float32)


def _radii(rng, p, case, box):
    """None, one radius for all, or: log-uniform (cube), or the smoothing
    lengths of a Plummer sphere, density^(-1/3) with scatter, in the interval."""
    n, lo, hi = len(p), case["h_min"], case["h_max"]
    if case["radii"] == "none":
        return None
    if case["radii"] == "uniform":
        return np.full(n, hi, np.float32)
    if case["where"] == "cube":
        return np.exp(rng.uniform(math.log(lo), math.log(hi), n)).astype(np.float32)
    r = np.linalg.norm(p.astype(np.float64) / box - 0.5, axis=1)
    h = (1 + (r / 0.1) ** 2) ** (5.0 / 6.0) * np.exp(0.1 * rng.standard_normal(n))
    return np.clip(h * lo * 1.5, lo, hi).astype(np.float32)


def _weights(rng, n, where):
    return rng.random(n, dtype=np.float32) if where == "cube" else rng.normal(1.0, 0.1, n).astype(np.float32) / n


def _particle_groups(case, seed, box=1.0):
    """The groups of a case: a list of (positions, weights, radii or None)."""
    rng = np.random.default_rng(seed)
    p = _positions(rng, case["n"], case["where"], box)
    h = _radii(rng, p, case, box)
    w = _weights(rng, case["n"], case["where"])
    groups = case.get("groups", 1)
    if groups == 1:
        return [(p, w, h)]
    if case["radii"] == "varying":  # by smoothing length, log-spaced
        edges = np.exp(np.linspace(math.log(case["h_min"]), math.log(case["h_max"]), groups + 1))
        b = np.clip(np.searchsorted(edges, h, side="right") - 1, 0, groups - 1)
    else:
        b = np.arange(case["n"]) % groups
    return [(p[b == k], w[b == k], None if h is None else h[b == k]) for k in range(groups) if np.any(b == k)]


def _batch_sets(case, seed):
    """Sets of log-uniform size, uniform or clustered, one h and lattice each;
    sizes and lattices depend on the case alone, values on the seed."""
    sizes = np.random.default_rng(7 + case["sets"])
    out = []
    for s in range(case["sets"]):
        n = int(np.exp(sizes.uniform(math.log(case["least"]), math.log(case["most"]))))
        g = int(sizes.choice([64, 96, 128, 192]))
        h = float(sizes.uniform(0.01, 0.04))
        rng = np.random.default_rng([seed, s])
        p = _positions(rng, n, "cube" if s % 2 == 0 else "plummer", 1.0)
        w = (rng.standard_normal(n) / math.sqrt(n)).astype(np.float32)
        out.append((p, w, np.full(n, h, np.float32), g))
    return out


def _rotation(count, seed):
    """count views turning about y, from an angle of the seed's."""
    t = 2 * math.pi * (np.arange(count) / count + (seed % 97) / 97.0)
    u = np.stack([np.cos(t), np.zeros(count), -np.sin(t)], axis=1).astype(np.float32)
    return u, np.tile(np.array([0, 1, 0], np.float32), (count, 1))


def _one_view(seed):
    u, v = _rotation(1, seed)
    return tuple(map(float, u[0])), tuple(map(float, v[0]))


def _views_spectrum(case, seed):
    """A half-spectrum like those computed: 4096 clustered Gaussians (FP32)."""
    rng = np.random.default_rng(seed)
    p = _positions(rng, 4096, "plummer", 1.0)
    h = np.full(4096, 0.5 / case["gx"], np.float32)
    return _spectrum64([(p, _weights(rng, 4096, "plummer"), h)], DECAYING, (case["gx"], case["gy"], case["gz"])).to(torch.complex64)


def _post_images(case, seed):
    """Images like those rendered: smooth, positive but for some ringing."""
    g = torch.Generator(device=_device()).manual_seed(seed)
    a = torch.rand((case["images"], 9, 9), generator=g, device=_device())
    a = torch.nn.functional.interpolate(a[:, None], size=(case["nx"], case["ny"]), mode="bicubic")[:, 0]
    noise = torch.randn(a.shape, generator=g, device=a.device)
    return (3.0 * a * a + 0.01 * noise - 0.02).contiguous()


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------- the calls
class _Buffer:
    """A device buffer of the library's as torch sees one (no copy); keeps the
    handle that owns it alive as long as a tensor of it is."""

    def __init__(self, owner, pointer, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=kind, data=(int(pointer), False), version=3)


def _tensor(owner, pointer, shape, kind="<f4"):
    return torch.as_tensor(_Buffer(owner, pointer, shape, kind), device="cuda")


def _spectrum_tensor(sp):
    return _tensor(sp, sp.lib.vis_spectrum_device_data(sp.ptr), sp.shape, "<c8")


def _dataset(groups, basis):
    from libmeshlessvis_b200 import meshless as M

    ids = {SPH: M.SPH, GAUSSIAN: M.GAUSSIAN, WENDLAND: M.WENDLAND_D3_C2, DECAYING: M.GAUSSIAN_DECAYING}
    return M.Dataset([(M.constraints_from_arrays(p, w), h, ids[basis]) for p, w, h in groups])


def prepare(case, seed):
    from libmeshlessvis_b200 import meshless as M

    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind in ("slice", "frame"):
        s["u"], s["v"] = _one_view(seed)
        s["cfg"] = M.Config(step=(case["step"],) * 2, cutoff=(case["cutoff"],) * 2, u=s["u"], v=s["v"],
                            samples=(case["nx"], case["ny"]), partial_sums=case["partial"])
        s["data"] = _dataset(_particle_groups(case, seed, case["box"]), case["basis"])
        if kind == "slice":
            s["cfg"].register(s["data"])
            s["image"] = _tensor(s["cfg"], s["cfg"].c._d_image, (case["nx"], case["ny"]))
    elif kind == "spectrum":
        grid = (case["gx"], case["gy"], case["gz"])
        s["cfg"] = M.Config(cutoff=(min(grid[0], case["nx"]) // 2, min(grid[1], case["ny"]) // 2),
                            samples=(case["nx"], case["ny"]))
        s["data"] = _dataset(_particle_groups(case, seed), case["basis"])
        s["cfg"].register(s["data"])
        s["sp"] = M.Spectrum(grid)
        s["u"], s["v"] = _rotation(case["views"], seed)
        s["images"] = torch.empty((case["views"], case["nx"], case["ny"]), device="cuda")
        s["spectrum"] = _spectrum_tensor(s["sp"])
    elif kind == "views":
        grid = (case["gx"], case["gy"], case["gz"])
        s["cfg"] = M.Config(cutoff=(min(grid[0], case["nx"]) // 2, min(grid[1], case["ny"]) // 2),
                            samples=(case["nx"], case["ny"]))
        s["sp"] = M.Spectrum(grid)
        _spectrum_tensor(s["sp"]).copy_(_views_spectrum(case, seed))
        s["u"], s["v"] = _rotation(case["views"], seed)
        s["images"] = torch.empty((case["views"], case["nx"], case["ny"]), device="cuda")
    elif kind == "batch":
        s["cfg"] = M.Config(cutoff=(32, 32), samples=(64, 64))
        s["batch"] = M.Batch(s["cfg"])
        s["data"] = []
        u, v = _rotation(case["views"], seed)
        for p, w, h, g in _batch_sets(case, seed):
            d = _dataset([(p, w, h)], WENDLAND)
            s["cfg"].register(d)
            s["data"].append(d)
            s["batch"].add(d, (g, g, g), 1.0, (1.0, 1.0), (g // 2, g // 2), (g, g), u, v)
    else:
        s["cfg"] = M.Config()
        s["images"] = _post_images(case, seed)
        s["grey"], s["colour"] = (torch.empty(s["images"].shape + (3,), device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    return s


def run(s):
    from libmeshlessvis_b200 import _lib as L

    kind = s["kind"]
    if kind == "slice":
        s["cfg"].set_axes(s["u"], s["v"])
        s["cfg"].render(s["data"])
        return s["image"]
    if kind == "frame":
        s["cfg"].register(s["data"])
        s["cfg"].set_axes(s["u"], s["v"])
        s["cfg"].render(s["data"])
        image = s["cfg"].image()
        s["cfg"].unregister(s["data"])
        return image
    if kind == "spectrum":
        s["sp"].compute(s["cfg"], s["data"])
        s["sp"].render_views(s["cfg"], s["u"], s["v"], d_images=ctypes.c_void_p(s["images"].data_ptr()), to_host=False)
        return s["spectrum"], s["images"]
    if kind == "views":
        s["sp"].render_views(s["cfg"], s["u"], s["v"], d_images=ctypes.c_void_p(s["images"].data_ptr()), to_host=False)
        return s["images"]
    if kind == "batch":
        b = s["batch"]
        b.execute()
        out = []
        for j, (grid, samples, views) in enumerate(b.jobs):
            lattice = (grid[0], grid[1], grid[2] // 2 + 1)
            out.append((_tensor((b, s["data"]), b.lib.vis_batch_spectrum(b.ptr, j), lattice, "<c8"),
                        _tensor((b, s["data"]), b.lib.vis_batch_images(b.ptr, j), (views,) + samples)))
        return out
    c, cfg, shape = s["case"], s["cfg"], L.int2(s["case"]["nx"], s["case"]["ny"])
    lib, images = cfg.lib, ctypes.c_void_p(s["images"].data_ptr())
    L.check(lib, lib.vis_images_normalize_to_rgb(cfg.ptr, images, c["images"], shape,
                                                 ctypes.c_void_p(s["grey"].data_ptr())))
    L.check(lib, lib.vis_images_colormap(cfg.ptr, images, c["images"], shape, 0.0, 3.0, int(c["log"]), c["map"],
                                         ctypes.c_void_p(s["colour"].data_ptr())))
    return s["grey"], s["colour"]


# ------------------------------------------------------ the same in FP64 torch
def _phi(basis, r):
    """The bases' transforms, with their branch points as the library defines them."""
    if basis == GAUSSIAN:
        return torch.exp(math.pi * r * r)
    if basis == DECAYING:
        return torch.exp(-math.pi * r * r)
    cut = float(np.float32(0.06 if basis == SPH else 0.24))
    m = math.pi * torch.clamp(r, min=cut)
    c, s = torch.cos(2 * m), torch.sin(2 * m)
    if basis == SPH:
        far = 0.75 * math.pi / m**6 * (c - 1) * (c + m * s - 1)
        near = math.pi + r * (-0.007968913156311 + r * -18.293608272337678)
    else:
        far = 7.5 * math.pi / m**8 * (4 * m * m - 6 + (6 - m * m) * c + 4.5 * m * s)
        near = 0.299199300341890 + r * (-0.002379178586124 + r * -0.370530218163545)
    return torch.where(r >= cut, far, near)


def _double(x):
    return torch.as_tensor(np.ascontiguousarray(x), device=_device()).double()


def _turns(freq, q):
    """exp(-2 pi i f q) for every frequency (rows) and particle (columns)."""
    t = freq[:, None] * q[None, :]
    return torch.polar(torch.ones_like(t), -2 * math.pi * (t - torch.round(t)))


def _sum64(ex, ey, ez, kx, ky, kz, w, h, basis):
    """sum_j w_j phi(|k| h_j) ex[a, j] ey[b, j] ez[c, j] -> [a, b, c]."""
    na, nb, nc = len(kx), len(ky), len(kz)
    k2 = kx[:, None, None] ** 2 + ky[None, :, None] ** 2 + kz[None, None, :] ** 2
    one = h is None or bool((h == h[0]).all())
    separable = not one and basis in (GAUSSIAN, DECAYING)
    out = torch.zeros((na * nb, nc), dtype=torch.complex128, device=w.device)
    if separable:
        g = math.pi if basis == GAUSSIAN else -math.pi
        ex, ey, ez = (e * torch.exp(g * k[:, None] ** 2 * h[None, :] ** 2) for e, k in ((ex, kx), (ey, ky), (ez, kz)))
    chunk = max(64, min(2048, int(2.5e8 / (na * nb))))
    if not one and not separable:
        levels, index = torch.unique(k2.reshape(na * nb, nc), return_inverse=True)
        levels = levels.sqrt()
        chunk = max(32, min(chunk, int(2e8 / len(levels))))
    for i in range(0, len(w), chunk):
        j = slice(i, i + chunk)
        a = (ex[:, None, j] * ey[None, :, j] * w[j]).reshape(na * nb, -1)
        if one or separable:
            out += a @ ez[:, j].T
            continue
        a = a.T.contiguous()
        phi = _phi(basis, h[j, None] * levels[None, :])
        for c in range(nc):
            out[:, c] += ez[c, j] @ (phi[:, index[:, c]] * a)
    if one:
        out *= _phi(basis, k2.sqrt() * (1.0 if h is None else float(h[0]))).reshape(na * nb, nc)
    return out.reshape(na, nb, nc)


def _spectrum64(groups, basis, grid):
    ks = [torch.arange(-g // 2, g // 2, device=_device()).double() for g in grid[:2]]
    ks.append(torch.arange(0, grid[2] // 2 + 1, device=_device()).double())
    total = 0
    for p, w, h in groups:
        p = _double(p)
        es = [_turns(k, p[:, i]) for i, k in enumerate(ks)]
        total = total + _sum64(*es, *ks, _double(w), None if h is None else _double(h), basis)
    return total


def _image64(f, cutoff, nx, ny):
    """f[view, x + cx - 1, y], x in (-cx, cx), y in [0, cy): the unnormalised 2D C2R."""
    cx, cy = cutoff
    half = torch.zeros((len(f), nx, ny // 2 + 1), dtype=torch.complex128, device=f.device)
    x = torch.arange(-cx + 1, cx, device=f.device)
    half[:, torch.where(x < 0, x + nx, x), :cy] = f
    return torch.fft.irfft2(half, s=(nx, ny), norm="forward")


def _views64(spec, u, v, cutoff, nx, ny):
    """Trilinear slices through the half-spectrum, then the C2R; step 1."""
    cx, cy = cutoff
    gx, gy, lz = spec.shape
    x = torch.arange(-cx + 1, cx, device=spec.device).double()[:, None, None]
    y = torch.arange(0, cy, device=spec.device).double()[None, :, None]
    out = []
    for uu, vv in zip(_double(u), _double(v)):
        p = x * uu + y * vv
        flip = p[..., 2] < 0
        p = torch.where(flip[..., None], -p, p)
        low = torch.floor(p)
        t = p - low
        low = low.long()
        f = torch.zeros(flip.shape, dtype=torch.complex128, device=spec.device)
        for c in range(8):
            d = [c & 1, c >> 1 & 1, c >> 2]
            wgt = 1.0
            for i in range(3):
                wgt = wgt * (t[..., i] if d[i] else 1 - t[..., i])
            i, j, l = low[..., 0] + d[0] + gx // 2, low[..., 1] + d[1] + gy // 2, low[..., 2] + d[2]
            ok = (i >= 0) & (i < gx) & (j >= 0) & (j < gy) & (l < lz)
            val = spec[i.clamp(0, gx - 1), j.clamp(0, gy - 1), l.clamp(0, lz - 1)].to(torch.complex128)
            f += torch.where(ok, val * wgt, torch.zeros_like(val))
        out.append(_image64(torch.where(flip, f.conj(), f)[None], cutoff, nx, ny)[0])
    return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("slice", "frame"):
        (p, w, h), = _particle_groups(case, seed, case["box"])
        u, v = (_double(np.array(a, np.float32)) for a in _one_view(seed))
        step, c = float(np.float32(case["step"])), case["cutoff"]
        x = torch.arange(-c + 1, c, device=_device()).double()
        y = torch.arange(0, c, device=_device()).double()
        p, w, h = _double(p), _double(w), None if h is None else _double(h)
        unit = torch.ones((1, len(w)), dtype=torch.complex128, device=w.device)
        f = _sum64(_turns(x, step * (p @ u)), _turns(y, step * (p @ v)), unit, step * x, step * y,
                   torch.zeros(1, dtype=torch.float64, device=w.device), w, h, case["basis"])
        return _image64(f[None, :, :, 0] * step * step, (c, c), case["nx"], case["ny"])[0]
    if kind == "spectrum":
        f = _spectrum64(_particle_groups(case, seed), case["basis"], (case["gx"], case["gy"], case["gz"]))
        u, v = _rotation(case["views"], seed)
        cutoff = (min(case["gx"], case["nx"]) // 2, min(case["gy"], case["ny"]) // 2)
        return f, _views64(f, u, v, cutoff, case["nx"], case["ny"])
    if kind == "views":
        u, v = _rotation(case["views"], seed)
        cutoff = (min(case["gx"], case["nx"]) // 2, min(case["gy"], case["ny"]) // 2)
        return _views64(_views_spectrum(case, seed), u, v, cutoff, case["nx"], case["ny"])
    if kind == "batch":
        u, v = _rotation(case["views"], seed)
        out = []
        for p, w, h, g in _batch_sets(case, seed):
            f = _spectrum64([(p, w, h)], WENDLAND, (g, g, g))
            out.append((f, _views64(f, u, v, (g // 2, g // 2), g, g)))
        return out
    a = _post_images(case, seed).double()
    grey = a.clamp(min=0) / a.amax(dim=(1, 2), keepdim=True)
    a = (a / 3.0).clamp(min=0)
    if case["log"]:
        eps, alpha = 1e-3, 0.01
        a = (torch.log(alpha * a + eps) - math.log(eps)) / (math.log(alpha + eps) - math.log(eps))
    knots, colours = {
        1: ((0, 0.475, 0.694, 0.745, 1), ((0, 0, 0), (0.686, 0.004, 0), (1, 0.42, 0), (1, 0.518, 0), (1, 1, 1))),
        2: ((0, 0.25, 0.5, 0.75, 1), ((0, 0, 1), (0, 1, 1), (0, 1, 0), (1, 1, 0), (1, 0, 0))),
        3: ((0, 0.475, 0.694, 0.745, 1), ((0, 0, 0), (0, 0.004, 0.686), (0, 0.42, 1), (0, 0.518, 1), (1, 1, 1))),
    }[case["map"]]
    k, col = (_double(np.array(x, np.float32)) for x in (knots, colours))
    i = torch.bucketize(a, k).clamp(1, 4)
    t = ((a - k[i - 1]) / (k[i] - k[i - 1])).clamp(max=1.0)[..., None]
    return grey[..., None].expand(grey.shape + (3,)), t * col[i] + (1 - t) * col[i - 1]


# ------------------------------------------------------------------ the minimum
def work(case):
    kind = case["kind"]
    if kind in ("slice", "frame"):
        freq = (2 * case["cutoff"] - 1) * case["cutoff"]
        per = 16 if case["radii"] == "none" else 20
        return dict(bytes=per * case["n"] + 4 * case["nx"] * case["ny"], flops=8.0 * case["n"] * freq)
    pixels = case.get("views", 0) * case.get("nx", 0) * case.get("ny", 0)
    if kind == "spectrum":
        freq = case["gx"] * case["gy"] * (case["gz"] // 2 + 1)
        per = 16 if case["radii"] == "none" else 20
        return dict(bytes=per * case["n"] + 8 * freq + 4 * pixels, flops=8.0 * case["n"] * freq)
    if kind == "views":
        touched = min(8 * case["gx"] * case["gy"] * (case["gz"] // 2 + 1), 8 * 8 * pixels // 2)
        return dict(bytes=touched + 4 * pixels,
                    flops=2.5 * pixels * math.log2(case["nx"] * case["ny"]) + 32.0 * pixels // 2)
    if kind == "batch":
        total = dict(bytes=0, flops=0.0)
        for p, _, _, g in _batch_sets(case, 0):
            freq = g * g * (g // 2 + 1)
            total["bytes"] += 20 * len(p) + 8 * freq + 4 * case["views"] * g * g
            total["flops"] += 8.0 * len(p) * freq
        return total
    n = case["images"] * case["nx"] * case["ny"]
    return dict(bytes=(4 + 12 + 12) * n, flops=20.0 * n)
