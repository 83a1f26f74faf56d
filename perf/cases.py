"""Performance cases of the snapshot imager and the source finder.

A case is one call that a program makes once per snapshot: an imaging call on
device buffers, a batch of imaging calls, an imaging call on host arrays (the
drop-in form), or a source-finder call.  The program keeps one `Context`, as a
long-running one does, and hands it a new snapshot in buffers of its own at
every call.

Real ranges: images of 256^2 to 8192^2 (powers of two and other round sizes,
with and without padding), one thousand to four million visibilities; uv
coverage filling a disk, concentrated towards the centre, or along the tracks
of an array's baselines; GaussianSinc and PSWF kernels, oversampled or exact;
no, truncated and untruncated W-kernels; FP64, FP32 and compensated FP32.
"""
import math

import numpy as np
import torch

from fastimaging_b200 import capi

PRECISION = {"fp64": capi.FP64, "fp32": capi.FP32, "fp32c": capi.FP32C}
CATALOGUE = 512  # more than the sources of any case
KERNEL = {"gsinc": capi.GaussianSinc, "pswf": capi.PSWF}

# Fields of an imaging case and their usual values: n visibilities ("vis":
# c128 or c64) of coverage "uv" reaching "reach" of the grid's half width and
# |w| <= wmax wavelengths, imaged to size^2 pixels of "cell" arcsec.
SNAPSHOT = {
    "do": "image", "n": 0, "vis": "c128", "uv": "disk", "reach": 0.9, "wmax": 0.0, "sources": 20, "size": 0,
    "cell": 1.0, "pad": 1.0, "precision": "fp32c", "kernel": "gsinc", "support": 3, "os": 8, "exact_kernel": False,
    "beam": False, "analytic": False, "planes": 0, "wsupport": 0, "trunc": 0.0,
}
FIND = {"do": "find", "rows": 0, "cols": 0, "dtype": "fp32", "sources": 150, "negative": True, "four": False,
        "fit": False}
BATCH = {"do": "batch", "count": 0, "nmin": 0, "nmax": 0, "sizes": "1024", "precision": "fp32c", "planes": 16,
         "wsupport": 16, "trunc": 1.0}


def _case(base, **kw):
    return dict(base, **kw)


def listed():
    return [
        # the smallest call: a quick look at a short integration, bound by latency and launches
        _case(SNAPSHOT, name="image_256_wproj_fp64", n=5_000, size=256, cell=2.0, sources=4, wmax=300.0, planes=4,
              wsupport=8, trunc=1.0, precision="fp64"),
        # the plain imager without W-projection, in the reference's own precision
        _case(SNAPSHOT, name="image_2048_plain_fp64", n=100_000, size=2048, sources=5, precision="fp64"),
        # the W-projection snapshot of the benchmark, compensated single and plain double precision
        _case(SNAPSHOT, name="image_4096_wproj_fp32c", n=1_000_000, size=4096, wmax=2000.0, planes=32, wsupport=16,
              trunc=1.0),
        _case(SNAPSHOT, name="image_4096_wproj_fp64", n=1_000_000, size=4096, wmax=2000.0, planes=32, wsupport=16,
              trunc=1.0, precision="fp64"),
        # the largest image: many visibilities concentrated at the centre of the uv plane, complex64 input
        _case(SNAPSHOT, name="image_8192_pswf_fp32c", n=4_000_000, vis="c64", uv="gauss", size=8192, kernel="pswf",
              support=4, os=16, analytic=True),
        # wide W-kernels (no truncation): the gridder's taps are the work
        _case(SNAPSHOT, name="image_4096_wide_fp32c", n=1_000_000, size=4096, wmax=2000.0, planes=32, wsupport=16),
        # the reference's default kernel mode (exact PSWF) with the beam and a padded grid, along uv tracks
        _case(SNAPSHOT, name="image_1500_exact_beam_fp64", n=77_777, uv="tracks", size=1500, pad=1.44, kernel="pswf",
              exact_kernel=True, beam=True, precision="fp64"),
        # an image coarser than the array's resolution: visibilities beyond the grid are left out
        _case(SNAPSHOT, name="image_1000_edge_fp32", n=333_333, uv="tracks", reach=1.05, size=1000, cell=2.0,
              wmax=800.0, planes=64, wsupport=12, trunc=2.0, os=4, kernel="pswf", precision="fp32"),
        # the drop-in call on host arrays: transfers both ways are part of it
        _case(SNAPSHOT, name="host_2048_wproj_fp32c", do="host", n=300_000, size=2048, wmax=500.0, planes=16,
              wsupport=16, trunc=1.0),
        # uneven snapshots of one observation imaged in one call
        _case(BATCH, name="batch_16_fp32c", count=16, nmin=50_000, nmax=1_000_000, sizes="1024,2048,4096"),
        # source finding on a large single-precision image and on an oblong double-precision one with fits
        _case(FIND, name="find_4096_fp32", rows=4096, cols=4096),
        _case(FIND, name="find_1502x1998_fp64_fit", rows=1502, cols=1998, dtype="fp64", sources=60, fit=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# even sizes with small factors, as users pick them (a multiple of four)
_ROUND = sorted({4 * 2 ** a * 3 ** b * 5 ** c for a in range(12) for b in range(3) for c in range(4)})


def _size(rng, lo, hi):
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_ROUND, key=lambda s: abs(math.log(s / want)))


def draw(rng):
    what = rng.choice(["image"] * 6 + ["find"] * 2 + ["batch", "host"])
    if what == "find":
        rows = _log(rng, 100, 2048) * 2
        return _case(FIND, rows=rows, cols=2 * min(2048, max(100, int(rows * rng.uniform(0.35, 0.7)))),
                     dtype=rng.choice(["fp32", "fp64"]), sources=rng.randint(5, 150), negative=rng.random() < 0.7,
                     four=rng.random() < 0.3, fit=rng.random() < 0.3)
    if what == "batch":
        lo = _log(rng, 2_000, 100_000)
        return _case(BATCH, count=rng.randint(2, 12), nmin=lo, nmax=min(700_000, lo * rng.randint(2, 20)),
                     sizes=rng.choice(["256,512", "512,1024,2048", "1000,1500,3000", "1024,2048,4096"]),
                     precision=rng.choice(["fp32c", "fp32c", "fp64"]), planes=rng.choice([8, 16, 32]))
    c = dict(SNAPSHOT)
    c["do"] = what
    c["precision"] = rng.choice(["fp64", "fp32c", "fp32c", "fp32"])
    c["n"] = _log(rng, 1_000, 3_000_000 if what == "image" else 500_000)
    c["size"] = _size(rng, 256, 6000 if what == "image" else 3000)
    c["vis"] = "c64" if c["precision"] != "fp64" and rng.random() < 0.4 else "c128"
    c["uv"] = rng.choice(["disk", "gauss", "tracks"])
    c["reach"] = rng.choice([0.5, 0.8, 0.9, 0.9, 1.05])
    c["cell"] = rng.choice([0.5, 1.0, 2.0])
    c["pad"] = rng.choice([1.0, 1.0, 1.0, 1.2, 1.5]) if c["size"] <= 4096 else 1.0
    c["kernel"], c["support"] = rng.choice([("gsinc", 3), ("pswf", 3), ("pswf", 4), ("pswf", 5)])
    c["os"] = rng.choice([4, 8, 8, 16])
    c["beam"] = rng.random() < 0.15
    # the transform of a truncated PSWF wider than S = 3 crosses zero inside the image: those take the analytic
    # correction, as the precision study does
    c["analytic"] = c["kernel"] == "pswf" and (c["support"] > 3 or rng.random() < 0.5)
    how = rng.random()
    if how < 0.15:
        c["exact_kernel"] = True
        c["n"] = min(c["n"], 150_000)
    elif how < 0.65:
        c["planes"] = rng.choice([4, 16, 32, 64, 128])
        c["wsupport"] = rng.choice([8, 12, 16])
        c["os"] = rng.choice([4, 8])
        c["wmax"] = float(rng.randint(50, 2000))
        c["trunc"] = rng.choice([0.5, 1.0, 1.0, 2.0])
        if rng.random() < 0.15:
            c["trunc"] = 0.0
            c["n"] = min(c["n"], 500_000)
    return c


# ------------------------------------------------------------------ inputs

_ctx = None


def _context():
    """The one library context that the program keeps."""
    global _ctx
    if _ctx is None:
        _ctx = capi.Context(0)
    return _ctx


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape, dtype=torch.float64):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


def _coverage(g, n, uv, radius, wmax):
    """(3, n) u, v, w in wavelengths."""
    if uv == "tracks":
        # an array of 48 antennas followed in hour angle: at every time one visibility per baseline
        ants = 48
        pos = _randn(g, ants, 3) * torch.tensor([1.0, 1.0, 0.2], device="cuda", dtype=torch.float64)
        i, j = torch.triu_indices(ants, ants, 1, device="cuda")
        b = pos[j] - pos[i]
        k = torch.arange(n, device="cuda")
        times = (n + b.shape[0] - 1) // b.shape[0]
        h = (((k // b.shape[0]).double() + 0.5) / times - 0.5) * (2 * math.pi / 3)
        b = b[k % b.shape[0]]
        sd, cd = math.sin(0.6), math.cos(0.6)
        sh, ch = torch.sin(h), torch.cos(h)
        u = sh * b[:, 0] + ch * b[:, 1]
        v = -sd * ch * b[:, 0] + sd * sh * b[:, 1] + cd * b[:, 2]
        w = cd * ch * b[:, 0] - cd * sh * b[:, 1] + sd * b[:, 2]
        s = radius / torch.maximum(u.abs().max(), v.abs().max())
        return torch.stack([u * s, v * s, w * (wmax / w.abs().max())])
    if uv == "gauss":
        # normal, sigma a quarter of the radius, cut at the radius (the radius of a Rayleigh law)
        r = radius * 0.25 * torch.sqrt(-2.0 * torch.log1p(-_rand(g, n) * (1.0 - math.exp(-8.0))))
    else:
        r = radius * torch.sqrt(_rand(g, n))
    t = 2 * math.pi * _rand(g, n)
    w = (2.0 * _rand(g, n) - 1.0) * wmax
    return torch.stack([r * torch.cos(t), r * torch.sin(t), w])


def _padded(c):
    """Grid size of a case: the padded size is a multiple of four, as the drop-in call rounds it."""
    p = int(c["size"] * c["pad"])
    return p + (-p) % 4


def _snapshot(c, seed):
    g = _gen(seed)
    n, cell = c["n"], math.radians(c["cell"] / 3600.0)
    uvw = _coverage(g, n, c["uv"], c["reach"] * 0.5 / cell, c["wmax"])
    half = int(0.4 * c["size"])
    l = torch.round((2 * _rand(g, c["sources"]) - 1) * half) * cell
    m = torch.round((2 * _rand(g, c["sources"]) - 1) * half) * cell
    flux = 0.1 * 100.0 ** _rand(g, c["sources"])
    vis = torch.complex(0.05 * _randn(g, n), 0.05 * _randn(g, n))
    for a, b, f in zip(l.tolist(), m.tolist(), flux.tolist()):
        nn = math.sqrt(1.0 - a * a - b * b)
        ph = 2 * math.pi * (uvw[0] * a + uvw[1] * b + uvw[2] * (nn - 1.0))
        vis += torch.polar(torch.full_like(ph, f * nn), ph)
    weights = 0.5 + _rand(g, n)
    return {"vis": vis.to(torch.complex64) if c["vis"] == "c64" else vis, "weights": weights, "uvw": uvw}


def _keywords(c):
    kw = {"image_size": c["size"], "cell_size": c["cell"], "kernel_func": KERNEL[c["kernel"]],
          "kernel_support": c["support"], "kernel_exact": c["exact_kernel"], "oversampling": c["os"],
          "analytic_gcf": c["analytic"], "generate_beam": c["beam"], "padded_image_size": _padded(c)}
    if c["planes"]:
        kw.update(num_wplanes=c["planes"], max_wpconv_support=c["wsupport"], kernel_trunc_perc=c["trunc"])
    return kw


def _parts(c):
    """The snapshots of a batch case: sizes and counts are the case's, whatever the seed."""
    sizes = [int(s) for s in c["sizes"].split(",")]
    out = []
    for i in range(c["count"]):
        # counts spread over [nmin, nmax] (logarithm), large and small in turn
        f = ((i * 7) % c["count"] + 0.5) / c["count"]
        out.append(_case(SNAPSHOT, n=int(c["nmin"] * (c["nmax"] / c["nmin"]) ** f), size=sizes[i % len(sizes)],
                         wmax=2000.0 * ((i * 5) % c["count"] + 1) / c["count"], sources=5, planes=c["planes"],
                         wsupport=c["wsupport"], trunc=c["trunc"], precision=c["precision"],
                         kernel="gsinc" if i % 2 == 0 else "pswf"))
    return out


def _sky(c, seed):
    """An image as the imager leaves it: noise with point-like and extended sources of either sign (flat, the first
    axis of the memory being the image's columns)."""
    g = _gen(seed)
    rows, cols = c["rows"], c["cols"]
    img = _randn(g, cols, rows, dtype=torch.float32 if c["dtype"] == "fp32" else torch.float64)
    k = c["sources"]
    at = torch.stack([_rand(g, k) * (cols - 1), _rand(g, k) * (rows - 1)], 1).tolist()
    amp = (8.0 * 30.0 ** _rand(g, k)).tolist()
    wide = (1.2 + 4.0 * _rand(g, k) ** 3).tolist()
    for s in range(k):
        (x, y), r = at[s], wide[s]
        b = int(6 * r) + 1
        x0, x1, y0, y1 = max(0, int(x) - b), min(cols, int(x) + b), max(0, int(y) - b), min(rows, int(y) + b)
        dx = torch.arange(x0, x1, device="cuda", dtype=torch.float64) - x
        dy = torch.arange(y0, y1, device="cuda", dtype=torch.float64) - y
        blob = amp[s] * torch.exp(-0.5 * (dx[:, None] ** 2 + (dy[None, :] / 1.3) ** 2) / r ** 2)
        img[x0:x1, y0:y1] += (blob if s % 5 else -blob).to(img.dtype)
    return (img * 0.003).reshape(-1)


def _out_type(c):
    return (torch.float64, capi.F64) if c["precision"] == "fp64" else (torch.float32, capi.F32)


def prepare(case, seed):
    ctx = _context()
    if case["do"] == "find":
        state = {"image": _sky(case, seed),
                 "labels": torch.empty(case["rows"] * case["cols"], dtype=torch.int32, device="cuda")}
    elif case["do"] == "batch":
        snaps = []
        for i, c in enumerate(_parts(case)):
            d = _snapshot(c, seed * 64 + i)
            d.update(_keywords(c), image=torch.empty(c["size"] ** 2, dtype=_out_type(c)[0], device="cuda"))
            snaps.append(d)
        state = {"snapshots": snaps}
    else:
        state = _snapshot(case, seed)
        if case["do"] == "host":
            state = {"vis": state["vis"].cpu().numpy(), "weights": state["weights"].cpu().numpy(),
                     "uvw": state["uvw"].cpu().numpy().T}
        else:
            state["image"] = torch.empty(case["size"] ** 2, dtype=_out_type(case)[0], device="cuda")
            state["beam"] = torch.empty_like(state["image"]) if case["beam"] else None
        state["keywords"] = _keywords(case)
    torch.cuda.synchronize()
    return dict(state, case=case, context=ctx)


def run(state):
    c, ctx = state["case"], state["context"]
    if c["do"] == "find":
        islands, labels, info = ctx.source_find(state["image"], 5.0, 3.0, find_negative_sources=c["negative"],
                                                ccl_4connectivity=c["four"], gaussian_fitting=c["fit"],
                                                device_ptrs=True, rows=c["rows"], cols=c["cols"],
                                                label_out=state["labels"])
        out = {"labels": labels, "counts": np.array([info.n_labels_pos, info.n_labels_neg, len(islands)])}
        out["stats"] = np.array([info.bg_level, info.rms_est, info.mean, info.sigma])
        # a catalogue of fixed length, unused entries zero
        v = np.zeros(CATALOGUE, dtype=np.dtype(capi.Island))
        if islands:
            v[:len(islands)] = np.frombuffer(b"".join(map(bytes, islands)), dtype=v.dtype)
        out["islands"] = np.stack([v[k] for k in ("label_idx", "sign", "extremum_y_idx", "extremum_x_idx",
                                                  "num_samples", "bbox_top", "bbox_bottom", "bbox_left",
                                                  "bbox_right")])
        out["extrema"] = v["extremum_val"]
        out["moments"] = v["moments_fit"]
        out["fits"] = v["leastsq_fit"]
        return out
    precision, out_dtype = PRECISION[c["precision"]], _out_type(c)[1]
    if c["do"] == "batch":
        images, infos, _ = ctx.image_batch(state["snapshots"], precision=precision, out_dtype=out_dtype)
        return {"images": images, "totals": np.array([i.sample_grid_total for i in infos])}
    device = c["do"] == "image"
    image, beam, info = ctx.image_visibilities(state["vis"], state["weights"], state["uvw"], precision=precision,
                                               out_dtype=out_dtype, device_ptrs=device,
                                               image_out=state.get("image"), beam_out=state.get("beam"),
                                               **state["keywords"])
    # a host image comes in column-major order; its memory order is the device image's
    image = image if device else image.reshape(-1, order="F")
    out = {"image": image, "total": info.sample_grid_total}
    if c["beam"]:
        out["beam"] = beam if device else beam.reshape(-1, order="F")
    return out


# ------------------------------------------------------------------ what a pass needs

def _imaging_work(c):
    n, size, N = c["n"], c["size"], _padded(c)
    taps = (2 * (c["wsupport"] if c["planes"] and not c["trunc"] else c["support"]) + 1) ** 2
    images = 2 if c["beam"] else 1
    out = (8 if c["precision"] == "fp64" else 4) * size * size * images
    # a complex multiply-add per tap; 2.5 N log2 N per real transform of N points
    flops = 8.0 * n * taps * images + 2.5 * N * N * math.log2(N * N) * images
    return n * ((8 if c["vis"] == "c64" else 16) + 24 + 8) + out, flops


def work(case):
    if case["do"] == "find":
        px = case["rows"] * case["cols"]
        return {"bytes": px * ((4 if case["dtype"] == "fp32" else 8) + 4), "flops": 4.0 * px}
    w = [_imaging_work(c) for c in (_parts(case) if case["do"] == "batch" else [case])]
    return {"bytes": sum(b for b, _ in w), "flops": sum(f for _, f in w)}


def tolerance(case):
    if case["do"] == "find":
        # double-precision sums; the least-squares fits stop at a relative step of about 1e-8
        return {"rel": 1e-6 if case["fit"] else 1e-9, "max": 1e-5 if case["fit"] else 1e-7}
    if case["precision"] == "fp64":
        return {"rel": 1e-11, "max": 1e-8}
    # Single-precision kernel values and products; the grid correction multiplies what they leave by up to 1/gcf^2
    # towards the image's edge (890 for GaussianSinc, 1.5e4 and more for PSWF): 4e-6, 5e-5 and, with plain
    # single-precision sums and transform, up to 8e-4 were measured against exact().
    if case["do"] == "batch" or case["kernel"] == "pswf":
        return {"rel": 3e-3, "max": 0.5} if case["precision"] == "fp32" else {"rel": 2e-4, "max": 0.1}
    return {"rel": 2e-5, "max": 4e-3}


# ------------------------------------------------------------------ the same in 64 bits

def _kernel(c, r):
    """Anti-aliasing kernel at the distances r (numpy), zero beyond its support."""
    trunc = float(c["support"])
    if c["kernel"] == "gsinc":
        x = r * (math.pi / 1.55)
        x = np.where(x == 0.0, 1e-20, x)
        v = np.exp(-(r * r) / (2.52 * 2.52)) * (np.sin(x) / x)
    else:
        nu = r / trunc
        v = _spheroidal(nu) * (1.0 - nu * nu)
    return np.where(np.abs(r) > trunc, 0.0, v)


def _spheroidal(nu):
    """Schwab's rational approximation of the prolate spheroidal wave function (m = 6, alpha = 1)."""
    p = np.array([[8.203343e-2, -3.644705e-1, 6.278660e-1, -5.335581e-1, 2.312756e-1],
                  [4.028559e-3, -3.697768e-2, 1.021332e-1, -1.201436e-1, 6.412774e-2]])
    q = np.array([[1.0, 8.212018e-1, 2.078043e-1], [1.0, 9.599102e-1, 2.918724e-1]])
    nu = np.abs(nu)
    part = np.where(nu < 0.75, 0, 1)
    d = nu * nu - np.where(part == 0, 0.75, 1.0) ** 2
    top = sum(p[part, k] * d ** k for k in range(5))
    return np.where(nu <= 1.0, top / sum(q[part, k] * d ** k for k in range(3)), 0.0)


def _image_domain(c, n):
    """Grid correction over n pixels, the phase centre at n // 2."""
    centre = n // 2
    x = np.arange(n) - centre
    if c["analytic"]:
        return _spheroidal(x / centre)
    k = _kernel(c, x.astype(np.float64))
    return np.fft.fftshift(np.fft.fft(np.fft.ifftshift(k / k.sum())).real)


def _w_kernels(c, N, w_mean):
    """Per plane (support, table (cs, cs, K, K) over the oversampled offsets in v and u; rows along v)."""
    os, smax = c["os"], c["wsupport"]
    area = 2
    while area < 2 * smax + 1:
        area *= 2
    arr, half = area * os, area // 2
    cell = math.radians(c["cell"] / 3600.0) * N / area
    aa = torch.from_numpy(_image_domain(c, area)[half:].copy()).cuda()
    x = torch.arange(half, device="cuda", dtype=torch.float64) * cell
    r2 = (x[:, None] ** 2 + x[None, :] ** 2)
    near = r2 < 1.0
    nn = torch.sqrt(torch.where(near, 1.0 - r2, 1.0))
    taper = aa[:half, None] * aa[None, :half]
    at = torch.cat([torch.arange(half), arr - torch.arange(1, half)]).cuda()
    quad = torch.cat([torch.arange(half), torch.arange(1, half)]).cuda()
    offs = torch.arange(2 * (os // 2) + 1, device="cuda")
    tables = []
    for w in w_mean:
        ph = torch.where(near, -2.0 * math.pi * w * (nn - 1.0), 0.0)
        q = torch.polar(1.0 / nn, ph) * taper
        full = torch.zeros(arr, arr, dtype=torch.complex128, device="cuda")
        full[at[:, None], at[None, :]] = q[quad][:, quad]
        conv = torch.fft.fft2(full)
        S = smax
        if c["trunc"] > 0.0:
            line = conv[torch.arange(0, min(smax * os, arr // 2) + 1, os, device="cuda"), 0].abs()
            big = (line > line[0] * (c["trunc"] / 100.0)).nonzero()
            S = int(big.max()) if len(big) else 0
        t = torch.arange(2 * S + 1, device="cuda")
        k = ((t[None, :] - S) * os + os // 2 - offs[:, None]) % arr  # (cs, K)
        tab = conv[k[:, None, :, None], k[None, :, None, :]]
        tables.append((S, tab / tab.real.sum((2, 3), keepdim=True)))
    return tables


def _exact_image(c, seed):
    """(image, beam or None, sampling total) of an imaging case, double precision."""
    s = _snapshot(c, seed)
    N, os, size = _padded(c), c["os"], c["size"]
    S = c["wsupport"] if c["planes"] else c["support"]
    scale = math.radians(c["cell"] / 3600.0) * N
    u, v, w = s["uvw"][0] * scale, s["uvw"][1] * scale, s["uvw"][2]
    vis, wt = s["vis"].to(torch.complex128), s["weights"]
    # the lower half plane is its mirror image, conjugated; near v = 0 a visibility is gridded on both sides
    flip = v < 0.0
    twice = torch.where(flip, v > -(S + 1), v < S + 1)
    sign = torch.where(flip, -1.0, 1.0)
    u, v, w, vis = u * sign, v * sign, w * sign, torch.where(flip, vis.conj(), vis)
    ru, rv = torch.round(u), torch.round(v)
    kx, ky = ru.long() + N // 2, rv.long() + N // 2
    good = (kx - S > 0) & (ky - S > 0) & (kx + S < N) & (ky + S < N)
    fx, fy = u - ru, v - rv
    ox = torch.round(fx * os).long().clamp(-(os // 2), os // 2) + os // 2
    oy = torch.round(fy * os).long().clamp(-(os // 2), os // 2) + os // 2
    total = 2.0 * float(wt[good].sum())
    plane = torch.zeros_like(kx)
    tables = None
    if c["planes"]:
        # planes of equal counts of the visibilities ordered by |w|; those beyond the grid take a place in the order
        order = torch.sort(w.abs(), stable=True).indices
        aw, gs = w.abs()[order], good[order]
        cum = torch.cumsum(gs.long(), 0)
        ngood, n, begin, means = int(cum[-1]), len(aw), 0, []
        pl = torch.zeros_like(order)
        for p in range(c["planes"]):
            want = max(0, math.ceil((ngood - begin) / (c["planes"] - p)))
            before = int(cum[begin - 1]) if begin else 0
            end = min(int(torch.searchsorted(cum, before + want)) + 1, n) if want else begin
            sel = aw[begin:end][gs[begin:end]]
            means.append(float(sel.mean()) if len(sel) else 0.0)
            pl[begin:(n if p == c["planes"] - 1 else end)] = p
            begin = end
        plane[order] = pl
        tables = _w_kernels(c, N, means)
    elif not c["exact_kernel"]:
        d = (np.arange(2 * (os // 2) + 1) - os // 2)[:, None] / os
        k1 = _kernel(c, (np.arange(2 * S + 1) - S)[None, :] - d)
        k1 = torch.from_numpy(k1 / k1.sum(1, keepdims=True)).cuda()
    wide = c["os"] if not c["exact_kernel"] else 1
    gx, gy = torch.where(kx < N // 2, kx + N // 2, kx - N // 2), torch.where(ky < N // 2, ky + N // 2, ky - N // 2)
    rows = N // 2 + 1
    grids = [torch.zeros(N * rows * 2, dtype=torch.float64, device="cuda") for _ in range(2 if c["beam"] else 1)]
    supports = sorted({t[0] for t in tables}) if tables else [S]
    for mirror in (False, True):
        for sup in supports:
            pick = good & twice if mirror else good
            if tables:
                has = torch.tensor([t[0] == sup for t in tables], device="cuda")
                where = torch.cumsum(has.long(), 0) - 1
                stack = torch.stack([t[1] for t in tables if t[0] == sup])
                pick = pick & has[plane]
            i = pick.nonzero()[:, 0]
            if not len(i):
                continue
            x, y, vi, ww = gx[i], gy[i], vis[i], w[i]
            cx, cy, ax, ay = ox[i], oy[i], fx[i], fy[i]
            if mirror:
                x, y, vi, ww, ax, ay = N - x, N - y, vi.conj(), -ww, -ax, -ay
                cx, cy = wide - cx, wide - cy
            K = 2 * sup + 1
            if c["exact_kernel"]:
                t = torch.arange(K, device="cuda", dtype=torch.float64) - sup
                ky1 = torch.from_numpy(_kernel(c, (t[None, :] - ay[:, None]).cpu().numpy())).cuda()
                kx1 = torch.from_numpy(_kernel(c, (t[None, :] - ax[:, None]).cpu().numpy())).cuda()
                norm = ky1.sum(1) * kx1.sum(1)
            for b in range(K):
                col = x - sup + b
                col = torch.where(col < 0, col + N, torch.where(col >= N, col - N, col))
                for a in range(K):
                    row = y - sup + a
                    if c["exact_kernel"]:
                        row = torch.where(row < 0, row + N, row)
                        k = (ky1[:, a] * kx1[:, b] / norm).to(torch.complex128)
                    elif tables:
                        k = stack[where[plane[i]], cy, cx, a, b]
                        k = torch.where(ww < 0.0, k.conj(), k)
                    else:
                        k = (k1[cy, a] * k1[cx, b]).to(torch.complex128)
                    row = torch.where(row >= N, row - N, row)
                    ok = (row >= 0) & (row < rows)
                    cell = torch.where(ok, col * rows + row, 0)
                    k = torch.where(ok, k * wt[i], 0.0)
                    for g, val in zip(grids, (vi * k, k)):
                        g.view(-1, 2).index_add_(0, cell, torch.view_as_real(val))
    keep = torch.cat([torch.arange(size // 2), N - size // 2 + torch.arange(size // 2)]).cuda()
    gcf = torch.fft.ifftshift(torch.from_numpy(_image_domain(c, N)).cuda())[keep]
    out = []
    for g in grids:
        img = torch.fft.irfft2(torch.view_as_complex(g.view(N, rows, 2)), s=(N, N), norm="forward")
        out.append((img[keep][:, keep] / total / gcf[:, None] / gcf[None, :]).reshape(-1))
    return out[0], (out[1] if c["beam"] else None), total


def _exact_stats(c, seed):
    """(background, rms, mean, sigma): the binned median of the samples within one sigma and the clipped deviation."""
    x = _sky(c, seed).double()
    n = x.numel()
    mean = float(x.mean())
    sigma = math.sqrt(float(((x - mean) ** 2).sum()) / n)
    scale, left = 1000.0 / (2.0 * sigma), mean - sigma
    b = ((x - left) * scale).trunc().long()
    count = torch.cumsum(torch.bincount(b.clamp(-1, 1001) + 1, minlength=1003), 0).cpu().numpy()[1:1002]
    k = (n + 1) // 2
    i = j = int(np.argmax(count >= k))
    if n % 2 == 0 and count[i] == k:
        j = int(np.argmax(count > k))
    median = (i + 0.5) / scale + left if n % 2 else (i + j + 1) / (2.0 * scale) + left
    kept, s = x - median, sigma
    for _ in range(5):
        inside = kept[kept.abs() <= 3.0 * s]
        if inside.numel() == kept.numel():
            break
        kept = inside
        s = math.sqrt(float((kept ** 2).mean()) - float(kept.mean()) ** 2)
    return np.array([median, s, mean, sigma])


def exact(case, seed):
    if case["do"] == "find":
        out = {"labels": None, "counts": None, "stats": _exact_stats(case, seed), "islands": None, "extrema": None,
               "moments": None, "fits": None}
        return out
    if case["do"] == "batch":
        got = [_exact_image(c, seed * 64 + i) for i, c in enumerate(_parts(case))]
        return {"images": [g[0] for g in got], "totals": np.array([g[2] for g in got])}
    image, beam, total = _exact_image(case, seed)
    out = {"image": image, "total": total}
    if case["beam"]:
        out["beam"] = beam
    return out
