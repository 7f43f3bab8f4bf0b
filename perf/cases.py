"""The workloads that performance work on this package is measured on.

Each case is one pass through a public entry point, as an acquisition program
makes it: a colour of a field of view, its DAPI block, a whole field from
pinned host memory, a stitched deconvolution, the per-tile loop, the spot
finder alone, the drift of a round and the background subtraction.  Sizes,
settings and synthetic data are those of ``bench.py``'s workloads and their
odd neighbours; the fields are sparse (a few thousand puncta) and the hyb
threshold lies between the noise and the puncta, as one is set in use.

The spot tables come back in no particular order and of no fixed length, so a
pass orders them by the raw value at each spot (a whole number), then along a
slanted line through the field, and puts them into the fixed table that the
program stores, zero past the last.
"""
import math

import numpy as np
import torch

from mermake_gb300 import align, deconvolver, maxima, pipeline, synth
from mermake_gb300 import math as mm_math

HYB = dict(overlap=89, beta=1e-4, blur_radius=30, delta=1, delta_fit=3, sigmaZ=1, sigmaXY=1.5, threshold=10000)
DAPI = dict(overlap=89, beta=0.01, blur_radius=50, delta=5, delta_fit=5, sigmaZ=1, sigmaXY=1.5, threshold=3.0)
# puncta and nuclei per voxel of the field (x, y)
PUNCTA = 4000 / 2048 ** 2
NUCLEI = 300 / 2048 ** 2


def listed():
    return [
        # one smFISH tile, the smallest call: launches and the single-tile forms
        dict(name="hyb_tile", path="hyb", Z=40, X=500, Y=500, tile=500, psfs=1, flat=False),
        # one colour of the usual field: 25 tiles of 500 behind a flat field
        dict(name="hyb_field", path="hyb", Z=50, X=2048, Y=2048, tile=500, psfs=1, flat=True),
        # a PSF per tile across an 8 x 8 grid of tiles of 300, the last ones cut
        dict(name="hyb_psf_grid", path="hyb", Z=40, X=2345, Y=2389, tile=300, psfs=64, flat=False),
        # a depth and a field that divide by nothing
        dict(name="hyb_odd", path="hyb", Z=37, X=1111, Y=1313, tile=500, psfs=1, flat=True),
        # the DAPI block: stitched volume, RMS, maxima of both signs with the wide sphere
        dict(name="dapi_block", path="dapi", Z=50, X=1500, Y=1302, tile=500),
        # a whole field, 3 colours and DAPI, from pinned host memory to host tables
        dict(name="field_from_host", path="fov", Z=50, X=2048, Y=2048, tile=500, colours=3),
        # a stitched deconvolution kept as a volume (no blur), uint16 in
        dict(name="apply_volume", path="apply", Z=50, X=1000, Y=1500, tile=500, blur=0, dtype="uint16"),
        # the same with the background blur, float32 in (a volume the user has worked on), smaller tiles
        dict(name="apply_float", path="apply", Z=30, X=650, Y=811, tile=300, blur=30, dtype="float32"),
        # the reference's own per-tile loop, tile by tile with its raw view
        dict(name="tile_loop", path="loop", Z=40, X=900, Y=870, tile=300),
        # the spot finder and fit alone, on a volume with tens of thousands of maxima
        dict(name="maxima_volume", path="maxima", Z=50, X=1024, Y=1000, delta=1, fit=3),
        # the drift of one round's DAPI maxima against the resident first round
        dict(name="drift_round", path="drift", points=6000),
        # a colour minus its background round, shifted by the drift (strided views)
        dict(name="background", path="background", Z=50, X=2048, Y=2048, dz=1, dx=7, dy=-12),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["hyb", "hyb", "hyb", "dapi", "fov", "apply", "loop", "maxima", "drift", "background"])
    depth = rng.choice([30, 40, 50, 50, rng.randint(24, 56)])
    if path in ("hyb", "dapi", "apply"):
        tile = rng.choice([200, 300, 300, 500, 500, 500])
        X, Y = _side(rng, 520, 2048), _side(rng, 520, 2048)
        if path == "hyb":
            one = rng.random() < 0.7 or tile == 500
            nt = -(-X // tile) * -(-Y // tile)
            return dict(path=path, Z=depth, X=X, Y=Y, tile=tile, psfs=1 if one else nt, flat=rng.random() < 0.6)
        if path == "dapi":
            return dict(path=path, Z=depth, X=min(X, 1500), Y=min(Y, 1500), tile=tile)
        return dict(path=path, Z=depth, X=X, Y=Y, tile=tile, blur=rng.choice([0, 30, 50]),
                    dtype=rng.choice(["uint16", "float32"]))
    if path == "fov":
        return dict(path=path, Z=depth, X=_side(rng, 600, 1800), Y=_side(rng, 600, 1800), tile=500,
                    colours=rng.randint(1, 3))
    if path == "loop":
        return dict(path=path, Z=depth, X=_side(rng, 520, 1300), Y=_side(rng, 520, 1300), tile=rng.choice([300, 500]))
    if path == "maxima":
        delta, fit = rng.choice([(1, 3), (1, 3), (2, 3), (5, 5)])
        return dict(path=path, Z=depth, X=_side(rng, 200, 1500), Y=_side(rng, 200, 1500), delta=delta, fit=fit)
    if path == "drift":
        return dict(path=path, points=_side(rng, 500, 12000))
    return dict(path=path, Z=depth, X=_side(rng, 512, 2048), Y=_side(rng, 512, 2048), dz=rng.randint(-2, 2),
                dx=rng.randint(-20, 20), dy=rng.randint(-20, 20))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _psfs(case):
    """One PSF, or one per tile with its width growing across the field."""
    n = case.get("psfs", 1)
    if n == 1:
        return synth.gaussian_psf((40, 40, 40), 2.0, 1.3)
    return {i: synth.gaussian_psf((40, 40, 40), 1.8 + 0.6 * i / (n - 1), 1.1 + 0.5 * i / (n - 1)) for i in range(n)}


def _colour(case, seed, gain=None):
    X, Y = case["X"], case["Y"]
    return synth.hyb_stack(case["Z"], X, Y, max(8, int(PUNCTA * X * Y)), seed, device="cuda", sigma_z=2.0,
                           sigma_xy=1.5, gain=gain)


def _nuclei(case, seed):
    X, Y = case["X"], case["Y"]
    return synth.dapi_stack(case["Z"], X, Y, seed, device="cuda", n_nuclei=max(4, int(NUCLEI * X * Y)))


def _hyb_dec(case):
    Z = case["Z"]
    return deconvolver.Deconvolver(_psfs(case), (Z, case["X"], case["Y"]), tile_size=case["tile"], zpad=Z - 1, **HYB)


def _dapi_dec(case):
    Z = case["Z"]
    return deconvolver.Deconvolver(_psfs(case), (Z, case["X"], case["Y"]), tile_size=case["tile"], zpad=(Z - 1) // 2,
                                   **DAPI)


def _points(n, seed):
    """A round's maxima (z, x, y) with heights, and those of the drifted next
    round: a tenth lost, a tenth new, a quarter of a pixel of jitter."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    box = torch.tensor([50.0, 2048.0, 2048.0], device="cuda")
    ref = torch.rand((n, 3), generator=g, device="cuda") * box
    shift = (torch.rand(3, generator=g, device="cuda") * 2 - 1) * torch.tensor([2.5, 19.0, 19.0], device="cuda")
    mov = ref + shift + 0.25 * torch.randn((n, 3), generator=g, device="cuda")
    lost = torch.rand(n, generator=g, device="cuda") < 0.1
    mov = torch.where(lost[:, None], torch.rand((n, 3), generator=g, device="cuda") * box, mov)
    h = 5 + torch.rand((n, 2), generator=g, device="cuda")
    return torch.cat([ref, h[:, :1]], 1), torch.cat([mov, h[:, 1:]], 1)


def prepare(case, seed):
    path = case["path"]
    s = dict(case=case, line=_line(case))
    if path == "hyb":
        gain = synth.flat_gain(case["X"], case["Y"]) if case["flat"] else None
        s["image"] = _colour(case, seed, gain)
        s["flat"] = None if gain is None else torch.from_numpy(gain).cuda()
        s["dec"] = _hyb_dec(case)
    elif path == "dapi":
        s["image"] = _nuclei(case, seed)
        s["dec"] = _dapi_dec(case)
        s["buffer"] = torch.empty((case["Z"], case["X"], case["Y"]), dtype=torch.float32, device="cuda")
    elif path == "fov":
        gain = synth.flat_gain(case["X"], case["Y"])
        s["dapi"] = _nuclei(case, seed).cpu().pin_memory()
        s["colours"] = [_colour(case, seed + 17 * (c + 1), gain).cpu().pin_memory() for c in range(case["colours"])]
        s["flats"] = [torch.from_numpy(gain).cuda()] * case["colours"]
        s["runner"] = pipeline.FovRunner(_hyb_dec(case), _dapi_dec(case), HYB, DAPI)
    elif path in ("apply", "loop"):
        s["image"] = _colour(case, seed)
        if case.get("dtype") == "float32":
            s["image"] = s["image"].to(torch.float32)
        s["dec"] = _hyb_dec(case)
        if path == "apply":
            s["output"] = torch.zeros((case["Z"], case["X"], case["Y"]), dtype=torch.float32, device="cuda")
    elif path == "maxima":
        # a deconvolved volume: puncta over noise, already float32, with the raw stack beside it
        raw = _colour(case, seed)
        g = torch.Generator(device="cuda")
        g.manual_seed(seed + 1)
        noise = torch.randn(raw.shape, generator=g, device="cuda")
        s["image"] = (raw.to(torch.float32) - 600.0) * 4.0 + 900.0 * noise
        s["raw"] = raw
    elif path == "drift":
        ref, s["moved"] = _points(case["points"], seed)
        s["aligner"] = align.Aligner(ref, th=4)
    elif path == "background":
        s["signal"] = _colour(case, seed)
        s["ground"] = _colour(case, seed + 1)
        sig, bk = [], []
        for d, n in zip((case["dz"], case["dx"], case["dy"]), s["signal"].shape):
            sig.append(slice(max(d, 0), n + min(d, 0)))
            bk.append(slice(max(-d, 0), n - max(d, 0)))
        s["slices"] = tuple(sig), tuple(bk)
    else:
        raise ValueError(path)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _order(rows, size, line):
    """A table of `size` rows, ordered by their place along `line` (``_line``)."""
    place = rows.double()
    place[:, 5].round_()
    table = rows.new_zeros((size, 8))
    table[:rows.shape[0]] = rows[torch.argsort(place @ line)]
    return table


def _line(case):
    """Weights of a row's columns in its place: the raw value at the spot first
    (for a volume given as it is the height in column 7, an input value), then a
    slanted line through the field, on which no mirrored pair shares a place."""
    by = [0.0, 2.0 ** 26] if case["path"] == "maxima" else [2.0 ** 13, 0.0]
    line = torch.tensor([1.37, 1.0, 0.618, 0.0, 0.0, by[0], 0.0, by[1]], dtype=torch.float64)
    return line if case["path"] == "fov" else line.cuda()


def _size(case):
    """Rows of the stored table: several times the spots a field of this size has."""
    area = case["X"] * case["Y"]
    if case["path"] == "maxima":
        return int(0.12 * area) + 1024
    return int(8 * PUNCTA * area) + 1024


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "hyb":
        rows = pipeline.hyb_spots(state["dec"], state["image"], state["flat"], **HYB)
        return _order(rows, _size(case), state["line"])
    if path == "dapi":
        plus, minus, buffer, rms = pipeline.dapi_spots(state["dec"], state["image"], None, buffer=state["buffer"],
                                                       **DAPI)
        n = _size(case)
        return dict(plus=_order(plus, n, state["line"]), minus=_order(minus, n, state["line"]), buffer=buffer, rms=rms)
    if path == "fov":
        r = state["runner"]
        plus, minus, colours = r.run(r.submit(state["dapi"], state["colours"]), state["flats"])
        return [_order(torch.from_numpy(t), _size(case), state["line"]) for t in [plus, minus] + colours]
    if path == "apply":
        return state["dec"].apply(state["image"], None, blur_radius=case["blur"] or None, output=state["output"])
    if path == "loop":
        # the reference's loop: maxima of each tile, kept inside its overlap, moved to the field's coordinates
        ov, out = HYB["overlap"], []
        for x, y, tile, raw in state["dec"].tile_wise(state["image"], None, **HYB):
            rows = maxima.find_local_maxima(tile, raw=raw, **HYB)
            hi = torch.tensor([tile.shape[1] - ov, tile.shape[2] - ov], device=rows.device)
            rows = rows[torch.all((rows[:, 1:3] >= ov) & (rows[:, 1:3] < hi), dim=-1)]
            rows[:, 1] += x - ov
            rows[:, 2] += y - ov
            out.append(rows)
        return _order(torch.cat(out), _size(case), state["line"])
    if path == "maxima":
        return _order(maxima.find_local_maxima(state["image"], threshold=3000.0, delta=case["delta"],
                                               delta_fit=case["fit"], raw=state["raw"]), _size(case),
                      state["line"])
    if path == "drift":
        t, n = state["aligner"].get_best_translation_points(state["moved"], return_counts=True)
        return dict(shift=t, count=int(n))
    sig, bk = state["slices"]
    out = mm_math.subtract_reflect(state["signal"][sig], state["ground"][bk])
    return out.view(torch.int16)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _deconv_work(case, zpad, dtype_bytes, flat):
    """Bytes and flops of the tiled deconvolution: the channel and the flat
    read once, the spectrum of the z step read once per PSF; real 2-D
    transforms of every tile's planes both ways, a complex transform pair
    along the padded depth per frequency and the product between them."""
    Z, X, Y, ts = case["Z"], case["X"], case["Y"], case["tile"]
    P, Zp = ts + 178, Z + 2 * zpad
    nt = -(-X // ts) * -(-Y // ts)
    spectrum = Zp * P * (P // 2 + 1)
    bytes_ = dtype_bytes * Z * X * Y + (4.0 * X * Y if flat else 0.0) + 8.0 * spectrum * case.get("psfs", 1)
    flops = nt * (2 * 2.5 * Z * P * P * math.log2(P * P) + spectrum * (2 * 5 * math.log2(Zp) + 6))
    return bytes_, flops


def work(case):
    path = case["path"]
    if path in ("hyb", "loop", "apply", "dapi", "fov"):
        Z, X, Y = case["Z"], case["X"], case["Y"]
        vox, puncta = Z * X * Y, PUNCTA * X * Y
        if path == "fov":
            b, f = _deconv_work(case, Z - 1, 2, True)
            bd, fd = _deconv_work(case, (Z - 1) // 2, 2, False)
            return dict(bytes=case["colours"] * (b + 32 * puncta) + bd, flops=case["colours"] * f + fd)
        b, f = _deconv_work(case, (Z - 1) // 2 if path == "dapi" else Z - 1, 4 if case.get("dtype") == "float32" else 2,
                            case.get("flat", False))
        return dict(bytes=b + (4.0 * vox if path in ("apply", "dapi") else 32 * puncta), flops=f)
    if path == "maxima":
        # the volume once; about a thousand flops a fitted spot are nothing beside it
        vox = case["Z"] * case["X"] * case["Y"]
        return dict(bytes=4.0 * vox, flops=(1 + 6) * vox)
    if path == "drift":
        n = case["points"]
        return dict(bytes=16.0 * 2 * n, flops=5 * 27.0 * 8 * n)
    vox = (case["Z"] - abs(case["dz"])) * (case["X"] - abs(case["dx"])) * (case["Y"] - abs(case["dy"]))
    return dict(bytes=6.0 * vox, flops=vox)


# ---------------------------------------------------------------------------
# the same results in 64 bits, from torch alone
# ---------------------------------------------------------------------------
def _place(n, first, d, ov):
    """Source index of each of the n padded positions along x or y (-1: zero):
    the tile placed at ov and mirrored inwards at a field's first edge, placed
    at 0 and mirrored outwards where it is cut."""
    j = torch.arange(n)
    if first:
        q = torch.where((j < ov) & (2 * ov - j < n), 2 * ov - j, j)
        return torch.where((q >= ov) & (q < ov + d), q - ov, torch.full_like(q, -1))
    q = torch.where(j < d, j, 2 * (d - 1) - j) if d < n else j
    return torch.where((q >= 0) & (q < d), q, torch.full_like(q, -1))


def _place_z(Z, zpad):
    n = Z + 2 * zpad
    src = torch.full((n,), -1, dtype=torch.long)
    src[zpad:zpad + Z] = torch.arange(Z)
    for j in range(zpad):  # inwards about the first plane, then outwards about the last
        if 2 * zpad - j < n:
            src[j] = src[2 * zpad - j].clone()
    for j in range(zpad + Z, n):
        if 2 * (zpad + Z - 1) - j >= 0:
            src[j] = src[2 * (zpad + Z - 1) - j].clone()
    return src


def _take(t, idx, dim):
    idx = idx.to(t.device)
    t = t.index_select(dim, idx.clamp(min=0))
    shape = [1] * t.dim()
    shape[dim] = -1
    return t * (idx >= 0).view(shape)


def _wiener(psf, Z, ts, zpad, ov, beta):
    p = torch.from_numpy(np.asarray(psf)).cuda().double()
    tgt = (Z, ts, ts)
    c = torch.zeros(tgt, dtype=torch.float64, device="cuda")
    to, fr = [], []
    for a, b in zip(tgt, p.shape):
        m = min(a, b)
        to.append(slice(max(0, (a - b) // 2), max(0, (a - b) // 2) + m))
        fr.append(slice(max(0, (b - a) // 2), max(0, (b - a) // 2) + m))
    c[tuple(to)] = p[tuple(fr)]
    c /= c.sum()
    full = torch.zeros((Z + 2 * zpad, ts + 2 * ov, ts + 2 * ov), dtype=torch.float64, device="cuda")
    full[zpad:zpad + Z, ov:ov + ts, ov:ov + ts] = c
    full = torch.roll(full, [(-n) // 2 for n in full.shape], (0, 1, 2))
    H = torch.fft.rfftn(full)
    lap = torch.zeros_like(full)
    z, x, y = (n // 2 for n in full.shape)
    lap[z, x, y] = 6
    for o in ((-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1)):
        lap[z + o[0], x + o[1], y + o[2]] = -1
    L = torch.fft.rfftn(lap)
    return H.conj() / ((H * H.conj()).real + beta * (L * L.conj()).real)


def _box_mean(a, d, dim):
    n = a.shape[dim]
    zero = torch.zeros_like(a.narrow(dim, 0, 1))
    c = torch.cat([zero, a.cumsum(dim)], dim)
    i = torch.arange(n, device=a.device)
    lo, hi = (i - d).clamp(min=0), (i + d + 1).clamp(max=n)
    shape = [1] * a.dim()
    shape[dim] = -1
    return (c.index_select(dim, hi) - c.index_select(dim, lo)) / (hi - lo).view(shape)


def _exact_tiles(image, psfs, flat, ts, ov, zpad, beta, blur):
    """(x, y, result, raw) of every tile, as Deconvolver.tile_wise yields them."""
    Z, X, Y = image.shape
    P, psfs = ts + 2 * ov, list(psfs.values()) if isinstance(psfs, dict) else [psfs]
    tiles = [(x, y) for x in range(0, X, ts) for y in range(0, Y, ts)]
    if len(psfs) > 1:
        tiles = tiles[:len(psfs)]
    W = _wiener(psfs[0], Z, ts, zpad, ov, beta) if len(psfs) == 1 else None
    for k, (x, y) in enumerate(tiles):
        x0, x1, y0, y1 = max(x - ov, 0), min(x + ts + ov, X), max(y - ov, 0), min(y + ts + ov, Y)
        xd, yd = x1 - x0, y1 - y0
        t = image[:, x0:x1, y0:y1].double()
        f = torch.ones((xd, yd), dtype=torch.float64, device="cuda") if flat is None else flat[x0:x1, y0:y1].double()
        plane = _take(_take(t / f, _place(P, x == 0, xd, ov), 1), _place(P, y == 0, yd, ov), 2)
        pad = _take(plane, _place_z(Z, zpad), 0)
        w = W if W is not None else _wiener(psfs[k], Z, ts, zpad, ov, beta)
        res = torch.fft.irfftn(torch.fft.rfftn(pad) * w, s=pad.shape)[zpad:zpad + Z]
        if blur:
            res = res - _box_mean(_box_mean(res, blur // 2, 1), blur // 2, 2)
        xs, ys = (ov if x == 0 else 0), (ov if y == 0 else 0)
        raw = plane.clone()
        raw[:, xs:xs + xd, ys:ys + yd] = t
        xe = min(xd + (ov if x == 0 or xd < P else 0), P)
        ye = min(yd + (ov if y == 0 or yd < P else 0), P)
        yield x, y, res[:, :xe, :ye], raw[:, :xe, :ye]


def _reflect(i, n):
    i = torch.where(i < 0, -i, i)
    return torch.where(i >= n, 2 * n - i - 2, i)


def _exact_maxima(vol, raw, th, delta, fit, sigma_z=1.0, sigma_xy=1.5, band=None):
    """Rows of the local maxima of a volume above th, by find_local_maxima's
    definition; band: only maxima with x and y this far inside the edges."""
    Z, X, Y = vol.shape

    def at(t, z, x, y):
        return t.reshape(-1)[(_reflect(z, Z) * X + _reflect(x, X)) * Y + _reflect(y, Y)]

    vol, raw = vol.contiguous(), raw.contiguous()
    up = vol > th
    if band is not None:
        keep = torch.zeros_like(up)
        keep[:, band:X - band, band:Y - band] = True
        up &= keep
    z, x, y = up.nonzero(as_tuple=True)
    v = at(vol, z, x, y)
    r = range(-delta, delta + 1)
    for o in ((a, b, c) for a in r for b in r for c in r):
        if 0 < o[0] ** 2 + o[1] ** 2 + o[2] ** 2 <= delta ** 2:
            ok = ~(v < at(vol, z + o[0], x + o[1], y + o[2]))
            z, x, y, v = z[ok], x[ok], y[ok], v[ok]
    r = range(-fit, fit + 1)
    ball = [(a, b, c) for a in r for b in r for c in r if a * a + b * b + c * c <= fit * fit]
    ball = torch.tensor(ball, device="cuda")
    dz, dx, dy = (ball[:, i].double() for i in range(3))
    G = torch.exp(-(dz ** 2 / (2 * sigma_z ** 2) + (dx ** 2 + dy ** 2) / (2 * sigma_xy ** 2)))[None]
    rows = []
    for c in range(0, max(1, len(z)), 50000):
        zc, xc, yc = z[c:c + 50000], x[c:c + 50000], y[c:c + 50000]
        idx = (zc[:, None] + ball[None, :, 0], xc[:, None] + ball[None, :, 1], yc[:, None] + ball[None, :, 2])
        a, b = at(vol, *idx).double(), at(raw, *idx).double()
        bg = a.min(1).values if len(zc) else a.sum(1)
        w = a - bg[:, None]
        sw = w.sum(1)
        cen = [torch.where(sw > 0, p + (w * d[None]).sum(1) / sw, p.double())
               for p, d in ((zc, dz), (xc, dx), (yc, dy))]
        g = G - G.mean()

        def corr(t):
            t = t - t.mean(1, keepdim=True)
            sd = t.square().mean(1).sqrt()
            return (t * g).mean(1) / (torch.where(sd > 0, sd, torch.ones_like(sd)) * g.square().mean().sqrt())

        high, top = at(raw, zc, xc, yc).double(), at(vol, zc, xc, yc).double()
        rows.append(torch.stack(cen + [bg, corr(b), high, corr(a), top], 1))
    return torch.cat(rows)


def _exact_spots(image, psfs, flat, case):
    ov, out = HYB["overlap"], []
    Z, fit = case["Z"], HYB["delta_fit"]
    for x, y, res, raw in _exact_tiles(image, psfs, flat, case["tile"], ov, Z - 1, HYB["beta"], HYB["blur_radius"]):
        if res.shape[1] <= 2 * ov or res.shape[2] <= 2 * ov:
            continue
        rows = _exact_maxima(res, raw, HYB["threshold"], HYB["delta"], fit, band=ov - fit - 1)
        hi = torch.tensor([res.shape[1] - ov, res.shape[2] - ov], device="cuda")
        rows = rows[torch.all((rows[:, 1:3] >= ov) & (rows[:, 1:3] < hi), dim=-1)]
        rows[:, 1] += x - ov
        rows[:, 2] += y - ov
        out.append(rows)
    return _order(torch.cat(out), _size(case), _line(case))


def _exact_volume(image, psfs, case, zpad, beta, blur):
    ov, ts = HYB["overlap"], case["tile"]
    out = torch.zeros(tuple(image.shape), dtype=torch.float64, device="cuda")
    for x, y, res, _ in _exact_tiles(image, psfs, None, ts, ov, zpad, beta, blur):
        nx, ny = min(res.shape[1] - 2 * ov, image.shape[1] - x), min(res.shape[2] - 2 * ov, image.shape[2] - y)
        out[:, x:x + nx, y:y + ny] = res[:, ov:ov + nx, ov:ov + ny]
    return out


def exact(case, seed):
    path = case["path"]
    if path in ("drift", "background", "fov") or case.get("psfs", 1) > 16:
        # whole numbers and a host search; a whole field and a PSF per tile repeat what the others do, and take too long
        return None
    s = dict(prepare(case, seed))
    s.pop("dec", None)
    if path in ("hyb", "loop"):
        return _exact_spots(s["image"], _psfs(case), s.get("flat"), case)
    if path == "apply":
        return _exact_volume(s["image"], _psfs(case), case, case["Z"] - 1, HYB["beta"], case["blur"])
    if path == "maxima":
        return _order(_exact_maxima(s["image"], s["raw"].to(torch.float32), 3000.0, case["delta"], case["fit"]),
                      _size(case), _line(case))
    vol = _exact_volume(s["image"], _psfs(case), case, (case["Z"] - 1) // 2, DAPI["beta"], DAPI["blur_radius"])
    rms = float(vol.square().mean().sqrt())
    raw = s["image"].to(torch.float32)
    rows = [_order(_exact_maxima(sign * vol / rms, raw, DAPI["threshold"], DAPI["delta"], DAPI["delta_fit"]),
                   _size(case), _line(case)) for sign in (1.0, -1.0)]
    return dict(plus=rows[0], minus=rows[1], buffer=vol, rms=rms)
