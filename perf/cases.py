"""Timed cases of the deconvolution framework: what users run, through the public entry points.

The volumes are device-resident (the form in which a pipeline hands a frame from its reader to the
deconvolution and on to the deskew), column-major ``[ny nx nz]`` as torch tensors of shape
``(nz, nx, ny)``; uint16 volumes are int16 tensors holding the same bits.  A case is one of

* ``decon``: ``decon.decon_device``, OMW (Wiener-type backprojector) or Biggs RL on one volume;
* ``batch``: ``pk_batch_decon`` on device chunks, each cropped to its core (chunked large volumes);
* ``dsr``:   ``deskew.deskew_rotate_device`` on a deconvolved uint16 frame.

Deconvolved volumes are returned in single precision (``save16bit`` false), so every digit of the
computation is seen; the deskew returns uint16, as the pipeline stores it.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from petakit5d_b200 import _lib, decon, deskew

BACKGROUND = 100.0
EPS = 2.0 ** -52


def _decon(name, method, shape, iters, psf, dtype="uint16", erosion=0, empty=False, border=0):
    ny, nx, nz = shape
    return {"name": name, "kind": "decon", "method": method, "ny": ny, "nx": nx, "nz": nz, "iters": iters, "psf": psf,
            "dtype": dtype, "erosion": erosion, "empty": empty, "border": border}


def listed():
    return [
        # preview of a small crop while a parameter (alpha, iterations) is being chosen: launches and latency
        _decon("omw_crop_96x96x48", "omw", (96, 96, 48), 2, "bead"),
        # the demo's small volume, 20 RL iterations
        _decon("rl_128x128x64", "rl", (128, 128, 64), 20, "bead"),
        # one light-sheet frame, the benchmark's headline volume
        _decon("omw_512x512x256", "omw", (512, 512, 256), 2, "lattice"),
        # traditional RL on a frame kept in single precision after flat-field correction
        _decon("rl_512x512x128_single", "rl", (512, 512, 128), 10, "bead", dtype="float32"),
        # a deskewed and rotated frame: ragged sizes, empty corners, eroded edges
        _decon("omw_dsr_512x1140x270_eroded", "omw", (512, 1140, 270), 2, "bead", erosion=8, empty=True),
        # a region of interest drawn by hand: odd sizes with large prime factors
        _decon("rl_roi_301x467x97", "rl", (301, 467, 97), 10, "bead"),
        # a wide-field image (one plane), traditional RL
        _decon("rl_plane_2048x2048", "rl", (2048, 2048, 1), 20, "bead", dtype="float32"),
        # one 512^3 chunk of a stitched volume with its overlap, cropped to the core
        _decon("omw_chunk_576x544x544", "omw", (576, 544, 544), 2, "bead", border=16),
        # a whole stitched tile
        _decon("omw_1024x1024x512", "omw", (1024, 1024, 512), 2, "lattice"),
        # uneven chunks with 16-voxel overlaps and three PSFs in one call
        {"name": "omw_batch_16_chunks", "kind": "batch", "iters": 2, "border": 16,
         "shapes": "224x288x128 288x288x160 352x224x224 416x416x288 288x352x128 224x416x160 416x352x224 352x288x288 "
                   "288x416x224 224x224x128 416x224x288 352x352x160 288x224x288 416x288x128 352x416x224 224x352x160"},
        # the deskew / rotate after the deconvolution, at the demo's geometry
        {"name": "dsr_512x512x256", "kind": "dsr", "ny": 512, "nx": 512, "nz": 256, "angle": 32.45, "dz": 0.3,
         "pixel": 0.108},
    ]


def _log_size(rng, lo, hi):
    """An integer between lo and hi, even over the logarithm; a multiple of 16 half of the time, as
    camera windows are."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, v // 16 * 16) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["omw", "omw", "omw", "rl", "rl", "plane", "batch", "dsr"])
    if kind == "dsr":
        return {"kind": "dsr", "ny": _log_size(rng, 128, 640), "nx": _log_size(rng, 128, 640),
                "nz": _log_size(rng, 64, 320), "angle": rng.choice([31.5, 32.45]), "dz": rng.choice([0.2, 0.3, 0.4]),
                "pixel": 0.108}
    if kind == "batch":
        n = rng.randint(4, 16)
        sh = ["%dx%dx%d" % (rng.choice([192, 256, 320, 384]) + 32, rng.choice([192, 256, 320, 384]) + 32,
                            rng.choice([96, 128, 192, 256]) + 32) for _ in range(n)]
        return {"kind": "batch", "iters": 2, "border": 16, "shapes": " ".join(sh)}
    dtype = rng.choice(["uint16", "uint16", "float32"])
    if kind == "plane":
        c = _decon("", "rl", (_log_size(rng, 256, 2048), _log_size(rng, 256, 2048), 1), rng.randint(5, 20), "bead", dtype)
    else:
        iters = rng.randint(1, 3) if kind == "omw" else rng.randint(4, 20)
        while True:
            shape = (_log_size(rng, 64, 1024), _log_size(rng, 64, 1024), _log_size(rng, 32, 512))
            if math.prod(shape) * iters <= 100e6:
                break
        erosion = rng.choice([0, 0, 0, 8])
        border = rng.choice([0, 0, 12]) if not erosion else 0
        c = _decon("", kind, shape, iters, rng.choice(["bead", "bead", "lattice"]), dtype, erosion,
                   erosion > 0 and rng.random() < 0.5, border)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _psf_pair(kind, ny, nx, nz, sigma=1.3):
    """(PSF, backprojector) for a volume: a bead's Gaussian, or a lattice light sheet's with side
    lobes in z; the backprojector is a Wiener filter under a Butterworth window, at the PSF's size."""
    size = (31, 31, 41) if kind == "bead" else (64, 64, 101)
    n = [min(a, b) for a, b in zip(size, (ny, nx, nz))]
    y, x, z = np.meshgrid(*[np.arange(k) - k // 2 for k in n], indexing="ij")
    sz = 3.0 if kind == "bead" else 4.0
    p = np.exp(-(z / sz) ** 2 / 2)
    if kind != "bead":
        p = p + 0.15 * (np.exp(-((z - 12) / sz) ** 2 / 2) + np.exp(-((z + 12) / sz) ** 2 / 2))
    p = p * np.exp(-(y * y + x * x) / (2 * sigma ** 2))
    p = (p / p.sum()).astype(np.float32)
    H = np.fft.fftn(np.fft.ifftshift(p.astype(np.float64)))
    f = np.meshgrid(*[np.fft.fftfreq(k) for k in n], indexing="ij")
    r2 = sum((a / c) ** 2 for a, c in zip(f, (0.28, 0.28, 0.14)))
    b = np.fft.fftshift(np.fft.ifftn(np.conj(H) / (np.abs(H) ** 2 + 0.005) / np.sqrt(1 + r2 ** 8)).real)
    return np.asfortranarray(p), np.asfortranarray(b.astype(np.float32))


def _blur(img, axis, sigma):
    out = torch.zeros_like(img)
    for k in range(-3, 4):
        out.add_(torch.roll(img, k, axis), alpha=math.exp(-k * k / (2 * sigma * sigma)))
    return out


def _frame(ny, nx, nz, seed, empty=False):
    """A (nz, nx, ny) int16 tensor with the bits of a uint16 frame: blurred puncta over a smooth background
    on the camera's offset, shot noise; ``empty`` zeroes the corners that a deskewed frame has."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    img = torch.rand((nz, nx, ny), generator=g, device="cuda")
    img = torch.where(img < 1.5e-4, img * 4.0e7, torch.zeros_like(img))
    for axis, sigma in ((0, 2.0), (1, 1.6), (2, 1.6)):
        if img.shape[axis] > 6:
            img = _blur(img, axis, sigma).mul_(1 / (sigma * math.sqrt(2 * math.pi)))
    w = [torch.sin(torch.arange(k, device="cuda", dtype=torch.float32) * (2 * math.pi / 200)) for k in (nz, nx, ny)]
    img.add_(150 * (1 + (w[0].view(-1, 1, 1) + 0.5) * w[1].view(1, -1, 1) * w[2].view(1, 1, -1)) + BACKGROUND)
    noise = torch.randn(img.shape, generator=g, device="cuda")
    img = torch.clamp(torch.round(img + noise.mul_(img.sqrt())), 1, 65535)
    if empty:
        z = torch.arange(nz, device="cuda").view(-1, 1)
        x = torch.arange(nx, device="cuda").view(1, -1)
        s = x * nz - z * (nx // 2)
        img = img * ((s >= 0) & (s < nz * (nx - nx // 2))).unsqueeze(2)
    img = img.to(torch.int32)
    return torch.where(img > 32767, img - 65536, img).to(torch.int16)


def _u16(t):
    return t.to(torch.int32) & 0xFFFF


def _volume(c, seed):
    v = _frame(c["ny"], c["nx"], c["nz"], seed, c["empty"])
    return _u16(v).to(torch.float32).mul_(1.03125) if c["dtype"] == "float32" else v


def _box(shape, border):
    """[y1 x1 z1 y2 x2 z2] without ``border`` voxels at each face (none off an axis too short for it)."""
    b = [border if n > 2 * border else 0 for n in shape]
    return [k + 1 for k in b] + [n - k for n, k in zip(shape, b)]


def _shapes(c):
    return [tuple(int(v) for v in s.split("x")) for s in c["shapes"].split()]


def prepare(case, seed):
    c = case
    if c["kind"] == "dsr":
        vol = _frame(c["ny"], c["nx"], c["nz"], seed)
        shape = (c["ny"], c["nx"], c["nz"])
        dims = deskew.deskew_rotate_device(vol, "uint16", shape, c["angle"], c["dz"], c["pixel"], reverse=True,
                                           save16bit=True)
        return {"case": c, "vol": vol, "shape": shape,
                "out": torch.zeros(dims[::-1], dtype=torch.int16, device="cuda")}
    if c["kind"] == "batch":
        shapes = _shapes(c)
        pairs = [_psf_pair("bead", 10 ** 6, 10 ** 6, 10 ** 6, s) for s in (1.3, 1.5, 1.8)]
        vols = [_frame(*s, seed * 1009 + i) for i, s in enumerate(shapes)]
        boxes = [_box(s, c["border"]) for s in shapes]
        outs = [torch.zeros(tuple(b[3 + k] - b[k] + 1 for k in (2, 1, 0)), dtype=torch.float32, device="cuda") for b in boxes]
        chunks = (_lib.Chunk * len(shapes))()
        for i, s in enumerate(shapes):
            chunks[i].in_, chunks[i].out, chunks[i].psf_id = vols[i].data_ptr(), outs[i].data_ptr(), i % len(pairs)
            chunks[i].dims, chunks[i].has_bbox = _lib.i64x3(s), 1
            for k in range(6):
                chunks[i].bbox[k] = boxes[i][k]
        params = _lib.DeconParams()
        _lib.lib.pk_params_default(params)
        params.background, params.save16bit = BACKGROUND, 0
        ptrs = [(ctypes.c_void_p * len(pairs))(*[p[k].ctypes.data for p in pairs]) for k in (0, 1)]
        dims = np.array([p[0].shape for p in pairs], np.int64)
        return {"case": c, "vols": vols, "outs": outs, "chunks": chunks, "params": params, "pairs": pairs, "ptrs": ptrs,
                "dims": dims, "ctx": _lib.default_context()}
    shape = (c["ny"], c["nx"], c["nz"])
    psf, psf_b = _psf_pair(c["psf"], *shape)
    box = _box(shape, c["border"])
    out = torch.zeros(tuple(box[3 + k] - box[k] + 1 for k in (2, 1, 0)), dtype=torch.float32, device="cuda")
    options = {"Background": BACKGROUND, "save16bit": False, "EdgeErosion": c["erosion"]}
    if c["border"]:
        options["bbox"] = box
    return {"case": c, "vol": _volume(c, seed), "shape": shape, "psf": psf, "psf_b": psf_b, "out": out, "options": options}


def run(state):
    c, s = state["case"], state
    if c["kind"] == "dsr":
        deskew.deskew_rotate_device(s["vol"], "uint16", s["shape"], c["angle"], c["dz"], c["pixel"], d_out=s["out"],
                                    reverse=True, save16bit=True)
        return s["out"]
    if c["kind"] == "batch":
        _lib.check(_lib.lib.pk_batch_decon(s["ctx"].handle, 1, len(s["vols"]), s["chunks"], _lib.PK_U16, len(s["pairs"]),
                                           s["ptrs"][0], s["ptrs"][1], s["dims"].ctypes.data, c["iters"], s["params"], 0, 1))
        return s["outs"]
    decon.decon_device(c["method"], s["vol"], c["dtype"], s["shape"], s["psf"],
                       s["psf_b"] if c["method"] == "omw" else None, c["iters"], out=s["out"], **s["options"])
    return s["out"]


# ------------------------------------------------------------------ what a pass cannot do without
def _decon_work(shape, out, iters, method, esize):
    n = math.prod(shape)
    spectrum = 8 * (shape[0] // 2 + 1) * shape[1] * shape[2]
    return {"bytes": n * esize + 4 * out + spectrum * (2 if method == "omw" else 1),
            "flops": iters * 4 * 2.5 * n * math.log2(n)}


def work(case):
    c = case
    if c["kind"] == "dsr":
        shape = (c["ny"], c["nx"], c["nz"])
        out = math.prod(deskew.deskew_rotate_device(None, "uint16", shape, c["angle"], c["dz"], c["pixel"], reverse=True,
                                                    save16bit=True))
        return {"bytes": 2 * math.prod(shape) + 2 * out, "flops": 7 * out}
    if c["kind"] == "batch":
        parts = []
        for s in _shapes(c):
            b = _box(s, c["border"])
            parts.append(_decon_work(s, math.prod(b[3 + k] - b[k] + 1 for k in range(3)), c["iters"], "omw", 2))
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    shape = (c["ny"], c["nx"], c["nz"])
    b = _box(shape, c["border"])
    return _decon_work(shape, math.prod(b[3 + k] - b[k] + 1 for k in range(3)), c["iters"], c["method"],
                       2 if c["dtype"] == "uint16" else 4)


# ------------------------------------------------------------------ the same in 64 bits
def _otf(psf, shape):
    """Half spectrum (real axis y, the last of the tensor) of the normalised PSF at the volume's size."""
    p = psf.astype(np.float64)
    p = torch.from_numpy(np.ascontiguousarray((p / p.sum()).astype(np.float32).astype(np.float64).transpose(2, 1, 0))).cuda()
    big = torch.zeros(shape[::-1], dtype=torch.float64, device="cuda")
    big[tuple(slice(0, k) for k in p.shape)] = p
    return torch.fft.rfftn(torch.roll(big, [-(k // 2) for k in p.shape], (0, 1, 2)))


def _conv(x, H):
    return torch.fft.irfftn(torch.fft.rfftn(x).mul_(H), s=x.shape)


def _decon64(I, psf, psf_b, method, iters):
    shape = tuple(I.shape)[::-1]
    H = _otf(psf, shape)
    if method == "omw":
        B, J = _otf(psf_b, shape), I
        for _ in range(iters):
            J = (_conv(I / _conv(J, H).clamp_(min=EPS), B) * J).clamp_(min=0)
        return J
    J2, J3, J4, Y, lam = I, torch.zeros_like(I), None, None, 0.0
    for k in range(1, iters + 1):
        if k > 2:
            lam = min(max(float(((J2 - Y) * J4).sum()) / (float((J4 * J4).sum()) + EPS), 0.0), 1.0)
        if k >= 2:
            J4 = J2 - Y
        Y = (J2 + lam * (J2 - J3)).clamp_(min=0)
        J3 = J2
        J2 = (Y * _conv(I / _conv(Y, H).clamp_(min=EPS), H.conj())).clamp_(min=0)
    return J2


def _disk(radius):
    """Offsets of MATLAB's strel('disk', radius) for radius >= 3: four periodic lines, widened by two short ones."""
    k = 2.0 * radius / (1 / math.tan(math.pi / 8) + 1 / math.sin(math.pi / 8))
    pts = {(0, 0)}
    for v in ((1, 0), (1, 1), (0, 1), (-1, 1)):
        m = int(k / math.hypot(*v))
        pts = {(a + i * v[0], b + i * v[1]) for a, b in pts for i in range(-m, m + 1)}
    h = radius - max(a for a, _ in pts) - 1
    if h >= 1:
        pts = {(a + i, b + j) for a, b in pts for i in range(-h, h + 1) for j in range(-h, h + 1)}
    return pts


def _shift_and(m, offsets, axes):
    """Binary erosion: the and of m shifted by each offset; what lies outside counts as set."""
    r = max(abs(v) for o in offsets for v in o)
    pad = [0] * 6
    for a in axes:
        pad[2 * (2 - a)] = pad[2 * (2 - a) + 1] = r
    big = torch.nn.functional.pad(m, pad, value=True)
    out = m.clone()
    for o in offsets:
        at = [slice(None)] * 3
        for a, v in zip(axes, o):
            at[a] = slice(r + v, r + v + m.shape[a])
        out &= big[tuple(at)]
    return out


def _eroded(mask, e):
    flat = mask.shape[0] == 1
    m = mask.clone()
    d = e if bool(mask.all()) else 1
    for axis in (1, 2) if flat else (0, 1, 2):
        m.narrow(axis, 0, min(d, m.shape[axis])).zero_()
        m.narrow(axis, max(m.shape[axis] - d, 0), min(d, m.shape[axis])).zero_()
    if bool(mask.all()):
        return m
    m = _shift_and(m, sorted(_disk(e - 1)), (2, 1))
    return m if flat else _shift_and(m, [(k,) for k in range(1 - e, e)], (0,))


def _raw64(vol):
    return _u16(vol).to(torch.float64) if vol.dtype == torch.int16 else vol.to(torch.float64)


def _crop(J, box):
    return J[box[2] - 1:box[5], box[1] - 1:box[4], box[0] - 1:box[3]]


def exact(case, seed):
    c = case
    if c["kind"] == "dsr":
        return None
    if c["kind"] == "batch":
        pairs = [_psf_pair("bead", 10 ** 6, 10 ** 6, 10 ** 6, s) for s in (1.3, 1.5, 1.8)]
        return [_crop(_decon64((_raw64(_frame(*s, seed * 1009 + i)) - BACKGROUND).clamp_(min=0), *pairs[i % 3], "omw",
                               c["iters"]), _box(s, c["border"])) for i, s in enumerate(_shapes(c))]
    shape = (c["ny"], c["nx"], c["nz"])
    raw = _raw64(_volume(c, seed))
    J = _decon64((raw - BACKGROUND).clamp_(min=0), *_psf_pair(c["psf"], *shape), c["method"], c["iters"])
    if c["erosion"]:
        J = J * _eroded(raw != 0, c["erosion"])
    return _crop(J, _box(shape, c["border"]))
