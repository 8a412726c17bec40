"""The measured workloads of the AV1 reconstruction and post-filter engine.

Each case is one pass through the public entry points, over the range that a
decoding service drives them with:

* ``filters`` — the in-loop filter chain (deblock, CDEF, superres, loop
  restoration, film grain) over a batch of reconstructed frames that are
  already on the GPU: ``postfilter.run_postfilter``;
* ``inter`` — reconstruction of inter frames: motion-compensated prediction,
  the residuals of the inter blocks, then the intra blocks and the intra halves
  of inter-intra blocks: ``postfilter.run_inter`` / ``run_recon`` / ``run_intra``;
* ``key`` — reconstruction of key frames, all intra: ``postfilter.run_intra``;
* ``engine`` — whole streams through the serving engine, host descriptors in,
  host frames out: ``engine.Stream.submit`` / ``Engine.poll`` / ``Stream.fetch``;
* ``decode`` — real bitstreams through the stream decoder, IVF bytes in, host
  frames out: ``decoder.decode``.

The descriptors follow ``synth``'s distributions.  Its generators run at a few
dozen microseconds per block, so a case draws small patches from them and lays
those patches out over the frame; edge availability across patches is set as a
tile walk over the whole frame sets it.  Every sample is an integer, and so is
every output.
"""
import base64
import ctypes as C
import functools
import gzip
import importlib.util
import json
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent


def _package():
    # the package's folder name is not an identifier
    if "oxideav_av1_b200" not in sys.modules:
        pkg = ROOT / "oxideav-av1_b200"
        spec = importlib.util.spec_from_file_location("oxideav_av1_b200", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["oxideav_av1_b200"] = mod
        spec.loader.exec_module(mod)


_package()
from oxideav_av1_b200 import abi, decoder, engine, postfilter, synth  # noqa: E402

PATCH = 384  # patch edge in luma samples: a multiple of both superblock sizes


def _case(name, kind, width, height, frames, bit_depth=8, chroma="420", **more):
    c = dict(name=name, kind=kind, width=width, height=height, frames=frames, bit_depth=bit_depth, chroma=chroma)
    c.update(superres=8, grain=False, sb=64, tiles=0, streams=0)
    c.update(more)
    return c


def listed():
    return [
        # one CIF frame: the smallest call, where launches and host work are all there is
        _case("filters_cif_1", "filters", 352, 288, 1),
        # a lane's batch of mid-size frames with grain, odd extents, full-resolution chroma
        _case("filters_718p_444_grain_12", "filters", 1277, 718, 12, 10, "444", grain=True),
        # the micro-benchmark batch: 64 frames of 1080p
        _case("filters_1080p_64", "filters", 1920, 1080, 64),
        # 4K 10-bit delivery with superres and film grain
        _case("filters_2160p_sr_grain_4", "filters", 3840, 2160, 4, 10, superres=12, grain=True),
        # inter frames: a small stream's single frame, two HD streams, one 4K 10-bit frame
        _case("inter_cif_1", "inter", 352, 288, 1),
        _case("inter_1080p_2", "inter", 1920, 1080, 2),
        _case("inter_2160p_10bit_1", "inter", 3840, 2160, 1, 10, sb=128),
        # key frames: several small streams starting together, one HD frame, one tiled 4K 10-bit frame
        _case("key_360p_8", "key", 640, 360, 8),
        _case("key_1080p_1", "key", 1920, 1080, 1),
        _case("key_2160p_10bit_tiles_1", "key", 3840, 2160, 1, 10, sb=128, tiles=1),
        # four 720p streams served together, key frame then inter frames, frames fetched by the host
        _case("engine_720p_4x4", "engine", 1280, 720, 4, streams=4),
        # conformance bitstreams of 64x64, 96x80 and 128x96 through the registry decoder
        _case("decode_small_9", "decode", 128, 96, 4, streams=9),
    ]


def draw(rng):
    kind = rng.choice(["filters", "filters", "inter", "inter", "key", "key", "engine"])
    most = {"filters": 40e6, "inter": 8.3e6, "key": 6e6, "engine": 2.1e6}[kind]
    height = round(math.exp(rng.uniform(math.log(144), math.log(2160 if kind != "engine" else 720))))
    width = round(height * rng.choice([4 / 3, 16 / 9, 1.0, 21 / 9]) + rng.randrange(-7, 8))
    width, height = max(64, min(3840, width)), max(64, height)
    bit_depth, chroma = rng.choice([8, 8, 8, 10, 10, 12]), rng.choice(["420", "420", "420", "444"])
    sb = rng.choice([64, 128])
    fit = max(1, int(most / (width * height * (2 if chroma == "444" else 1))))
    if kind == "filters":
        return _case("drawn", kind, width, height, rng.randint(1, min(64, fit)), bit_depth, chroma, sb=64,
                     superres=rng.choice([8, 8, rng.randint(9, 16)]), grain=rng.random() < 0.4)
    if kind == "engine":
        return _case("drawn", kind, width, height, rng.randint(2, 4), bit_depth, chroma, sb=sb,
                     streams=rng.randint(1, min(5, max(1, fit))), grain=rng.random() < 0.25)
    n = rng.randint(1, min(8, fit))
    if kind == "inter":
        return _case("drawn", kind, width, height, n, bit_depth, chroma, sb=sb)
    return _case("drawn", kind, width, height, n, bit_depth, chroma, sb=sb, tiles=rng.choice([0, 0, 1]))


def work(case):
    """Bytes of one pass, each input read once and each output written once;
    the arithmetic is all integer."""
    c, s = dict(case), 1 if case["bit_depth"] == 8 else 2
    if c["kind"] == "decode":  # the frames out, and about as many bytes of levels and references in
        area = 64 * 64 + 96 * 80 + c["width"] * c["height"]
        return {"bytes": c["streams"] // 3 * c["frames"] * 1.5 * area * 4, "flops": 0}
    px = c["width"] * c["height"] * (3.0 if c["chroma"] == "444" else 1.5)
    cells = c["width"] * c["height"] / 16.0
    if c["kind"] == "filters":
        # the reconstruction in, the reference payload out, the grained output out, the per-4x4 decode state
        up, outs = px * s, 2 if c["grain"] else 1
        return {"bytes": c["frames"] * (up * 8 / c["superres"] + up * outs + 12 * cells), "flops": 0}
    # levels: about one int32 per sample; descriptors: about 64 bytes per prediction or transform unit
    levels, lists = 4 * px * 0.7, 64 * px / 60
    if c["kind"] == "key":
        return {"bytes": c["frames"] * (px * s + levels + lists), "flops": 0}
    if c["kind"] == "inter":
        return {"bytes": c["frames"] * (2.3 * px * s + levels + 2 * lists), "flops": 0}
    return {"bytes": c["streams"] * c["frames"] * (3 * px * s + levels + 2 * lists + 12 * cells), "flops": 0}


def exact(case, seed):
    return None  # whole numbers throughout: they are compared value for value


# ---- inputs -----------------------------------------------------------------

def _ss(case):
    return (0, 0) if case["chroma"] == "444" else (1, 1)


def _header(base, case):
    """The patch's header with the frame's own sizes."""
    h = abi.FrameHeader()
    C.memmove(C.addressof(h), C.addressof(base), C.sizeof(h))
    up, d = case["width"], case["superres"]
    h.upscaled_width = up
    h.frame_width = (up * 8 + d // 2) // d if d != 8 else up
    h.use_superres = int(d != 8)
    h.frame_height = case["height"]
    h.mi_cols, h.mi_rows = 2 * ((h.frame_width + 7) >> 3), 2 * ((h.frame_height + 7) >> 3)
    return h


def _wrap(a, rows, cols, r0=0, c0=0):
    """rows x cols of the array repeated in both directions, from (r0, c0)."""
    return np.ascontiguousarray(a[(np.arange(rows) + r0) % a.shape[0]][:, (np.arange(cols) + c0) % a.shape[1]])


def _side_data(f, base, shift=(0, 0)):
    """Grids, CDEF indices and restoration units of the frame, from the patch's."""
    h = f.hdr
    r0, c0 = shift[0] * 16, shift[1] * 16
    f.grid = {k: _wrap(a, h.mi_rows, h.mi_cols, r0, c0) for k, a in base.grid.items()}
    f.cdef_idx = _wrap(base.cdef_idx, (h.mi_rows + 15) >> 4, (h.mi_cols + 15) >> 4, *shift)
    sx, sy = h.subsampling_x, h.subsampling_y
    f.lr_units = [None] * 3
    for p in range(h.num_planes):
        us = h.lr_unit_size[p]
        ph, pw = (h.frame_height, h.upscaled_width) if p == 0 else ((h.frame_height + sy) >> sy,
                                                                     (h.upscaled_width + sx) >> sx)
        f.lr_units[p] = _wrap(base.lr_units[p], max((ph + us // 2) // us, 1), max((pw + us // 2) // us, 1), *shift)


def _samples(gen, n, dims, bit_depth, planes):
    """Device planes as ``synth`` draws them: a 16x16 uniform field upsampled
    bilinearly, plus uniform noise of +-12 (8-bit scale).  One byte tensor
    [n, rows, pitch] per plane, rows 64-byte aligned."""
    out, bps, top = [], 1 if bit_depth == 8 else 2, (1 << bit_depth) - 1
    for p in range(planes):
        rows, cols = dims[p]
        pitch = (cols * bps + 63) // 64 * 64
        t = torch.zeros((n, rows, pitch), dtype=torch.uint8, device="cuda")
        for i in range(n):
            field = torch.rand((1, 1, 16, 16), generator=gen, device="cuda") * top
            v = torch.nn.functional.interpolate(field, size=(rows, cols), mode="bilinear", align_corners=True)[0, 0]
            noise = torch.randint(-12, 13, (rows, cols), generator=gen, device="cuda", dtype=torch.int32)
            v = (v.round().int() + noise * (1 << (bit_depth - 8))).clamp_(0, top)
            v = v.to(torch.uint8) if bps == 1 else v.to(torch.int16).view(torch.uint8)
            t[i, :, : cols * bps] = v
        out.append(t)
    return out


def _blank(n, dims, bit_depth, planes):
    bps = 1 if bit_depth == 8 else 2
    return [torch.zeros((n, dims[p][0], (dims[p][1] * bps + 63) // 64 * 64), dtype=torch.uint8, device="cuda")
            for p in range(planes)]


def _plane(t, dims, hbd):
    """A DevPlane over a slice of a batch tensor."""
    pl = postfilter.DevPlane.__new__(postfilter.DevPlane)
    pl.h, pl.w, pl.hbd, pl.bps, pl.pitch, pl.t = dims[0], dims[1], hbd, 2 if hbd else 1, t.shape[1], t
    return pl


def _dims(h, padded=True):
    res = []
    for p in range(h.num_planes):
        sx, sy = (h.subsampling_x, h.subsampling_y) if p else (0, 0)
        res.append(((h.mi_rows * 4) >> sy, (h.mi_cols * 4) >> sx) if padded
                   else ((h.frame_height + sy) >> sy, (h.upscaled_width + sx) >> sx))
    return res


def _spread(a, h):
    """Copies of the patch's list over the frame, in raster order of patches:
    (entries, each one's patch origin x and y in luma samples, its copy number)."""
    nx, ny = -(-h.mi_cols * 4 // PATCH), -(-h.mi_rows * 4 // PATCH)
    k = np.repeat(np.arange(nx * ny), len(a))
    return np.tile(a, nx * ny), (k % nx) * PATCH, (k // nx) * PATCH, k


def _inside(h, plane, x, y):
    sx, sy = np.where(plane > 0, h.subsampling_x, 0), np.where(plane > 0, h.subsampling_y, 0)
    return (x < ((h.mi_cols * 4) >> sx)) & (y < ((h.mi_rows * 4) >> sy)), sx, sy


def _lay_out_calls(fr, h):
    """The patch's inter calls, neighbours and warps over the frame."""
    a, ox, oy, k = _spread(fr.preds, h)
    sx, sy = np.where(a["plane"] > 0, h.subsampling_x, 0), np.where(a["plane"] > 0, h.subsampling_y, 0)
    a["x"] += (ox >> sx).astype(np.uint16)
    a["y"] += (oy >> sy).astype(np.uint16)
    a["mi_col"] += (ox // 4).astype(np.uint16)
    a["mi_row"] += (oy // 4).astype(np.uint16)
    a["warp"] += np.where(a["warp"] >= 0, k * len(fr.warps), 0).astype(np.int32)
    a["obmc_first"] += (k * len(fr.neighbours)).astype(np.uint32)
    copies = int(k[-1]) + 1
    nb, nox, noy, nk = _spread(fr.neighbours, h)
    # a neighbour's position lies along the edge it was listed for
    left = np.zeros(len(fr.neighbours), bool)
    for d in fr.preds[fr.preds["motion_mode"] == 1]:
        f0 = int(d["obmc_first"]) + int(d["obmc_above"])
        left[f0:f0 + int(d["obmc_left"])] = True
    nb["axis_pos4"] += np.where(np.tile(left, copies), noy // 4, nox // 4).astype(np.uint16)
    ok, _, _ = _inside(h, a["plane"], a["x"], a["y"])
    # an edge block whose OBMC neighbours lie past the frame keeps those inside it
    keep = np.ones(len(a), bool)
    for i in np.nonzero(ok & (a["motion_mode"] == 1))[0]:
        f0, na, nl = int(a["obmc_first"][i]), int(a["obmc_above"][i]), int(a["obmc_left"][i])
        lim_c, lim_r = h.mi_cols, h.mi_rows
        keep[i] = not (np.any(nb["axis_pos4"][f0:f0 + na] >= lim_c) or
                       np.any(nb["axis_pos4"][f0 + na:f0 + na + nl] >= lim_r))
    a["motion_mode"][~keep] = 0
    return a[ok], nb, np.tile(fr.warps, copies)


def _lay_out_tus(tus, ncoeffs, h):
    a, ox, oy, k = _spread(tus, h)
    sx, sy = np.where(a["plane"] > 0, h.subsampling_x, 0), np.where(a["plane"] > 0, h.subsampling_y, 0)
    a["x"] += (ox >> sx).astype(np.uint16)
    a["y"] += (oy >> sy).astype(np.uint16)
    a["coeff_offset"] += (k * ncoeffs).astype(np.uint32)
    ok, _, _ = _inside(h, a["plane"], a["x"], a["y"])
    return a[ok]


def _lay_out_intra(tus, ncoeffs, nmaps, h, sb, tiles, key):
    """The patch's intra TUs over the frame, in decode order (tiles, then
    superblocks in raster order), with the edge availability of a walk over the
    whole frame at patch and superblock boundaries."""
    a, ox, oy, k = _spread(tus, h)
    sx, sy = np.where(a["plane"] > 0, h.subsampling_x, 0), np.where(a["plane"] > 0, h.subsampling_y, 0)
    a["x"] += (ox >> sx).astype(np.uint16)
    a["y"] += (oy >> sy).astype(np.uint16)
    a["res"]["x"], a["res"]["y"] = a["x"], a["y"]
    a["res"]["coeff_offset"] += (k * ncoeffs).astype(np.uint32)
    a["palette_map"] += (k * nmaps * (a["mode"] == abi.INTRA_MODE_PALETTE)).astype(np.uint32)
    cfl = (a["flags"] & abi.INTRA_CFL) > 0
    # MaxLumaW / MaxLumaH stop at the luma that the frame has
    a["max_luma_w"] = np.where(cfl, np.minimum(a["max_luma_w"] + ox, h.mi_cols * 4), a["max_luma_w"])
    a["max_luma_h"] = np.where(cfl, np.minimum(a["max_luma_h"] + oy, h.mi_rows * 4), a["max_luma_h"])
    ok, sx, sy = _inside(h, a["plane"], a["x"], a["y"])
    a, sx, sy = a[ok], sx[ok], sy[ok]
    sbx, sby = (a["x"].astype(int) << sx) // sb, (a["y"].astype(int) << sy) // sb
    tc, tr = synth.tile_grid(h.mi_rows, h.mi_cols, sb, tiles, tiles)
    cols, rows = np.array([e[0] // sb for e in tc]), np.array([e[0] // sb for e in tr])
    tcol, trow = np.searchsorted(cols, sbx, "right") - 1, np.searchsorted(rows, sby, "right") - 1
    if key:
        x, y = a["x"].astype(int), a["y"].astype(int)
        w, hh = np.array(synth.TX_W)[a["tx_size"]], np.array(synth.TX_H)[a["tx_size"]]
        x0, y0 = (cols[tcol] * sb) >> sx, (rows[trow] * sb) >> sy
        x1 = np.minimum(np.append(cols, 1 << 20)[tcol + 1] * sb, h.mi_cols * 4) >> sx
        y1 = np.minimum(np.append(rows, 1 << 20)[trow + 1] * sb, h.mi_rows * 4) >> sy
        top, left = (y % (sb >> sy)) == 0, (x % (sb >> sx)) == 0
        keep = ~np.uint8(abi.INTRA_HAVE_ABOVE | abi.INTRA_HAVE_LEFT)
        f = a["flags"] & keep
        f |= np.where(y > y0, abi.INTRA_HAVE_ABOVE, 0).astype(np.uint8)
        f |= np.where(x > x0, abi.INTRA_HAVE_LEFT, 0).astype(np.uint8)
        # the superblock row above is decoded; so is the superblock to the left
        ar = np.where(top, (y > y0) & (x + w < x1), ((f & abi.INTRA_HAVE_ABOVE_RIGHT) > 0) & (x + w < x1))
        bl = np.where(left, (x > x0) & (y + hh < y1) & ((y + hh) % (sb >> sy) != 0),
                      ((f & abi.INTRA_HAVE_BELOW_LEFT) > 0) & (y + hh < y1))
        f &= ~np.uint8(abi.INTRA_HAVE_ABOVE_RIGHT | abi.INTRA_HAVE_BELOW_LEFT)
        f |= np.where(ar, abi.INTRA_HAVE_ABOVE_RIGHT, 0).astype(np.uint8)
        f |= np.where(bl, abi.INTRA_HAVE_BELOW_LEFT, 0).astype(np.uint8)
        a["flags"] = f
    order = np.lexsort((np.arange(len(a)), sbx, sby, tcol, trow))
    return np.ascontiguousarray(a[order])


def _stream_frames(case, seed, n):
    """n frames of one stream (a key frame, then inter frames) as
    ``synth.StreamFrame`` descriptors over the whole frame."""
    ssx, ssy = _ss(case)
    m = min(n, 2)  # one patch of each kind, its copies shifted from frame to frame
    base = synth.make_stream(seed % 100003 + 1, m, PATCH, PATCH, case["bit_depth"], ssx, ssy, film_grain=case["grain"],
                             sb_size=case["sb"])
    rng = np.random.default_rng(seed)
    out = []
    for i in range(n):
        b = base[min(i, m - 1)]
        fr = synth.StreamFrame()
        fr.__dict__.update(b.__dict__)
        fr.hdr = _header(b.hdr, case)
        _side_data(fr, b)
        copies = (-(-fr.hdr.mi_cols * 4 // PATCH)) * (-(-fr.hdr.mi_rows * 4 // PATCH))
        nm = 0 if b.palette_maps is None else len(b.palette_maps)
        if b.preds is not None:
            fr.preds, fr.neighbours, fr.warps = _lay_out_calls(b, fr.hdr)
            fr.preds["mv"] += rng.integers(-24, 25, (2, 2)).astype(np.int16)  # another motion each frame
        if b.inter_tus is not None:
            fr.inter_tus = _lay_out_tus(b.inter_tus, len(b.coeffs), fr.hdr)
        fr.intra_tus = _lay_out_intra(b.intra_tus, len(b.coeffs), nm, fr.hdr, case["sb"], case["tiles"], i == 0)
        fr.coeffs = np.tile(b.coeffs, copies)
        fr.palette_maps = np.tile(b.palette_maps, copies) if nm else np.zeros(0, np.uint8)
        fr.refresh = 0xFF if i == 0 else b.refresh
        out.append(fr)
    return out


# ---- states -----------------------------------------------------------------

class Filters:
    def __init__(self, case, seed):
        ssx, ssy = _ss(case)
        n = case["frames"]
        gen = torch.Generator("cuda").manual_seed(seed)
        bases = [synth.make_frame(seed % 100003 * 8 + k, PATCH, PATCH, case["bit_depth"], ssx, ssy,
                                  film_grain=case["grain"]) for k in range(min(n, 6))]
        self.frames = []
        for i in range(n):
            b = bases[i % len(bases)]
            f = synth.SyntheticFrame()
            f.hdr = _header(b.hdr, case)
            f.hdr.film_grain.grain_seed = (b.hdr.film_grain.grain_seed + 977 * i) & 0xFFFF
            _side_data(f, b, (i // len(bases), i // len(bases) * 2))
            f.recon = [None] * 3
            self.frames.append(postfilter.DeviceFrame(f))
        h = self.frames[0].hdr
        sr = h.use_superres and h.upscaled_width > h.frame_width
        pad, out = _dims(h), _dims(h, False)
        src = _samples(gen, n, pad, h.bit_depth, h.num_planes)
        self.lr = _blank(n, out if sr else pad, h.bit_depth, h.num_planes)
        self.out = _blank(n, out, h.bit_depth, h.num_planes) if case["grain"] else []
        hbd = h.bit_depth > 8
        for i, f in enumerate(self.frames):
            for p in range(h.num_planes):
                f.recon[p] = _plane(src[p][i], pad[p], hbd)
                f.lr[p] = _plane(self.lr[p][i], (out if sr else pad)[p], hbd)
                if self.out:
                    f.out[p] = _plane(self.out[p][i], out[p], hbd)
        self.jobs = postfilter.jobs_array(self.frames)

    def run(self):
        postfilter.run_postfilter(self.frames, jobs=self.jobs)
        return self.lr + self.out


class _Recon(postfilter.DeviceRecon):
    def __init__(self, fr, planes, coeffs):
        self.frame, self.planes, self.coeffs, self.tus = fr, planes, coeffs, fr.inter_tus


class _Intra(postfilter.DeviceIntra):
    def __init__(self, fr, planes, coeffs, side):
        self.frame, self.planes, self.coeffs, self.tus, self.side = fr, planes, coeffs, fr.intra_tus, side


class _Inter(postfilter.DeviceInter):
    def __init__(self, fr, planes, side, refs, ref_dims):
        self.frame, self.planes, self.side = fr, planes, side
        self.preds, self.neighbours, self.warps = fr.preds, fr.neighbours, fr.warps
        self.refs = (abi.RefFrame * 7)()
        for r in range(7):
            self.refs[r].upscaled_width, self.refs[r].frame_height = fr.hdr.upscaled_width, fr.hdr.frame_height
            for p in range(fr.hdr.num_planes):
                self.refs[r].planes[p] = _plane(refs[p][r], ref_dims[p], fr.hdr.bit_depth > 8).cplane()


class Recon:
    """Key or inter frames, one of each of ``frames`` streams, in one batch."""

    def __init__(self, case, seed, key):
        gen = torch.Generator("cuda").manual_seed(seed)
        n, distinct = case["frames"], min(case["frames"], 2)
        self.key, self.inter, self.recon, self.intra = key, [], [], []
        descs = [_stream_frames(case, seed * 7 + k, 1 if key else 2)[-1] for k in range(distinct)]
        for d in descs:
            d.sb_size = case["sb"]
        h = descs[0].hdr
        pad, out, hbd, np_ = _dims(h), _dims(h, False), h.bit_depth > 8, h.num_planes
        self.planes = _blank(n, pad, h.bit_depth, np_)
        self.side = [] if key else _blank(n, pad, h.bit_depth, np_)
        self.refs = [] if key else [_samples(gen, 7, out, h.bit_depth, np_) for _ in range(n)]
        for i in range(n):
            d = descs[i % distinct]
            coeffs = torch.from_numpy(d.coeffs).cuda()
            if i >= distinct:  # another stream's levels
                coeffs = -coeffs
            planes = [_plane(self.planes[p][i], pad[p], hbd) for p in range(np_)]
            side = None if key else [_plane(self.side[p][i], pad[p], hbd) for p in range(np_)]
            if not key:
                self.inter.append(_Inter(d, planes, side, self.refs[i], out))
                self.recon.append(_Recon(d, planes, coeffs))
            self.intra.append(_Intra(d, planes, coeffs, side))

    def run(self):
        if not self.key:
            for t in self.planes:  # CurrFrame starts at zero
                t.zero_()
            postfilter.run_inter(self.inter)
            postfilter.run_recon(self.recon)
        postfilter.run_intra(self.intra)
        return self.planes


@functools.lru_cache(None)
def _engine():
    return engine.Engine(device=0)  # a serving process keeps one


class Serving:
    def __init__(self, case, seed):
        self.eng = _engine()
        self.frames = [_stream_frames(case, seed * 11 + k, case["frames"]) for k in range(case["streams"])]
        self.streams = [self.eng.open_stream(synth.stream_seq(f, case["sb"])) for f in self.frames]

    def run(self):
        tickets = [(st, st.submit(fr)) for t in range(len(self.frames[0]))
                   for st, fr in ((s, f[t]) for s, f in zip(self.streams, self.frames))]
        out = []
        for st, t in tickets:
            if self.eng.poll(t, 60.0) != abi.AV1G_OK:
                raise RuntimeError("a frame failed")
            out.append(st.fetch(t)[1])
        return out

    def __del__(self):
        for s in self.streams:
            s.close()


@functools.lru_cache(None)
def _bitstreams(width, height, frames):
    """The conformance streams of that size and frame count, 8-bit 4:2:0."""
    every = json.load(gzip.open(ROOT / "tests" / "golden" / "framing_fixtures.json.gz"))["ivf_streams"]
    pool = [base64.b64decode(s["ivf"]) for s in every if s["shown_frames"] == frames]
    size = width.to_bytes(2, "little") + height.to_bytes(2, "little")
    pool = [d for d in pool if d[12:16] == size]
    heads = [decoder.parse_stream(d)[1][0].hdr for d in pool]
    return [d for d, h in zip(pool, heads) if h.bit_depth == 8 and h.num_planes == 3 and h.subsampling_x == 1
            and h.subsampling_y == 1 and h.upscaled_width == width and h.frame_height == height]


class Decode:
    def __init__(self, case, seed):
        self.eng = _engine()
        rng = np.random.default_rng(seed)
        self.data = []
        for w, h in ((64, 64), (96, 80), (case["width"], case["height"])):
            pool = _bitstreams(w, h, case["frames"])
            self.data += [pool[k] for k in rng.permutation(len(pool))[: case["streams"] // 3]]

    def run(self):
        return [np.frombuffer(b"".join(f.tobytes() for f in decoder.decode(d, self.eng)), np.uint8) for d in self.data]


def prepare(case, seed):
    torch.cuda.set_device(0)
    kind = case["kind"]
    if kind == "filters":
        return Filters(case, seed)
    if kind in ("key", "inter"):
        return Recon(case, seed, kind == "key")
    return Serving(case, seed) if kind == "engine" else Decode(case, seed)


def run(state):
    return state.run()
