"""The post-filter and intra kernels at the edges of their tiles, against the oracle.

Sizes one below, at and one above a tile or a run of tiles, the smallest planes,
every subsampling and bit depth, and batches on both sides of each dispatch rule
(CDEF takes tiles of 16, 32 or 64 rows by the number of blocks in the launch).
Integer path: the tolerance is zero.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from oxideav_av1_b200 import abi, postfilter, synth  # noqa: E402

pytestmark = pytest.mark.gpu


def _run(frames):
    abi.load()
    dev = [postfilter.DeviceFrame(f) for f in frames]
    postfilter.run_postfilter(dev)
    torch.cuda.synchronize()
    return dev


def _same(stage, got, exp):
    for p, (g, e) in enumerate(zip(got, exp)):
        assert g.shape == e.shape
        bad = np.argwhere(g.astype(np.int64) != e)
        assert len(bad) == 0, f"{stage} plane {p}: {len(bad)} samples differ, first at {tuple(bad[0])}"


def _oracle_cdef_lr(f):
    deb = oracle.loop_filter(f, [r.astype(np.int32) for r in f.recon])
    cd = oracle.cdef(f, deb)
    lr = oracle.loop_restoration(f, deb, cd)
    return deb, cd, [lr[p][: f.out_dims(p)[0], : f.out_dims(p)[1]] for p in range(f.hdr.num_planes)]


# widths and heights around the 64-sample tiles, their 8-sample blocks and the smallest frame
FILTER_SIZES = [(8, 8), (16, 72), (57, 65), (64, 64), (72, 136), (127, 63), (129, 130), (200, 33)]
FORMATS = [dict(), dict(bit_depth=10), dict(bit_depth=12), dict(ssx=1, ssy=0), dict(ssx=0, ssy=0),
           dict(ssx=0, ssy=0, bit_depth=10), dict(mono=True)]


@pytest.mark.parametrize("fmt", FORMATS, ids=["-".join(f"{k}{v}" for k, v in f.items()) or "420" for f in FORMATS])
def test_filters_at_tile_edges(fmt):
    """Deblocking, CDEF and loop restoration alone and as one launch over all the sizes."""
    frames = [synth.make_frame(seed=700 + i, width=w, height=h, **fmt) for i, (w, h) in enumerate(FILTER_SIZES)]
    exp = [_oracle_cdef_lr(f) for f in frames]
    for dev in (_run(frames), [_run([f])[0] for f in frames]):
        for d, (deb, cd, lr) in zip(dev, exp):
            _same("deblock", d.download("deblocked"), deb)
            _same("cdef", d.download("cdef"), cd)
            _same("loop restoration", d.download("lr"), lr)


@pytest.mark.parametrize("fmt", [dict(), dict(ssx=0, ssy=0), dict(bit_depth=12)], ids=["420", "444", "12-bit"])
@pytest.mark.parametrize("n", [1, 3, 4, 14])
def test_cdef_tile_heights(fmt, n):
    """48 blocks of 64x64 a frame: batches of 48, 144, 192 and 672 blocks lie on the three
    sides of the lines at 148 and 592."""
    f = synth.make_frame(seed=730, width=512, height=384, **fmt)
    deb, cd, _ = _oracle_cdef_lr(f)
    for d in _run([f] * n):
        _same("cdef", d.download("cdef"), cd)


# (upscaled width, denominator): around the 256, 512 and 1024 wide tiles and their groups of four
SR_CASES = [(16, 16), (33, 9), (255, 16), (257, 9), (511, 12), (514, 13), (1023, 16), (1030, 10)]


@pytest.mark.parametrize("fmt", [dict(), dict(bit_depth=10, ssx=0, ssy=0), dict(bit_depth=12, ssx=1, ssy=0)],
                         ids=["420", "444-10", "422-12"])
@pytest.mark.parametrize("height", [8, 15, 26])
def test_superres_at_tile_edges(fmt, height):
    """Eight-row tiles with one to eight rows left over, with and without the second source set."""
    frames = [synth.make_frame(seed=750 + i, width=w, height=height, superres_denom=d, cdef=False, deblock=False,
                               lr=bool(i & 1), **fmt) for i, (w, d) in enumerate(SR_CASES)]
    for f, d in zip(frames, _run(frames)):
        exp = oracle.upscale(f, [r.astype(np.int32) for r in f.recon])
        _same("superres", [p.download() for p in d.stage_planes()["up_cdef"]], exp)


GRAIN_FORMATS = [dict(), dict(bit_depth=10), dict(bit_depth=12, ssx=1, ssy=0), dict(ssx=0, ssy=0),
                 dict(bit_depth=10, ssx=0, ssy=0), dict(mono=True)]


@pytest.mark.parametrize("fmt", GRAIN_FORMATS,
                         ids=["-".join(f"{k}{v}" for k, v in f.items()) or "420" for f in GRAIN_FORMATS])
@pytest.mark.parametrize("lag", [0, 1, 2, 3])
def test_film_grain_at_tile_edges(fmt, lag):
    """Every lag of the auto-regressive filter; 256-column, 32-row tiles with every remainder of
    a thread's eight columns that matters; scaling from luma, no luma grain, no overlap."""
    frames = []
    for i, (w, h) in enumerate([(8, 8), (31, 33), (66, 64), (255, 31), (257, 65), (264, 97), (301, 40)]):
        f = synth.make_frame(seed=770 + i, width=w, height=h, film_grain=True, deblock=False, cdef=False, lr=False, **fmt)
        g = f.hdr.film_grain
        g.ar_coeff_lag = lag
        g.overlap_flag = i != 1
        if i == 2:
            g.num_y_points = 0
        if i == 3 and not fmt.get("mono"):
            g.chroma_scaling_from_luma, g.num_cb_points, g.num_cr_points = 1, 0, 0
        if i == 4:
            g.num_cb_points = 0
        frames.append(f)
    for f, d in zip(frames, _run(frames)):
        exp = oracle.film_grain(f, [f.recon[p][: f.out_dims(p)[0], : f.out_dims(p)[1]].astype(np.int32)
                                    for p in range(f.hdr.num_planes)])
        _same("film grain", d.download("out"), exp)


@pytest.mark.parametrize("off", [1, 2, 3])
def test_deblock_grid_at_any_address(off):
    """The block grid's arrays may start at any address of their type's alignment."""
    f = synth.make_frame(seed=790, width=136, height=72)
    d = postfilter.DeviceFrame(f)
    for name, t in d.grid.items():
        assert t.element_size() == 1
        buf = torch.empty(t.numel() + off, dtype=torch.uint8, device=t.device)
        buf[off:].copy_(t.reshape(-1).view(torch.uint8))
        d.grid[name] = buf[off:]
    postfilter.run_postfilter([d])
    torch.cuda.synchronize()
    _same("deblock", d.download("deblocked"), oracle.loop_filter(f, [r.astype(np.int32) for r in f.recon]))


INTRA = [
    # frame edges off every TU size; all formats and depths, with the tools that take the general path
    dict(width=8, height=8), dict(width=72, height=40, ssx=0, ssy=0, bit_depth=10), dict(width=136, height=88, ssx=1, ssy=0),
    dict(width=200, height=136, bit_depth=12, sb_size=128, ssx=0, ssy=0), dict(width=104, height=200, mono=True, split=0.1),
    # large TUs alone, then thousands of small ones per superblock
    dict(width=264, height=136, split=0.0), dict(width=264, height=136, bit_depth=10, split=0.05, sb_size=128),
    dict(width=136, height=136, bit_depth=10, split=0.99), dict(width=192, height=128, edge_filter=False, split=0.9),
    dict(width=128, height=128, sb_size=128, ssx=0, ssy=0, split=0.99, palette=0.5),
]


@pytest.mark.parametrize("case", INTRA, ids=["-".join(f"{k}{v}" for k, v in c.items()) for c in INTRA])
def test_intra_paths(case):
    abi.load()
    f = synth.make_intra_frame(seed=801, **case)
    d = postfilter.DeviceIntra(f)
    postfilter.run_intra([d])
    torch.cuda.synchronize()
    _same("intra", d.download(), oracle.intra(f))
