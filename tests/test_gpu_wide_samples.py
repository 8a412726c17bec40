"""Deblocking, loop restoration and superres of 16-bit planes whose samples have
more bits than the frame's depth: the filters' arithmetic is defined for them all
the same, tile by tile.  Against the oracle, no tolerance."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from oxideav_av1_b200 import postfilter, synth  # noqa: E402

pytestmark = pytest.mark.gpu

FORMATS = [dict(bit_depth=10), dict(bit_depth=10, ssx=0, ssy=0), dict(bit_depth=12)]
IDS = ["10", "10-444", "12"]


def _raise(f, seed, most):
    """Lifts a few areas of each plane, their shape kept, and single samples, to values up to `most`."""
    rng = np.random.default_rng(seed)
    for p, a in enumerate(f.recon):
        v = a.astype(np.int64)
        h, w = v.shape
        for k in range(3):
            y, x = int(rng.integers(0, h)), int(rng.integers(0, w))
            v[y:y + 24, x:x + 40] += int(rng.integers(1, most - int(v.max())))
        v = np.minimum(v, most)
        v[int(rng.integers(0, h)), int(rng.integers(0, w))] = most
        f.recon[p] = v.astype(np.uint16)


def _run(f):
    d = postfilter.DeviceFrame(f)
    postfilter.run_postfilter([d])
    torch.cuda.synchronize()
    return d


def _same(got, exp):
    for p, (g, e) in enumerate(zip(got, exp)):
        bad = np.argwhere(g.astype(np.int64) != e)
        assert len(bad) == 0, f"plane {p}: {len(bad)} samples differ, first at {tuple(bad[0])}"


@pytest.mark.parametrize("fmt", FORMATS, ids=IDS)
@pytest.mark.parametrize("most", [1024 + 200, 65535])
def test_deblock(fmt, most):
    f = synth.make_frame(seed=901, width=328, height=200, cdef=False, lr=False, **fmt)
    f.hdr.lf_level[2], f.hdr.lf_level[3] = 40, 50
    if most > 1 << fmt["bit_depth"]:
        _raise(f, 7, most)
    _same(_run(f).download("deblocked"), oracle.loop_filter(f, [r.astype(np.int32) for r in f.recon]))


# at 10 bits up to 12: beyond, the box sums' products pass 32 bits
@pytest.mark.parametrize("fmt", FORMATS[:2], ids=IDS[:2])
@pytest.mark.parametrize("unit", [1, 2])
def test_loop_restoration(fmt, unit):
    f = synth.make_frame(seed=902, width=328, height=200, deblock=False, cdef=False, lr_types=(unit,) * 3, **fmt)
    for u in f.lr_units:
        u["type"] = unit
    _raise(f, 8, 4095)
    src = [r.astype(np.int32) for r in f.recon]
    exp = oracle.loop_restoration(f, src, src)
    _same(_run(f).download("lr"), [e[: f.out_dims(p)[0], : f.out_dims(p)[1]] for p, e in enumerate(exp)])


@pytest.mark.parametrize("fmt", FORMATS, ids=IDS)
def test_superres(fmt):
    f = synth.make_frame(seed=903, width=600, height=60, superres_denom=13, deblock=False, cdef=False, lr=False, **fmt)
    _raise(f, 9, 65535)
    exp = oracle.upscale(f, [r.astype(np.int32) for r in f.recon])
    _same([p.download() for p in _run(f).stage_planes()["up_cdef"]], exp)
