"""Intra reconstruction with an odd number of mode info columns: subsampled
planes are then not a multiple of four samples wide, and their last columns are
read, predicted and written like the others, the row padding after them not at all."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from oxideav_av1_b200 import postfilter, synth  # noqa: E402

pytestmark = pytest.mark.gpu


def _odd(**case):
    """A frame of synth's, one mode info column narrower."""
    f = synth.make_intra_frame(**case)
    f.hdr.mi_cols -= 1
    f.hdr.frame_width = f.hdr.upscaled_width = f.hdr.mi_cols * 4
    f.planes = [np.ascontiguousarray(a[:, : f.plane_dims(p)[1]]) for p, a in enumerate(f.planes)]
    w = np.array([f.plane_dims(p)[1] for p in range(3)])
    f.tus = f.tus[f.tus["x"] < w[f.tus["plane"]]]
    f.tus["max_luma_w"] = np.minimum(f.tus["max_luma_w"], w[0])  # chroma from the luma that there is
    assert f.plane_dims(1)[1] % 4 == (2 if f.hdr.subsampling_x else 0)
    return f


@pytest.mark.parametrize("case", [
    dict(seed=401, width=176, height=144),
    dict(seed=402, width=200, height=120, bit_depth=10, palette=0.2),
    dict(seed=403, width=136, height=96, bit_depth=12, sb_size=128),
    dict(seed=404, width=72, height=64, intrabc=0.3),      # a superblock of one luma group of eight
    dict(seed=405, width=144, height=80, ssx=1, ssy=0),
    dict(seed=406, width=144, height=80, ssx=0, ssy=0),
], ids=lambda c: f"c{c['seed']}")
def test_odd_mode_info_columns(case):
    f = _odd(**case)
    d = postfilter.DeviceIntra(f)
    for pl in d.planes:
        pl.t[:, pl.w * pl.bps:] = 0xA5
    postfilter.run_intra([d])
    torch.cuda.synchronize()
    for p, (g, e) in enumerate(zip(d.download(), oracle.intra(f))):
        diff = np.argwhere(g.astype(np.int64) != e)
        assert len(diff) == 0, f"plane {p}: {len(diff)} samples differ, first {tuple(diff[0])}"
    for p, pl in enumerate(d.planes):
        assert bool((pl.t[:, pl.w * pl.bps:] == 0xA5).all()), f"plane {p}: row padding written"
