"""Outputs and reference payloads through the engine's plane copies, against the oracle.

Rows that are and are not a multiple of 16 bytes, planes smaller than one copy
unit, steps of more planes than one launch takes, and frames on both sides of the
512 KiB line above which the copy engine moves the output.  Tolerance zero.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from oxideav_av1_b200 import abi, engine, synth  # noqa: E402

pytestmark = pytest.mark.gpu

SHAPES = [
    dict(width=8, height=8), dict(width=17, height=9), dict(width=177, height=143), dict(width=99, height=35, mono=True),
    dict(width=37, height=21, bit_depth=10), dict(width=130, height=66, ssx=0, ssy=0, bit_depth=12),
    dict(width=161, height=50, ssx=1, ssy=0), dict(width=200, height=120, superres_denom=11, film_grain=True),
    dict(width=720, height=484), dict(width=720, height=488), dict(width=721, height=501),  # 522,720 to 542,472 bytes
]


@pytest.mark.parametrize("copies", [1, 9], ids=["alone", "72-streams"])
def test_engine_outputs(copies):
    shapes = SHAPES if copies == 1 else SHAPES[:8]
    streams = [synth.make_stream(seed=840 + i, n_frames=3, **s) for i, s in enumerate(shapes)]
    exp = [oracle.decode_stream(fr) for fr in streams]
    e = engine.Engine(device=0)
    try:
        handles = [(i, e.open_stream(synth.stream_seq(streams[i]))) for _ in range(copies) for i in range(len(shapes))]
        tickets = [[] for _ in handles]
        for k in range(3):
            for (i, h), t in zip(handles, tickets):
                if k < len(streams[i]):
                    t.append(h.submit(streams[i][k]))
        for (i, h), ts in zip(handles, tickets):
            for k, t in enumerate(ts):
                assert e.poll(t, 60.0) == abi.AV1G_OK
                status, planes, _ = h.fetch(t)
                assert status == abi.AV1G_OK
                if exp[i][k] is None:
                    assert planes is None
                    continue
                for p, (g, x) in enumerate(zip(planes, exp[i][k])):
                    assert np.array_equal(g.astype(np.int64), x), f"{shapes[i]} frame {k} plane {p}"
            h.close()
    finally:
        e.close()
