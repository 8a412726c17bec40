"""What a frame leaves in its reference slots when its own output, or another
frame's, goes wrong: a frame whose output cannot be delivered fails alone, and
the frames after it are predicted from it all the same.  The failures are made
on the host (av1g_test_engine_faults); nothing of them reaches the GPU."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from oxideav_av1_b200 import abi, engine, synth  # noqa: E402

pytestmark = pytest.mark.gpu


def _run(eng, st, fr):
    t = st.submit(fr)
    eng.poll(t, 60.0)
    status, planes, _ = st.fetch(t)
    return status, planes


def _same(planes, want, tag):
    for p, (g, e) in enumerate(zip(planes, want)):
        assert np.array_equal(g.astype(np.int64), e), f"{tag} plane {p} differs from the oracle"


# outputs written by the copying kernel, and by the copy engine (more than 512 KiB)
@pytest.mark.parametrize("width,height", [(176, 144), (832, 480)])
def test_frame_without_output_still_refreshes_its_slots(width, height):
    frames = synth.make_stream(seed=221, n_frames=4, width=width, height=height)
    want = oracle.decode_stream(frames)
    assert frames[0].show and frames[1].show and frames[1].refresh
    eng = engine.Engine(device=0)
    try:
        st = eng.open_stream(synth.stream_seq(frames))
        got = [_run(eng, st, frames[0])]
        abi.check(eng.lib.av1g_test_engine_faults(eng.h, 1, 0))
        got += [_run(eng, st, f) for f in frames[1:]]
        st.close()
    finally:
        eng.close()
    assert [s for s, _ in got] == [abi.AV1G_OK, abi.AV1G_EDEVICE, abi.AV1G_OK, abi.AV1G_OK]
    for k in (0, 2, 3):
        _same(got[k][1], want[k], f"frame {k}")


def test_failed_copy_launch_fails_only_the_frames_that_own_a_copy():
    """A copy launch that fails takes the frames whose slots or small outputs it
    was to copy, and none that has no copy in it; a frame whose slots were not
    copied refreshes none."""
    frames = synth.make_stream(seed=222, n_frames=3, width=176, height=144)
    want = oracle.decode_stream(frames)
    hidden = synth.StreamFrame()
    hidden.__dict__.update(frames[1].__dict__)
    hidden.show, hidden.refresh = 0, 0  # decoded, neither shown nor kept: no copy at all
    eng = engine.Engine(device=0)
    try:
        st = eng.open_stream(synth.stream_seq(frames))
        first = _run(eng, st, frames[0])
        abi.check(eng.lib.av1g_test_engine_faults(eng.h, 0, 1))
        nothing = _run(eng, st, hidden)
        abi.check(eng.lib.av1g_test_engine_faults(eng.h, 0, 1))
        lost = _run(eng, st, frames[1])
        again = _run(eng, st, frames[1])  # predicted from the same slots as before
        last = _run(eng, st, frames[2])
        st.close()
    finally:
        eng.close()
    assert [r[0] for r in (first, nothing, lost, again, last)] == [
        abi.AV1G_OK, abi.AV1G_OK, abi.AV1G_EDEVICE, abi.AV1G_OK, abi.AV1G_OK]
    _same(first[1], want[0], "frame 0")
    _same(again[1], want[1], "frame 1")
    _same(last[1], want[2], "frame 2")
