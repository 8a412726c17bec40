"""The helper threads that share a call's host preparation: several callers at
once, a forked child, exceptions, and which of two bad descriptors in different
parts is reported.  Plans are only made, and bad calls refused on the host."""
import ctypes as C
import shutil
import subprocess
import sys
import threading
from pathlib import Path

import numpy as np
import pytest

from oxideav_av1_b200 import abi, synth

ROOT = Path(__file__).resolve().parent.parent


def _planes(job, f, field="planes"):
    for p in range(f.hdr.num_planes):
        h, w = f.plane_dims(p)
        pitch = (w * (2 if f.hdr.bit_depth > 8 else 1) + 63) // 64 * 64
        getattr(job, field)[p] = abi.Plane(1 << 20, pitch, w, h)  # an aligned address that nothing reads


def _intra_job(f, tus):
    j = abi.IntraJob()
    j.hdr, j.quant = C.pointer(f.hdr), C.pointer(f.quant)
    j.tus, j.num_tus, j.sb_size, j.coeffs = tus.ctypes.data, len(tus), f.sb_size, 1 << 20
    _planes(j, f)
    return j


def _stats(job):
    st = abi.IntraPlanStats()
    abi.check(abi.load().av1g_intra_plan_stats_get(C.byref(job), 1, C.byref(st)))
    return tuple(getattr(st, n) for n, _ in st._fields_)


@pytest.fixture(scope="module")
def frames():
    """Enough TUs for several parts each (at least 2,048 a part)."""
    fs = [synth.make_intra_frame(seed=601, width=640, height=480, split=0.9),
          synth.make_intra_frame(seed=602, width=512, height=448, split=0.9, bit_depth=10, sb_size=128)]
    assert all(len(f.tus) > 3 * 2048 for f in fs)
    return fs


@pytest.mark.gpu  # the call takes its status words before it makes the plan
def test_intra_reports_the_first_bad_tu_of_several_parts(frames):
    lib, f = abi.load(), frames[0]
    n = len(f.tus)
    for bad in ([n // 2, n - 5], [3, n // 3, n - 1], [n - 1]):
        tus = f.tus.copy()
        tus["tx_size"][bad] = 19
        jobs = (abi.IntraJob * 1)(_intra_job(f, tus))
        for _ in range(5):
            assert lib.av1g_run_intra(jobs, 1, None) == abi.AV1G_EINVAL
            assert f"job 0: TU {bad[0]} " in lib.av1g_last_error().decode()


def test_inter_reports_the_first_bad_call_of_several_parts():
    lib = abi.load()
    f = synth.make_inter_frame(seed=603, width=176, height=144)
    preds = np.resize(f.preds, 8000)  # parts of at least 1,024
    j = abi.InterJob()
    refs = (abi.RefFrame * 7)()
    for r, ref in enumerate(f.refs):
        refs[r].upscaled_width, refs[r].frame_height = ref["upscaled_width"], ref["frame_height"]
        for p in range(f.hdr.num_planes):
            refs[r].planes[p] = abi.Plane(1 << 20, 1 << 14, 1 << 12, 1 << 12)
    j.hdr, j.refs = C.pointer(f.hdr), refs
    j.num_preds, j.num_neighbours, j.num_warps = len(preds), len(f.neighbours), len(f.warps)
    j.neighbours = f.neighbours.ctypes.data if len(f.neighbours) else None
    j.warps = f.warps.ctypes.data if len(f.warps) else None
    _planes(j, f)
    for bad in ([2500, 7000], [7999]):
        some = preds.copy()
        some["kind"][bad] = 3
        j.preds = some.ctypes.data
        for _ in range(5):
            assert lib.av1g_run_inter(C.byref(j), 1, None) == abi.AV1G_EINVAL
            assert f"job 0: call {bad[0]}: kind" in lib.av1g_last_error().decode()


def test_callers_on_several_threads_share_the_helpers(frames):
    jobs = [_intra_job(f, f.tus) for f in frames]
    alone = [_stats(j) for j in jobs]
    wrong = []

    def caller(k):
        for i in range(8):
            if _stats(jobs[(k + i) % 2]) != alone[(k + i) % 2]:
                wrong.append(k)

    ts = [threading.Thread(target=caller, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong


def test_forked_child_prepares_on_its_own_thread():
    """The helpers do not survive a fork: the child's calls do without them."""
    code = """
import os, sys
sys.path[:0] = [%r, %r]
import conftest, test_host_pool as t
from oxideav_av1_b200 import synth
f = synth.make_intra_frame(seed=604, width=640, height=480, split=0.9)
job = t._intra_job(f, f.tus)
want = t._stats(job)  # the helpers run from here on
pid = os.fork()
if pid == 0:
    os._exit(0 if t._stats(job) == want else 1)
sys.exit(os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]))
""" % (str(ROOT / "tests"), str(ROOT))
    assert subprocess.run([sys.executable, "-c", code], timeout=300).returncode == 0


@pytest.mark.skipif(not shutil.which("g++"), reason="no g++")
def test_exceptions_reach_the_caller_and_only_it(tmp_path):
    """Callers on several threads, some of whose parts throw: every part runs
    once, the throwing callers get an exception, the others none."""
    src = tmp_path / "main.cpp"
    src.write_text("""
#include <atomic>
#include <stdexcept>
#include <thread>
#include <vector>
#include "host_pool.h"
int main() {
    std::atomic<int> wrong{0};
    std::vector<std::thread> ts;
    for (int c = 0; c < 6; c++)
        ts.emplace_back([&, c] {
            for (int round = 0; round < 300; round++) {
                std::vector<std::atomic<int>> seen(17);
                bool caught = false;
                const bool throws = (c + round) % 3 == 0;
                try {
                    av1g::parallel_for(17, 1 << 20, [&](int i) {
                        seen[i]++;
                        if (throws && i % 5 == 1) throw std::runtime_error("part");
                    });
                } catch (const std::runtime_error&) {
                    caught = true;
                }
                for (auto& s : seen) wrong += s != 1;
                wrong += caught != throws;
            }
        });
    for (auto& t : ts) t.join();
    return wrong ? 1 : 0;
}
""")
    csrc = ROOT / "oxideav-av1_b200" / "csrc"
    exe = tmp_path / "pool"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{csrc}", str(src), str(csrc / "host_pool.cpp"), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=120).returncode == 0
