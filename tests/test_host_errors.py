"""Which of several bad descriptors a call reports: the first in call order,
whatever runs of the lists the host checks on several threads.  All of it is
refused on the host, before any device work."""
import ctypes as C

import numpy as np
import pytest

from oxideav_av1_b200 import abi, synth


def _planes(job, f, field="planes"):
    for p in range(f.hdr.num_planes):
        h, w = f.plane_dims(p)
        pitch = (w * (2 if f.hdr.bit_depth > 8 else 1) + 63) // 64 * 64
        getattr(job, field)[p] = abi.Plane(1 << 20, pitch, w, h)  # an aligned address that nothing reads


def _recon_job(f, tus):
    j = abi.ReconJob()
    j.hdr, j.quant = C.pointer(f.hdr), C.pointer(f.quant)
    j.tus, j.num_tus, j.coeffs = tus.ctypes.data, len(tus), 1 << 20
    _planes(j, f)
    return j


def _refused(rc):
    assert rc == abi.AV1G_EINVAL
    return abi.load().av1g_last_error().decode()


def test_recon_reports_the_first_problem_in_call_order():
    lib = abi.load()
    f = synth.make_recon_frame(seed=501, width=176, height=144)
    good = np.resize(f.tus, 20000)  # enough for several runs
    bad = good.copy()
    bad["tx_size"][[15000, 19000]] = 19
    wrong = synth.make_recon_frame(seed=502, width=176, height=144)
    wrong.hdr.bit_depth = 9
    jobs = (abi.ReconJob * 3)(_recon_job(f, good), _recon_job(f, bad), _recon_job(wrong, good))
    assert "job 1: TU 15000 " in _refused(lib.av1g_run_recon(jobs, 3, None))
    jobs = (abi.ReconJob * 2)(_recon_job(wrong, good), _recon_job(f, bad))
    assert "job 0" in _refused(lib.av1g_run_recon(jobs, 2, None))
