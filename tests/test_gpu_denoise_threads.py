"""One session denoised from several threads."""

import ctypes
import threading

import pytest

from sundog_b200 import abi, workloads
from sundog_b200 import scene as sc

pytestmark = pytest.mark.gpu


def device_bytes(ses):
    st = abi.SessionStats()
    abi.check(ses.lib.sundog_session_info(ses.handle, ctypes.byref(st)), "info", ses.lib)
    return st.device_bytes


def test_threads_denoise_one_session(lib):
    """The session keeps one set of buffers: no call may free or overwrite
    what another works in, the first calls (which make them) least of all. The
    filter is deterministic, so every result is the same byte for byte."""
    s = workloads.cornell(width=333, height=217, spp=4)
    with sc.Session(s, aov=True) as alone:
        alone.render()
        want = alone.denoise().tobytes()
    with sc.Session(s, aov=True) as ses:
        ses.render()
        held = device_bytes(ses)
        got = []

        def work():
            for _ in range(8):
                got.append(ses.denoise().tobytes())
        threads = [threading.Thread(target=work) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert len(got) == 32 and all(g == want for g in got)
        assert device_bytes(ses) - held == 3 * 16 * 333 * 217
