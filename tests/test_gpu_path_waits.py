"""The waits between the blocks of a path-sample launch: paths that hold the
tiles behind them up for many times the limit change nothing while they are
worked on, and a wait that does run out (for tiles that nobody takes) fails
the whole launch and leaves the device usable."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    src = os.path.join(ROOT, "tests", "cuda", "path_wait_check.cu")
    lib = str(tmp_path_factory.mktemp("path_wait") / "libpathwait.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-gencode=arch=compute_103a,code=sm_103a", "-O3", "--fmad=false",
                    "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off", "-shared",
                    "-I" + os.path.join(ROOT, "openpgl_gb300", "csrc"), src, "-o", lib], check=True)
    dll = ctypes.CDLL(lib)

    def run(lengths, limit, left_out=0):
        from openpgl_gb300 import synthetic as syn

        begin = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32)
        segs, _ = syn.path_segments(int(begin[-1]) // 2 + 64, 61)
        segs = np.ascontiguousarray(segs[:begin[-1]])
        out = np.zeros(len(segs) * 40, np.uint8)
        off = np.zeros(len(begin), np.uint32)
        rc = dll.path_wait_check(segs.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(len(segs)),
                                 begin.ctypes.data_as(ctypes.c_void_p), len(begin) - 1, ctypes.c_float(30.0),
                                 ctypes.c_uint32(limit), left_out, out.ctypes.data_as(ctypes.c_void_p),
                                 off.ctypes.data_as(ctypes.c_void_p))
        assert rc == 0
        return segs, begin, out, off

    return run


# eight paths of 4,000 segments in the first tile take some hundred milliseconds, 8,192 looks
# in vain some five; a sign of work comes twice a millisecond
def test_long_paths_hold_the_others_up(check):
    import openpgl_gb300 as pgl

    lengths = np.concatenate([[4000] * 8, np.full(4000, 6)])
    segs, begin, out, off = check(lengths, 8192)
    st = pgl.PathSegmentStorage(reserve=4000)
    st.set_max_distance(30.0)
    want, counts = [], [0]
    for b, e in zip(begin[:-1], begin[1:]):
        st.clear()
        st.add_segments(segs[int(b):int(e)])
        st.prepare_samples(False, True, True)
        want.append(np.asarray(st.samples()).tobytes())
        counts.append(len(want[-1]) // 40)
    assert np.array_equal(off, np.cumsum(counts))
    want = b"".join(want)
    assert out[:len(want)].tobytes() == want


@pytest.mark.parametrize("paths,left_out", [(4000, 1), (60000, 3)])
def test_a_wait_that_runs_out_fails_the_launch(check, paths, left_out):
    _, _, _, off = check([6] * paths, 4096, left_out)
    assert off[-1] == 0xFFFFFFFF
    _, _, _, off = check([6] * paths, 4096)  # and the next one runs
    assert 0 < off[-1] < 6 * paths
