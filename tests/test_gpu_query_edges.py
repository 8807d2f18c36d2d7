"""The guided-query kernels at their edges: the helpers of their arithmetic bit
for bit, batches of every remainder of the queries that share a warp, and
random numbers at the ends of their range against the per-object calls."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def math(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("qmath") / "libqmath.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-gencode=arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-Xcompiler",
                    "-fPIC", "-shared", "-I" + os.path.join(ROOT, "openpgl_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "query_math_check.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


def test_two_pi_times(math):
    assert math.two_pi_check() == 0


def test_phi_and_its_sine_and_cosine(math):
    assert math.phi_check() == 0
    assert math.sincos_check() == 0


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_div3(math, mode):
    assert math.div3_check(1 << 26, mode) == 0


@pytest.fixture(scope="module", params=[(300, 100, 1), (131072, 4000, 1), (262144, 64000, 4)], ids="n{0[0]}".format)
def field(request):
    """Fields of sparse regions and of regions with few, and with many lobes."""
    import openpgl_gb300 as pgl
    from openpgl_gb300 import synthetic as syn

    n, leaf, frames = request.param
    dev = pgl.Device()
    f = pgl.Field(dev, pgl.FieldConfig(True, leaf))
    st = pgl.SampleStorage()
    for i in range(frames):
        st.add_samples(syn.cube_face_samples(n, 300 + i, volume_fraction=0.5))
        f.update(st)
        st.clear()
    yield pgl, f
    f.release()


def _rows_equal(a, b):
    return all(np.array_equal(np.ascontiguousarray(a[k]).view(np.uint8), np.ascontiguousarray(b[k]).view(np.uint8))
               for k in a.dtype.names)


def test_batches_of_every_remainder(field):
    from openpgl_gb300 import synthetic as syn

    pgl, f = field
    q = syn.queries(64, 301)
    q["position"][5::7] = 1e6  # outside the field
    g = np.linspace(-0.99, 0.99, 64).astype(np.float32)
    g[3] = 0.0
    v = syn.vertices(64, 302)
    plain, hg, vert = f.sample_batch(q), f.sample_batch_hg(q, g), f.sample_vertices(v)
    for n in (1, 2, 3, 4, 5, 7, 9, 33):
        assert _rows_equal(f.sample_batch(q[:n]), plain[:n]), n
        assert _rows_equal(f.sample_batch_hg(q[:n], g[:n]), hg[:n]), n
        assert _rows_equal(f.sample_vertices(v[:n]), vert[:n]), n


def test_small_batches_equal_their_rows_in_large_ones(field):
    """Batches on either side of the sizes that take the kernels for few queries
    (16,384, with the phase function 4,096)."""
    from openpgl_gb300 import synthetic as syn

    pgl, f = field
    q, v = syn.queries(20000, 307), syn.vertices(20000, 308)
    g = np.linspace(-0.99, 0.99, 20000).astype(np.float32)
    plain, hg, vert = f.sample_batch(q), f.sample_batch_hg(q, g), f.sample_vertices(v)
    for n in (4096, 4097, 16384, 16385):
        assert _rows_equal(f.sample_batch(q[:n]), plain[:n]), n
        assert _rows_equal(f.sample_batch_hg(q[:n], g[:n]), hg[:n]), n
        assert _rows_equal(f.sample_vertices(v[:n]), vert[:n]), n


def test_ends_of_the_random_numbers(field):
    from openpgl_gb300 import synthetic as syn

    pgl, f = field
    q = syn.queries(96, 303)
    ends = np.array([0.0, 2.0 ** -33, 0.5, np.nextafter(np.float32(1), np.float32(0))], np.float32)
    q["u"][:, 0] = ends[np.arange(96) % 4]
    q["u"][:, 1] = ends[np.arange(96) // 4 % 4]
    g = np.linspace(-0.99, 0.99, 96).astype(np.float32)
    for volume, out in ((False, f.sample_batch(q)), (True, f.sample_batch_hg(q, g))):
        sd = pgl.VolumeSamplingDistribution(f) if volume else pgl.SurfaceSamplingDistribution(f)
        for i in range(len(q)):
            ok, _ = sd.init(tuple(q["position"][i]), float(q["sample1d"][i]))
            assert ok == bool(out["ok"][i])
            if not ok:
                continue
            if volume:
                sd.apply_hg_product(tuple(q["normal"][i]), float(g[i]))
            else:
                sd.apply_cosine_product(tuple(q["normal"][i]))
            d, pdf = sd.sample_pdf(tuple(q["u"][i]))
            assert np.array(d, np.float32).tobytes() == out["dir"][i].tobytes(), i
            assert np.float32(pdf).tobytes() == out["pdf"][i].tobytes(), i
        sd.release()


def test_untrained_side():
    """Queries on a side of the field without regions, and on a field before its
    first Update: all refused, nothing read."""
    import openpgl_gb300 as pgl
    from openpgl_gb300 import synthetic as syn

    dev = pgl.Device()
    f = pgl.Field(dev, pgl.FieldConfig(True, 4000))
    q, v = syn.queries(100, 304), syn.vertices(100, 305)
    g = np.full(100, 0.5, np.float32)
    st = pgl.SampleStorage()
    st.add_samples(syn.cube_face_samples(20000, 306))
    for trained in (False, True):
        if trained:
            f.update(st)
        assert not f.sample_batch_hg(q, g)["ok"].any()
        assert not f.sample_batch(q, volume=True, cosine=False)["ok"].any()
        assert f.sample_batch(q)["ok"].any() == trained
        assert f.sample_vertices(v)["ok"].any() == trained
    f.release()
