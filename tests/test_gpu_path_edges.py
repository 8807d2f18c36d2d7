"""Device path samples at the edges of a tile (480 staged segments, 8 to 256
paths) against the host's per-path objects, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(lengths, start=0, seed=41, flags=range(8), backwards=()):
    import openpgl_gb300 as pgl
    import torch
    from openpgl_gb300 import synthetic as syn

    begin = start + np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    segs, _ = syn.path_segments(int(begin[-1]) // 2 + 64, seed)
    assert len(segs) >= begin[-1]
    for p in backwards:  # such a path has no segments, and the next one starts here
        begin[p + 1] = begin[p] - 1
    d_segs = torch.from_numpy(segs.view(np.uint8)).cuda()
    d_begin = torch.from_numpy(begin.astype(np.uint32).view(np.int32)).cuda()
    room = int(np.maximum(np.diff(begin), 0).sum())
    for fl in flags:
        d_out = torch.full(((room + 1) * 40,), 0x5A, dtype=torch.uint8, device="cuda")
        d_off = torch.full((len(begin) + 1,), -7, dtype=torch.int32, device="cuda")
        pgl.path_samples_device(d_segs.data_ptr(), d_begin.data_ptr(), len(begin) - 1, 30.0, d_out.data_ptr(),
                                d_off.data_ptr(), bool(fl & 1), bool(fl & 2), bool(fl & 4))
        torch.cuda.synchronize()
        off, out = d_off.cpu().numpy(), d_out.cpu().numpy()
        want, counts = [], [0]
        st = pgl.PathSegmentStorage(reserve=2000)
        st.set_max_distance(30.0)
        for b, e in zip(begin[:-1], begin[1:]):
            if e > b:
                st.clear()
                st.add_segments(segs[int(b):int(e)])
                st.prepare_samples(bool(fl & 1), bool(fl & 2), bool(fl & 4))
                want.append(np.asarray(st.samples()).tobytes())
                counts.append(len(want[-1]) // 40)
            else:
                counts.append(0)
        assert np.array_equal(off[:-1], np.cumsum(counts)), fl
        assert off[-1] == -7
        want = b"".join(want)
        assert out[:len(want)].tobytes() == want, fl
        assert (out[len(want):] == 0x5A).all()  # nothing past the samples


@pytest.mark.parametrize("length", [1, 2, 65, 66, 479, 480, 481, 513, 1025, 1500])
def test_one_path(length):
    _check([length])


@pytest.mark.parametrize("paths", [1, 7, 8, 9, 257, 4000])
@pytest.mark.parametrize("length", [0, 1, 2, 8, 40])
def test_paths_of_one_length(paths, length):
    _check([length] * paths, flags=(2, 5))


def test_mixed_lengths_and_starts():
    rng = np.random.default_rng(5)
    lengths = rng.integers(0, 20, 700)
    lengths[rng.integers(0, 700, 40)] = 0
    lengths[[10, 64, 127, 300]] = (600, 481, 480, 1300)
    for start in (0, 1, 3):  # odd first segments lie 8 bytes off the copies' boundary
        _check(lengths, start=start, flags=(0, 2, 7))


def test_paths_whose_ends_lie_before_their_beginnings():
    _check([5] * 3000, start=10, backwards=(3, 70, 2999), flags=(2,))
    _check([5] * 150, start=10, backwards=(3, 70, 149), flags=(2,))


def test_no_paths():
    _check([], flags=(0,))
