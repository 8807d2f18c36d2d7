"""Device path samples on several streams of one thread at the same time, and
from a replayed CUDA graph beside ordinary calls: every call's samples are
those of the same call alone."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(paths, seed):
    import torch
    from openpgl_gb300 import synthetic as syn

    segs, begin = syn.path_segments(paths, seed)
    d_segs = torch.from_numpy(segs.view(np.uint8)).cuda()
    d_begin = torch.from_numpy(begin.astype(np.uint32).view(np.int32)).cuda()
    torch.cuda.synchronize()
    return d_segs, d_begin, len(begin) - 1, len(segs)


def _outputs(call):
    import torch

    out = torch.zeros(call[3] * 40, dtype=torch.uint8, device="cuda")
    off = torch.full((call[2] + 1,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return out, off


def _run(call, to, stream):
    import openpgl_gb300 as pgl

    pgl.path_samples_device(call[0].data_ptr(), call[1].data_ptr(), call[2], 30.0, to[0].data_ptr(), to[1].data_ptr(),
                            stream=stream.cuda_stream)


def _alone(call):
    import torch

    to = _outputs(call)
    _run(call, to, torch.cuda.Stream())
    torch.cuda.synchronize()
    assert 0 < int(to[1][-1]) <= call[3]
    return to


# more streams than a thread keeps buffers for, too
@pytest.mark.parametrize("count", [2, 7])
def test_streams_of_one_thread(count):
    import torch

    # long and short launches, so that each stream starts one while the others' run
    calls = [_call((200000, 3000, 40000)[i % 3], 51 + i % 3) for i in range(count)]
    want = [_alone(c) for c in calls]
    streams = [torch.cuda.Stream() for _ in calls]
    got = [[_outputs(c) for c in calls] for _ in range(8)]
    for round_ in got:
        for c, to, s in zip(calls, round_, streams):
            _run(c, to, s)
    torch.cuda.synchronize()
    for round_ in got:
        for to, w in zip(round_, want):
            assert torch.equal(to[1], w[1]) and torch.equal(to[0], w[0])


def test_graph_beside_calls():
    import torch

    call = _call(60000, 53)
    want = _alone(call)
    captured, stream, other = _outputs(call), torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        _run(call, captured, stream)
    for _ in range(6):
        captured[0].zero_()
        captured[1].fill_(-7)
        beside = _outputs(call)
        graph.replay()
        _run(call, beside, other)
        torch.cuda.synchronize()
        for to in (captured, beside):
            assert torch.equal(to[1], want[1]) and torch.equal(to[0], want[0])
