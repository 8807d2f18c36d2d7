"""Device path samples read their segments as PGLPathSegmentData (8 bytes
aligned) by wide copies: an address that is not is refused on the host."""

import pytest

pytestmark = pytest.mark.gpu


def test_misaligned_segments_are_refused():
    import numpy as np
    import openpgl_gb300 as pgl
    import torch
    from openpgl_gb300 import synthetic as syn

    segs, begin = syn.path_segments(100, 71)
    d = torch.zeros(len(segs) * 136 + 16, dtype=torch.uint8, device="cuda")
    d_begin = torch.from_numpy(begin.astype(np.uint32).view(np.int32)).cuda()
    out = torch.zeros(len(segs) * 40, dtype=torch.uint8, device="cuda")
    off = torch.zeros(len(begin), dtype=torch.int32, device="cuda")
    for shift in (4, 8):
        d[shift:shift + len(segs) * 136] = torch.from_numpy(segs.view(np.uint8).reshape(-1)).cuda()
        torch.cuda.synchronize()
        args = (d.data_ptr() + shift, d_begin.data_ptr(), len(begin) - 1, 30.0, out.data_ptr(), off.data_ptr())
        if shift % 8:
            with pytest.raises(RuntimeError, match="aligned"):
                pgl.path_samples_device(*args)
        else:
            pgl.path_samples_device(*args)
            torch.cuda.synchronize()
            assert 0 < int(off[-1]) < len(segs)
