"""Guided queries on either side of the size up to which surface and volume
batches take the kernel for few queries (12,160): the same rows as in a batch
that takes the other one."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("volume", [False, True], ids=["surface", "volume"])
@pytest.mark.parametrize("n", [12159, 12160, 12161])
def test_rows_are_those_of_a_larger_batch(n, volume):
    import openpgl_gb300 as pgl
    from openpgl_gb300 import synthetic as syn

    dev = pgl.Device()
    f = pgl.Field(dev, pgl.FieldConfig(True, 3000))
    storage = pgl.SampleStorage()
    storage.add_samples(syn.cube_face_samples(40000, 311, volume_fraction=0.4))
    f.update(storage)
    q = syn.queries(20000, 312)
    large, small = f.sample_batch(q, volume=volume), f.sample_batch(q[:n], volume=volume)
    assert int(large["ok"].sum()) > 10000
    assert np.array_equal(small.view(np.uint32), large[:n].view(np.uint32))
