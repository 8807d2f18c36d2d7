"""Fits of leaves whose size lies at the edges of the passes' chunks (by lobe
count 320 to 416 samples of an E-step, added 16 at a time, 112 to 448 of a
split-statistics pass, 480 of a distance pass), and fits whose quotients leave
the range of the fast division: one region, a first Update and a second one,
every mixture bit for bit the oracle's."""

import os

import numpy as np
import pytest

from helpers import compare_fields, summary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 15, 16, 17, 112, 113, 140, 141, 224, 225, 320, 321, 352, 383, 384, 385, 416, 417, 448,
                               449, 480, 481, 833, 1153])
def test_leaf_sizes_at_chunk_edges(n):
    from openpgl_gb300 import synthetic as syn

    _check([syn.cube_face_samples(n, 700 + i) for i in range(2)])


@pytest.mark.parametrize("weight,pdf", [(1e-7, 1.0), (3e6, 1.0), (1.0, 1e7), (1.0, 1e-8), (0.0, 1.0)])
def test_out_of_range_quotients(weight, pdf):
    """Every seventh sample's weight, every fifth's pdf scaled."""
    from openpgl_gb300 import synthetic as syn

    frames = [syn.cube_face_samples(3001, 720 + i) for i in range(2)]
    for f in frames:
        f["weight"][::7] *= np.float32(weight)
        f["pdf"][::5] *= np.float32(pdf)
    _check(frames)


@pytest.mark.parametrize("seed", [740, 741, 742])
def test_mixtures_that_run_out_of_slots(seed):
    """Many clusters in one region: more components want to split than there
    are slots left."""
    from openpgl_gb300 import synthetic as syn

    _check([syn.cluster_samples(10000, seed + 10 * i) for i in range(3)])


def _check(frames):
    import openpgl_gb300 as pgl
    import pyoracle

    dev = pgl.Device()
    field = pgl.Field(dev, pgl.FieldConfig(True, 32000))
    orc = pyoracle.OracleField(32000, deterministic=True, threads=os.cpu_count() or 8)
    storage = pgl.SampleStorage()
    for f in frames:
        storage.add_samples(f)
        field.update(storage)
        storage.clear()
        orc.update(f)
        r = compare_fields(field.field_bytes(), orc.field_bytes())
        assert r["tree_equal"] and r["numbering_equal"] and r["stats_equal"], summary(r)
        assert r["bit_exact_regions"] == r["regions"] == 1, summary(r)
