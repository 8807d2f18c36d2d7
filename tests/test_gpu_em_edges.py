"""Fits of leaves whose size lies at the edges of the E-step's chunks (320 to
416 samples by lobe count, added 16 at a time): one region, a first Update and
a second one, every mixture bit for bit the oracle's."""

import os

import pytest

from helpers import compare_fields, summary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 15, 16, 17, 320, 321, 352, 383, 384, 385, 416, 417, 833, 1153])
def test_leaf_sizes_at_chunk_edges(n):
    import openpgl_gb300 as pgl
    import pyoracle
    from openpgl_gb300 import synthetic as syn

    frames = [syn.cube_face_samples(n, 700 + i) for i in range(2)]
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
