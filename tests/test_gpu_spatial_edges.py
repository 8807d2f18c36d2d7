"""Regions in numbers around the neighbour search's eight neighbours and 32
lanes, and frames at the edges of the kd passes' tiles: the tree, the regions'
statistics and the queries (which choose among a region's neighbours) against
the oracle."""

import os

import numpy as np
import pytest

from helpers import compare_fields, compare_queries, summary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regions", [1, 2, 7, 8, 9, 31, 32, 33, 64, 65, 300])
def test_numbers_of_regions(regions):
    _check(regions * 60, 80, frames=2)


@pytest.mark.parametrize("n", [255, 256, 257, 1023, 1024, 1025, 2047, 2048, 2049, 4097])
def test_frames_at_the_tiles_edges(n):
    _check(n, 700, frames=2)


def _check(n, leaf, frames):
    import openpgl_gb300 as pgl
    import pyoracle
    from openpgl_gb300 import synthetic as syn

    dev = pgl.Device()
    field = pgl.Field(dev, pgl.FieldConfig(True, leaf))
    orc = pyoracle.OracleField(leaf, deterministic=True, threads=os.cpu_count() or 8)
    storage = pgl.SampleStorage()
    for i in range(frames):
        f = syn.cube_face_samples(n, 800 + i)
        f["position"][:: 50] *= np.float32(1e4) if i else np.float32(1)  # far outside the first frame's bounds
        storage.add_samples(f)
        field.update(storage)
        storage.clear()
        orc.update(f)
        r = compare_fields(field.field_bytes(), orc.field_bytes())
        assert r["tree_equal"] and r["numbering_equal"] and r["stats_equal"], (i, summary(r))
        assert r["bit_exact_regions"] == r["regions"], (i, summary(r))
    q = syn.queries(2048, 810)
    r = compare_queries(field.sample_batch(q), orc.query(q))
    assert r["ok_equal"] and r["id_equal"] and r["sample1d_equal"], r
    assert r["worst_pdf_rel"] <= 1e-3 and r["worst_dir"] <= 1e-3, r
    field.release()
