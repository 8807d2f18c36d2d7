"""Quadtree updates at the edges of how the update kernel works (a matrix of
shares up to 40 leaves, masks and slots, every leaf tested up to 512 leaves,
descents beyond, trees in shared memory up to 768 nodes, more leaves than the
masks hold), with boxes from none to several leaves wide, against the oracle:
the same structure after every frame, node values within 1e-3 (the oracle's
atan2f is the host library's)."""

import os

import numpy as np
import pytest

from helpers import compare_dqt_fields

pytestmark = pytest.mark.gpu


# factory arguments (estimator, metric, threshold, footprint, levels), samples, frames, directions, node count at the end
@pytest.mark.parametrize("args,n,frames,uniform,nodes", [
    ((0, 0, 0.01, 1.0, 12), 1, 2, True, (1, 200)),
    ((0, 0, 0.01, 1.0, 12), 513, 2, False, (40, 400)),
    ((0, 0, 0.01, 0.0, 12), 3000, 2, False, (40, 600)),
    ((1, 1, 0.01, 0.5, 12), 3000, 2, False, (40, 600)),
    ((0, 0, 0.02, 4.0, 5), 3000, 2, False, (40, 400)),
    ((0, 0, 0.002, 1.0, 12), 9000, 3, False, (500, 3000)),
    ((0, 1, 0.0015, 2.5, 12), 5000, 2, True, (769, 6000)),
    ((0, 0, 0.0002, 1.0, 12), 4000, 4, True, (12000, 100000)),
])
def test_edges(args, n, frames, uniform, nodes):
    import openpgl_gb300 as pgl
    import pyoracle
    from openpgl_gb300 import synthetic as syn

    dev = pgl.Device()
    field = pgl.Field(dev, pgl.FieldConfig(True, 1000000, dqt=True, dqt_args=args))
    orc = pyoracle.OracleField(1000000, deterministic=True, threads=os.cpu_count() or 8, dqt=True, dqt_args=args)
    storage = pgl.SampleStorage()
    for i in range(frames):
        f = syn.cube_face_samples(n, 900 + i)
        if uniform:
            d = syn._unit_sphere(np.random.Generator(np.random.PCG64(950 + i)), n)
            f["direction"] = d.astype(np.float32)
            f["weight"] = np.float32(1.0)
        storage.add_samples(f)
        field.update(storage)
        storage.clear()
        orc.update(f)
        r = compare_dqt_fields(field.field_bytes(), orc.field_bytes(), "surface")
        assert r["structure_equal"] and r["stats_equal"] and r["valid_equal"], (i, r)
        assert r["worst_rel"] <= 1e-3, (i, r)
    import fieldfile

    tree = fieldfile.read_field_file(field.field_bytes())["surface"]["regions"][0]["dqt"]["nodes"]
    assert nodes[0] <= len(tree) <= nodes[1], len(tree)
