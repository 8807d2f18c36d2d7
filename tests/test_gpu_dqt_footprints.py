"""Quadtree updates whose sample boxes have no area (a footprint so small that
the box's sides round to its point) and whose leaves have none (trees so deep
that a leaf's sides round together), against the oracle: the same structure,
statistics and validity after every frame."""

import os

import numpy as np
import pytest

from helpers import compare_dqt_fields

pytestmark = pytest.mark.gpu


def _frames(kind, n, frames, seed):
    from openpgl_gb300 import synthetic as syn

    for i in range(frames):
        f = syn.cube_face_samples(n, seed + i)
        rng = np.random.Generator(np.random.PCG64(seed + 500 + i))
        if kind == "uniform":
            f["direction"] = syn._unit_sphere(rng, n).astype(np.float32)
        elif kind == "cluster":  # within a thousandth of one direction
            d = np.array([0.6, 0.48, 0.64]) + 1e-3 * rng.standard_normal((n, 3))
            f["direction"] = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        else:  # one direction, the far edge of the square
            f["direction"] = np.float32([0.0, 0.0, 1.0])
        f["weight"] = np.float32(1.0)
        yield f


def _check(args, kind, n, frames, seed):
    import openpgl_gb300 as pgl
    import pyoracle

    dev = pgl.Device()
    field = pgl.Field(dev, pgl.FieldConfig(True, 1000000, dqt=True, dqt_args=args))
    orc = pyoracle.OracleField(1000000, deterministic=True, threads=os.cpu_count() or 8, dqt=True, dqt_args=args)
    storage = pgl.SampleStorage()
    for i, f in enumerate(_frames(kind, n, frames, seed)):
        storage.add_samples(f)
        field.update(storage)
        storage.clear()
        orc.update(f)
        r = compare_dqt_fields(field.field_bytes(), orc.field_bytes(), "surface")
        assert r["structure_equal"] and r["stats_equal"] and r["valid_equal"], (i, r)
        assert r["worst_rel"] <= 1e-3, (i, r)
    import fieldfile

    tree = fieldfile.read_field_file(field.field_bytes())["surface"]["regions"][0]["dqt"]["nodes"]
    return len(tree)


# factory arguments (estimator, metric, threshold, footprint, levels): boxes without area at the
# root (1e-8) and in leaves twelve levels down (1e-4), few leaves and more than forty
@pytest.mark.parametrize("args,kind,n,frames", [
    ((0, 0, 0.01, 1e-8, 12), "uniform", 513, 2),
    ((0, 0, 0.02, 1e-4, 12), "edge", 300, 10),
    ((0, 0, 0.02, 1e-4, 12), "cluster", 3000, 4),
    ((0, 1, 0.01, 1e-4, 12), "cluster", 3000, 4),
    ((0, 0, 0.01, 1e-6, 12), "uniform", 3000, 3),
])
def test_boxes_without_area(args, kind, n, frames):
    _check(args, kind, n, frames, 7100)


# a leaf 25 levels down the square's far edge has no width; without a footprint the samples
# count for the leaf that their points descend to all the same
@pytest.mark.parametrize("threshold,n", [(0.1, 64), (0.02, 700)])
def test_leaves_without_area(threshold, n):
    nodes = _check((0, 0, threshold, 0.0, 30), "edge", n, 32, 7300)
    assert nodes > 4 * 24  # as deep as where the sides round together
