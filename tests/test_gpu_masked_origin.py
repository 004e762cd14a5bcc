"""Masked templates whose origin lies outside the box of their samples on a
coarser level: a block beside a comb of one-pixel lines, which the 2 x 2 mask
reduction removes while the origin stays the level-0 centroid.  Lowest pyramid
level 2, the part so near an image edge that the origin's own cell lies outside
the level while every sample lies inside.

On the first row and column the search is compared with the FP64 oracle.  On the
last ones the oracle, like the reference's coarse scan
(src/ncc_matching/matcher.cpp:542-594), would write scores past the last row of
its plane, so the match there is compared with the oracle's on the mirrored image
and template (sides are multiples of four: the pyramids mirror too).  In all
cases every full-resolution score is compared with the FP64 NCC of its pose.
Tolerances: the operator's (0.05 px, 0.05 degrees, 1e-4), and 1e-4 for scores as
in the stage tests."""
import math

import numpy as np
import pytest

import oracle_lib
from mvkit_gb300 import workloads as W

A = math.radians(6)
CONTROLS = (-A, 2 * A, 0.6, 1, 0.5)


def edge_case(maxval, transpose):
    """(image, template, mask): the part at an integer offset, its centroid a
    quarter pixel below the first row (transposed: right of the first column)."""
    dtype = np.uint8 if maxval == 255 else np.uint16
    mask = np.zeros((96, 64), np.uint8)
    mask[0:64:2] = 1
    mask[64:] = 1
    tmpl = np.clip(W.scene(91, 240, 240, maxval=maxval)[60:156, 70:134], 0, maxval).astype(dtype)
    image = np.clip(W.scene(92, 304, 284, maxval=maxval), 0, maxval).astype(dtype)
    for r in range(55, 96):
        image[r - 55, 100:164][mask[r] != 0] = tmpl[r][mask[r] != 0]
    return [np.ascontiguousarray(x.T if transpose else x) for x in (image, tmpl, mask)]


def mirrored(arrays, axis):
    return [np.ascontiguousarray(np.flip(x, axis)) for x in arrays]


def level1_samples(tmpl, mask):
    """(dr, dc, weight) of the unrotated level-1 raster about its origin."""
    om = oracle_lib.oracle().create(tmpl, levels=3, mask=mask)
    _, _, orow, ocol = om.level(1)
    p = om.patch(1, 0)
    return p["rows"] - orow, p["cols"] - ocol, p["weights"]


def level1_positions(samples, pose):
    dr, dc, _ = samples
    ca, sa = math.cos(pose[2]), math.sin(pose[2])
    return (pose[0] - .5) / 2 + ca * dr - sa * dc, (pose[1] - .5) / 2 + sa * dr + ca * dc


def level1_score(level, samples, pose):
    y, x = level1_positions(samples, pose)
    if y.min() < 0 or x.min() < 0 or y.max() > level.shape[0] - 1 or x.max() > level.shape[1] - 1:
        return None
    i, j = np.floor(y).astype(int), np.floor(x).astype(int)
    i1, j1 = np.minimum(i + 1, level.shape[0] - 1), np.minimum(j + 1, level.shape[1] - 1)
    fy, fx = y - i, x - j
    q = (1 - fy) * ((1 - fx) * level[i, j] + fx * level[i, j1]) + fy * ((1 - fx) * level[i1, j] + fx * level[i1, j1])
    q -= q.mean()
    return float((samples[2] * q).sum() / math.sqrt((q * q).sum()))


def oracle_match(arrays):
    image, tmpl, mask = arrays
    orc = oracle_lib.oracle()
    om = orc.create(tmpl, levels=3, angle_start=-A, angle_extent=2 * A, mask=mask)
    (pose,) = orc.find(om, image, *CONTROLS, True, 3, 2)
    return pose


def expected(arrays, flip, axis):
    """The match of `arrays`, by way of the mirror image when flipped."""
    if not flip:
        return oracle_match(arrays)
    pose = oracle_match(mirrored(arrays, axis))
    pose[axis] = arrays[0].shape[axis] - 1 - pose[axis]
    pose[2] = -pose[2]
    return pose


CASES = [(maxval, flip, transpose) for maxval in (255, 4095) for flip in (False, True) for transpose in (False, True)]


def case_arrays(maxval, flip, transpose):
    axis = 1 if transpose else 0
    arrays = edge_case(maxval, transpose)
    return (mirrored(arrays, axis) if flip else arrays), axis


@pytest.mark.parametrize("maxval, flip, transpose", CASES)
def test_origin_cell_lies_outside(maxval, flip, transpose):
    """What makes the case: on level 1 the match's samples lie inside the level
    with more than a cell to spare, and the cell of its origin does not."""
    arrays, axis = case_arrays(maxval, flip, transpose)
    pose = expected(arrays, flip, axis)
    assert pose[3] > 0.95 and abs(pose[2]) < 0.02
    y, x = level1_positions(level1_samples(*arrays[1:]), pose)
    size = [n // 2 for n in arrays[0].shape]
    assert y.min() > 1 and x.min() > 1 and y.max() < size[0] - 2 and x.max() < size[1] - 2
    cell = math.floor((pose[axis] - .5) / 2)
    assert cell + 1 >= size[axis] if flip else cell < 0


@pytest.mark.gpu
@pytest.mark.parametrize("maxval, flip, transpose", CASES)
def test_part_at_the_edge(maxval, flip, transpose):
    import mvkit_gb300 as mg

    arrays, axis = case_arrays(maxval, flip, transpose)
    image, tmpl, mask = arrays
    model = mg.create_ncc_model(tmpl, 3, -A, 2 * A, "auto", "use_polarity", domain=mask)
    scored = mg.find_ncc_model_stage(image, model, *CONTROLS, "true", [3, 2], stage=100)
    if not flip:
        orc = oracle_lib.oracle()
        om = orc.create(tmpl, levels=3, angle_start=-A, angle_extent=2 * A, mask=mask)
        want = {tuple(r[:3]) for r in orc.find(om, image, *CONTROLS, True, 3, 2, stage=100) if np.isfinite(r[3])}
        assert len(want) > 0 and len(want ^ {tuple(r[:3]) for r in scored}) <= 2
    level = image.astype(np.float64).reshape(image.shape[0] // 2, 2, image.shape[1] // 2, 2).sum((1, 3))
    samples = level1_samples(tmpl, mask)
    assert len(scored) > 0
    for r in scored:
        assert abs(r[3] - level1_score(level, samples, r)) < 1e-4
    got = np.stack(mg.find_ncc_model(image, model, *CONTROLS, "true", [3, 2]), 1)
    assert got.shape == (1, 4)
    d = np.abs(got - oracle_lib.to_halcon(expected(arrays, flip, axis)))[0]
    assert d[:2].max() <= 0.05 and d[2] <= math.radians(0.05) and d[3] <= 1e-4
