"""Masked templates whose origin lies outside the box of their samples on a
coarser level: a block beside a comb of one-pixel lines, which the 2 x 2 mask
reduction removes while the origin stays the level-0 centroid.  Lowest pyramid
level 2, the part so near an image edge that the origin's own cell lies outside
the level while every sample lies inside, against the FP64 oracle.
Tolerances: the operator's (0.05 px, 0.05 degrees, 1e-4) and the stage tests'
1e-4 for full-resolution scores."""
import math

import numpy as np
import pytest

import oracle_lib
from mvkit_gb300 import workloads as W

A = math.radians(6)


def comb_case(maxval, flip, transpose):
    """(image, template, mask): the part at an integer offset, its centroid on
    the first row or, flipped, on the last one; transposed, on a column."""
    dtype = np.uint8 if maxval == 255 else np.uint16
    mask = np.zeros((96, 64), np.uint8)
    mask[0:64:2] = 1
    mask[64:] = 1
    tmpl = np.clip(W.scene(91, 240, 240, maxval=maxval)[60:156, 70:134], 0, maxval).astype(dtype)
    image = np.clip(W.scene(92, 301, 283, maxval=maxval), 0, maxval).astype(dtype)
    if flip:
        tmpl, mask = tmpl[::-1], mask[::-1]
    centre = float((np.arange(96) * mask.sum(1)).sum() / mask.sum())
    shift = image.shape[0] - 1 - math.ceil(centre) if flip else -math.floor(centre)
    for r in range(96):
        if 0 <= r + shift < image.shape[0]:
            image[r + shift, 100:164][mask[r] != 0] = tmpl[r][mask[r] != 0]
    if transpose:
        image, tmpl, mask = image.T, tmpl.T, mask.T
    return np.ascontiguousarray(image), np.ascontiguousarray(tmpl), np.ascontiguousarray(mask)


CASES = [(maxval, flip, transpose) for maxval in (255, 4095) for flip in (False, True) for transpose in (False, True)]
CONTROLS = (-A, 2 * A, 0.6, 1, 0.5)


@pytest.mark.parametrize("maxval, flip, transpose", CASES)
def test_case_has_its_origin_cell_outside(maxval, flip, transpose):
    """What makes the case: on level 1 the match's sample box lies inside the
    image, by more than a cell, and the cell of the origin does not."""
    image, tmpl, mask = comb_case(maxval, flip, transpose)
    orc = oracle_lib.oracle()
    om = orc.create(tmpl, levels=3, angle_start=-A, angle_extent=2 * A, mask=mask)
    (row, col, angle, score), = orc.find(om, image, *CONTROLS, True, 3, 2)
    assert abs(angle) < 0.02 and score > 0.95
    _, _, orow, ocol = om.level(1)
    ca, sa = math.cos(angle), math.sin(angle)
    first = orc.create(tmpl, levels=3, mask=mask).patch(1, 0)  # the unrotated raster
    dr, dc = first["rows"] - orow, first["cols"] - ocol
    y = (row - .5) / 2 + ca * dr - sa * dc
    x = (col - .5) / 2 + sa * dr + ca * dc
    h, w = image.shape[0] // 2, image.shape[1] // 2
    assert y.min() > 1 and x.min() > 1 and y.max() < h - 2 and x.max() < w - 2
    cell = (math.floor((row - .5) / 2), math.floor((col - .5) / 2))
    k = 1 if transpose else 0
    assert cell[k] + 1 >= (h, w)[k] if flip else cell[k] < 0


@pytest.mark.gpu
@pytest.mark.parametrize("maxval, flip, transpose", CASES)
def test_part_at_the_edge_matches_oracle(maxval, flip, transpose):
    import mvkit_gb300 as mg

    image, tmpl, mask = comb_case(maxval, flip, transpose)
    orc = oracle_lib.oracle()
    om = orc.create(tmpl, levels=3, angle_start=-A, angle_extent=2 * A, mask=mask)
    model = mg.create_ncc_model(tmpl, 3, -A, 2 * A, "auto", "use_polarity", domain=mask)
    want = orc.find(om, image, *CONTROLS, True, 3, 2, stage=100)
    want = {tuple(r[:3]): r[3] for r in want if np.isfinite(r[3])}
    got = {tuple(r[:3]): r[3]
           for r in mg.find_ncc_model_stage(image, model, *CONTROLS, "true", [3, 2], stage=100)}
    assert len(want) > 0 and len(set(want) ^ set(got)) <= 2
    assert all(abs(got[k] - want[k]) < 1e-4 for k in got if k in want)
    a = np.stack(mg.find_ncc_model(image, model, *CONTROLS, "true", [3, 2]), 1)
    b = oracle_lib.to_halcon(orc.find(om, image, *CONTROLS, True, 3, 2))
    assert a.shape == b.shape == (1, 4)
    d = np.abs(a - b)
    assert d[:, :2].max() <= 0.05 and d[:, 2].max() <= math.radians(0.05) and d[:, 3].max() <= 1e-4
