"""MaxOverlap decisions at angles far from zero (AngleStart may be any finite
angle).  Two bars overlap by a known ratio at one angle near 65536 rad, where a
float angle is off by up to 0.0039 rad: their rectangles then overlap by more
than 0.5 % of the bar more or less.  The second bar is found exactly when MaxOverlap
is above the FP64 ratio, with thresholds 0.2 % to either side."""
import math

import numpy as np
import pytest

import oracle_lib
from mvkit_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def far_angle(sign):
    """Nearly a whole number of turns, as far from a float as one can be."""
    for k in range(10440, 10700):
        a = sign * (2 * math.pi * k + 1e-4)
        if abs(a - float(np.float32(a))) > 0.0036:
            return a
    raise AssertionError("no such angle")


def scene_of_bars():
    tmpl = np.clip(W.scene(21, 300, 300), 0, 255).astype(np.uint8)[100:124, 60:220]
    image = np.clip(W.scene(22, 240, 480), 0, 255).astype(np.uint8)
    image[100:124, 60:220] = tmpl
    image[112:136, 160:320] = tmpl
    return image, np.ascontiguousarray(tmpl)


@pytest.mark.parametrize("sign", [1, -1])
def test_overlap_at_a_far_angle(sign):
    import mvkit_gb300 as mg

    image, tmpl = scene_of_bars()
    a = far_angle(sign)
    orc = oracle_lib.oracle()
    om = orc.create(tmpl, levels=2, angle_start=a, angle_extent=0.0)
    p, q = orc.find(om, image, a, 0.0, 0.5, 2, 0.5, False, 2, 1)
    # both at the same angle, within 1e-4 rad of upright (less than 2e-4 of the bar)
    ratio = (160 - abs(p[1] - q[1])) * (24 - abs(p[0] - q[0])) / (160 * 24)
    model = mg.create_ncc_model(tmpl, 2, a, 0.0, "auto", "use_polarity")
    second = oracle_lib.to_halcon(q)[0, :2]
    found = lambda rows: any(np.abs(r[:2] - second).max() < 0.01 for r in rows)
    for thr in (ratio - 0.002, ratio + 0.002):
        assert found(oracle_lib.to_halcon(orc.find(om, image, a, 0.0, 0.5, 2, thr, False, 2, 1))) == (thr > ratio)
        got = np.stack(mg.find_ncc_model(image, model, a, 0.0, 0.5, 2, thr, "false", 2), 1)
        assert found(got) == (thr > ratio), (thr, got)
