"""Search moments at level widths around the prefix scan's steps (128 columns,
four per lane) and on both sum widths (uint8 levels short, 16-bit levels
long), against the FP64 oracle's candidates after every stage."""
import math

import numpy as np
import pytest

import oracle_lib
from mvkit_gb300 import workloads as W

pytestmark = pytest.mark.gpu
A = math.radians(12)


@pytest.mark.parametrize("maxval", [255, 65535])
@pytest.mark.parametrize("w", [253, 256, 258, 511, 514])
def test_stages_at_scan_widths(w, maxval):
    import mvkit_gb300 as mg

    orc = oracle_lib.oracle()
    wl = W.make_workload(60 + w, 200, w, 40, 1, angle_range=(-A, A), maxval=maxval,
                         noise_sigma=3 if maxval == 255 else 20)
    om = orc.create(wl.template, levels=3, angle_start=-A, angle_extent=2 * A)
    model = mg.create_ncc_model(wl.template, 3, -A, 2 * A, "auto", "use_polarity")
    for stage in range(3):
        want = orc.find(om, wl.image, -A, 2 * A, 0.6, 1, 0.5, True, 3, 1, stage=stage)
        got = mg.find_ncc_model_stage(wl.image, model, -A, 2 * A, 0.6, 1, 0.5, "true", 3, stage)
        a, b = ({tuple(r[:3]): r[3] for r in x} for x in (got, want))
        assert len(b) > 0 and len(set(a) ^ set(b)) <= 2
        assert all(abs(a[k] - b[k]) < 2e-5 for k in a if k in b)
