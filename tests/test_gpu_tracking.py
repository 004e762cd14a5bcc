"""Tracking kernels at the sizes where their work split changes, against the
FP64 oracle: the candidates of every tracking step and their scores.

Scores are FP32 sums of at most 70,000 products of a unit-norm template and a
window of at most 24-bit integers; 2e-5 is the bound the stage tests use."""
import math

import numpy as np
import pytest

import oracle_lib
from mvkit_gb300 import workloads as W

pytestmark = pytest.mark.gpu
D = math.radians


def holes(n):
    """A template domain whose rows fall apart into several runs, one row empty."""
    m = np.ones((n, n), dtype=np.uint8)
    m[n // 3:n // 2, n // 4:n // 2] = 0
    m[2 * n // 3, :] = 0
    m[:, 3 * n // 4] = 0
    return m


# template side, half angle range, levels, masked, maximum grey value, correlation path
CASES = [
    (17, 6, 2, False, 255, "plain"),     # less than a strip of columns
    (33, 15, 2, False, 4095, "tensor"),  # one column past two strips; uint16 lists on the CUDA cores
    (64, 40, 3, False, 4095, "tensor"),
    (96, 10, 3, True, 255, "plain"),     # several runs per row
    (96, 10, 3, True, 255, "tensor"),
    (130, 90, 4, False, 255, "tensor"),  # long lists: several warps per candidate, the unrotated patch beside them
    (520, 1, 3, False, 255, "plain"),    # a window larger than shared memory
]


@pytest.mark.parametrize("side, deg, levels, masked, maxval, path", CASES)
def test_tracking_steps_match_oracle(side, deg, levels, masked, maxval, path):
    import mvkit_gb300 as mg

    orc = oracle_lib.oracle()
    h, w = max(240, 2 * side - 301), max(311, 2 * side - 200)
    wl = W.make_workload(5 + side, h, w, side, 1, angle_range=(-D(deg), D(deg)), maxval=maxval,
                         noise_sigma=3 if maxval == 255 else 20)
    mask = holes(side) if masked else None
    om = orc.create(wl.template, levels=levels, angle_start=-D(deg), angle_extent=D(2 * deg), mask=mask)
    model = mg.create_ncc_model(wl.template, levels, -D(deg), D(2 * deg), "auto", "use_polarity", domain=mask)
    mg.set_correlation_path(path)
    try:
        for stage in range(1, levels):
            want = orc.find(om, wl.image, -D(deg), D(2 * deg), 0.6, 2, 0.5, True, levels, 1, stage=stage)
            got = mg.find_ncc_model_stage(wl.image, model, -D(deg), D(2 * deg), 0.6, 2, 0.5, "true", levels, stage)
            a = {tuple(r[:3]): r[3] for r in got}
            b = {tuple(r[:3]): r[3] for r in want}
            assert len(b) > 0 and len(set(a) ^ set(b)) <= 2, (stage, len(a), len(b))
            assert all(abs(a[k] - b[k]) < 2e-5 for k in a if k in b)
    finally:
        mg.set_correlation_path("tensor")
