"""Refinement by a cluster of blocks (templates of 12288 samples or more) on
plain floats: a 16-bit level below the finest, and a model whose cells another
model of the same call has replaced.  Against the FP64 oracle within the
operator's tolerances (0.05 px, 0.05 degrees, 1e-4), and against the model's own
search within what a rounding of the first sample's value can move: 1e-3 px
(the acceptance near convergence), 2e-5 rad, 1e-6."""
import math

import numpy as np
import pytest

import oracle_lib
from mvkit_gb300 import workloads as W

pytestmark = pytest.mark.gpu
A = math.radians(6)


def test_float_cells_against_oracle():
    import mvkit_gb300 as mg

    orc = oracle_lib.oracle()
    wl = W.make_workload(51, 561, 603, 232, 1, angle_range=(-A, A), maxval=4095, noise_sigma=20)
    om = orc.create(wl.template, levels=4, angle_start=-A, angle_extent=2 * A)
    model = mg.create_ncc_model(wl.template, 4, -A, 2 * A, "auto", "use_polarity")
    want = oracle_lib.to_halcon(orc.find(om, wl.image, -A, 2 * A, 0.6, 1, 0.5, True, 4, 2))
    got = np.stack(mg.find_ncc_model(wl.image, model, -A, 2 * A, 0.6, 1, 0.5, "true", [4, 2]), 1)
    assert got.shape == want.shape == (1, 4)
    d = np.abs(got - want)[0]
    assert d[:2].max() <= 0.05 and d[2] <= math.radians(0.05) and d[3] <= 1e-4


def test_cells_of_another_model():
    import mvkit_gb300 as mg

    wl = W.make_multi_workload(52, 340, 460, (120, 64), (1, 1), angle_range=(-A, A))
    models = [mg.create_ncc_model(t, 3, -A, 2 * A, "auto", "use_polarity") for t in wl.templates]
    r, c, a, s, which = mg.find_ncc_models(wl.image, models, [-A] * 2, [2 * A] * 2, [0.6] * 2, [1] * 2, [0.5] * 2,
                                           ["true"] * 2, [3, 1, 3, 2])
    got = np.stack([r, c, a, s], 1)[which == 0]
    alone = np.stack(mg.find_ncc_model(wl.image, models[0], -A, 2 * A, 0.6, 1, 0.5, "true", [3, 1]), 1)
    assert got.shape == alone.shape == (1, 4)
    assert np.all(np.abs(got - alone)[0] <= [1e-3, 1e-3, 2e-5, 1e-6])
