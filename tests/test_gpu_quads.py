"""Full-resolution scores and poses on every layout of the finest level's
bilinear cells (8-bit and 16-bit quads, plain floats), at image sizes that
leave ragged tiles, against the FP64 oracle.  Tolerances: the operator's
(0.05 px, 0.05 degrees, 1e-4); full-resolution scores are FP32 sums, 1e-4 as
in the stage tests."""
import math

import numpy as np
import pytest

import oracle_lib
from mvkit_gb300 import workloads as W

pytestmark = pytest.mark.gpu
A = math.radians(25)


# maximum grey value, lowest level: level 0 of uint8 (8 bits), level 1 of
# uint8 and level 0 of uint16 (16 bits), level 1 of uint16 (floats)
@pytest.mark.parametrize("maxval, lowest", [(255, 1), (255, 2), (65535, 1), (4095, 2)])
@pytest.mark.parametrize("h, w", [(241, 313), (256, 320), (239, 310)])
def test_scores_and_poses(maxval, lowest, h, w):
    import mvkit_gb300 as mg

    orc = oracle_lib.oracle()
    wl = W.make_workload(40 + h, h, w, 56, 1, angle_range=(-A, A), maxval=maxval, border=41,
                         noise_sigma=3 if maxval == 255 else 20)
    om = orc.create(wl.template, levels=3, angle_start=-A, angle_extent=2 * A)
    model = mg.create_ncc_model(wl.template, 3, -A, 2 * A, "auto", "use_polarity")
    ctl = (-A, 2 * A, 0.6, 1, 0.5)
    want = orc.find(om, wl.image, *ctl, True, 3, lowest, stage=100)
    want = {tuple(r[:3]): r[3] for r in want if np.isfinite(r[3])}
    got = {tuple(r[:3]): r[3] for r in mg.find_ncc_model_stage(wl.image, model, *ctl, "true", [3, lowest], stage=100)}
    assert len(set(want) ^ set(got)) <= 2 and len(want) > 0
    assert all(abs(got[k] - want[k]) < 1e-4 for k in got if k in want)
    a = np.stack(mg.find_ncc_model(wl.image, model, *ctl, "true", [3, lowest]), 1)
    b = oracle_lib.to_halcon(orc.find(om, wl.image, *ctl, True, 3, lowest))
    assert a.shape == b.shape
    d = np.abs(a - b)
    assert d[:, :2].max() <= 0.05 and d[:, 2].max() <= math.radians(0.05) and d[:, 3].max() <= 1e-4


def test_models_of_different_finest_levels():
    """One image, models whose finest levels differ: the cells' buffer of a
    fresh thread grows with the second model, and the first one's refinement
    reads it after the third has filled it again.  Per-model quotas: each
    model's matches are those of its own search."""
    import threading

    import mvkit_gb300 as mg

    wl = W.make_multi_workload(77, 300, 420, (56, 64, 48), (1, 1, 1), angle_range=(-A, A))
    models = [mg.create_ncc_model(t, 3, -A, 2 * A, "auto", "use_polarity") for t in wl.templates]
    low = [2, 1, 2]
    out = {}

    def run():
        out["all"] = mg.find_ncc_models(wl.image, models, [-A] * 3, [2 * A] * 3, [0.6] * 3, [1] * 3, [0.5] * 3,
                                        ["true"] * 3, [v for k in low for v in (3, k)])

    t = threading.Thread(target=run)
    t.start()
    t.join()
    got = np.stack(out["all"][:4], 1)
    for k, m in enumerate(models):
        alone = np.stack(mg.find_ncc_model(wl.image, m, -A, 2 * A, 0.6, 1, 0.5, "true", [3, low[k]]), 1)
        assert np.array_equal(got[out["all"][4] == k], alone)
