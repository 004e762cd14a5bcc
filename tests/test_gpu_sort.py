"""The candidate sort at its split sizes: one 256-entry segment, one merge of
up to 64 segments, two and three merges.  The sorted list holds the last tracking
step's candidates that could be scored, in the reference's order (score
descending, then row, column, angle; src/ncc_matching/matcher.cpp:824-827),
each once."""
import numpy as np
import pytest

from golden.cases import CASES, make_inputs

pytestmark = pytest.mark.gpu


# rows of the scene, tiles of it, MinScore, bounds on the number of sorted candidates
@pytest.mark.parametrize("rows, tiles, min_score, least, most", [
    (72, (1, 1), 0.95, 1, 256), (160, (1, 1), 0.95, 257, 16384), (480, (3, 3), 0.7, 16385, 1 << 20),
    (480, (10, 10), 0.7, (1 << 20) + 1, 1 << 21)])
def test_sorted_list(rows, tiles, min_score, least, most):
    import mvkit_gb300 as mg

    case = CASES["budget_360"]
    wl, _ = make_inputs(case)
    image = np.ascontiguousarray(np.tile(wl.image[:rows], tiles))
    c, f = case["create"], case["find"]
    model = mg.create_ncc_model(wl.template, "auto", c["angle_start"], c["angle_extent"], "auto", "use_polarity")
    levels = mg.get_ncc_model_params(model)[0]
    ctl = (f["angle_start"], f["angle_extent"], min_score, f["num_matches"], f["max_overlap"], "true", [0, 1])
    with mg.extended_budgets(samples=600_000_000, pixels=1 << 30, candidates=1 << 21):
        got = mg.find_ncc_model_stage(image, model, *ctl, stage=100)
        last = mg.find_ncc_model_stage(image, model, *ctl, stage=levels - 1)
    assert least <= len(got) <= most, (len(got), len(last))
    order = np.lexsort((got[:, 2], got[:, 1], got[:, 0], -got[:, 3]))
    assert np.array_equal(order, np.arange(len(got)))
    poses = {tuple(r[:3]) for r in got}
    assert len(poses) == len(got) and poses <= {tuple(r[:3]) for r in last}
    # a candidate whose template lies inside the image has a score
    reach = np.hypot(*wl.template.shape) / 2 + 2
    inside = (last[:, 0] > reach) & (last[:, 1] > reach) & (last[:, 0] < image.shape[0] - 1 - reach) & \
        (last[:, 1] < image.shape[1] - 1 - reach)
    assert {tuple(r[:3]) for r in last[inside]} <= poses
